// LSTM forward recurrence as ONE cooperative kernel for the whole sequence (bf16, B <= 128, H = 8 * G with
// G <= number of SMs; the translation stages use H = 1024: 128 CTAs).
//
// CTA c owns hidden units u0 = 8c .. 8c+7, i.e. the 32 gate columns {g*H + u0 + j}.  Its slice of W_hh
// (32 x H, 64 KB at H = 1024) is loaded into shared memory once and stays there for all T steps.  Per step:
// the previous hidden state h_{t-1} ([B, H], a slab of the output y) streams through a ring of TMA stages,
// tcgen05.mma accumulates the [128 x 32] recurrent projection in tensor memory, and the epilogue warps - one
// thread per batch row, which then holds all four gates of its 8 units - add the input projection and the
// bias, apply the cell update (cell state kept in registers across steps) and write h_t, c_t and the gate
// activations.  A grid-wide counter separates the steps: a CTA starts loading h_t only when all CTAs have
// published their part of it.  Compared with one contraction launch plus one cell launch per step this
// removes the launches, the round trip of the projection through HBM and the per-step reload of W_hh.
//
// Every wait is bounded; a wait that runs out (or an error seen by another role / CTA) sets the error word
// of the tensor-core kernels and makes every role leave its loop, after which tensor memory is freed.
#include "pd_gemm.cuh"
#include "pd_sm100_ptx.cuh"
#include <mutex>

namespace {

using namespace pd_sm100;

constexpr int kMaxStages = 16;
// warp 0: TMA producer, warp 1: MMA issuer, warps 2-5: cell epilogue, warps 6...: more MMA issuers.  A step is a chain
// of 64 (backward: 32) small MMAs, and their issue costs more than their work; the K-blocks of a
// step are dealt out to the issuers, each adds up in columns of its own, and the epilogue adds the parts.
constexpr int kFwdIssuers = 4;           // one where two CTAs share an SM: more would not leave them the registers
constexpr int kFwdParts = 4;
constexpr int kBwdIssuers = 2;
constexpr int block_threads(int issuers) { return 192 + 32 * (issuers - 1); }
constexpr int kBwdThreads = block_threads(kBwdIssuers);
constexpr int kUnits = 8;                // hidden units per CTA
constexpr int kCols = 4 * kUnits;        // gate columns per CTA = MMA N
constexpr uint32_t kStageBytes = 128 * kBlockK * 2;      // one [128 x 64] K-block of h: 16 KiB
constexpr uint32_t kWBlockBytes = kCols * kBlockK * 2;   // one [32 x 64] K-block of the W_hh slice: 4 KiB

struct LstmP {
  int T, B, H, G, num_stages, issuers;
  int parts;                   // accumulators that a step's K-blocks are dealt out to, whatever the number of issuers
  int Bt, b0;                  // the tensors hold Bt batch rows per time step; this launch works on rows b0 .. b0 + B - 1
  uint32_t stage_bytes;        // one K-block of the h tile in shared memory: B rows rounded up to 8, 128 bytes each
  const __nv_bfloat16* gx;     // [T, B, 4H]
  const __nv_bfloat16* b_hh;   // [4H] or null
  __nv_bfloat16* y;            // [T, B, H]
  __nv_bfloat16* act;          // [T, B, 4H]
  float* c_all;                // [T, B, H]
  unsigned int* counter;       // zeroed before the launch
  int* err;
  uint32_t idesc;
};

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// One thread waits for the grid-wide counter; returns false when the bound ran out or an error is pending.  The poll
// is the link of the per-step chain that every CTA sits on: it is one acquire load per trip, and the error word
// (another round trip to L2) and the clock are looked at on every 32nd trip only.
__device__ __forceinline__ bool wait_counter(const unsigned int* counter, unsigned int target, int* err, int code) {
  const long long t0 = clock64();
  unsigned int trips = 0;
  while (ld_acquire(counter) < target) {
    if ((++trips & 31u) == 0u) {
      if (*(volatile int*)err != 0) return false;
      if (clock64() - t0 > kWaitCycles) { atomicCAS(err, 0, code); return false; }
    }
  }
  return true;
}

// Publish after a named barrier of the 128 epilogue threads: their global writes are ordered before the barrier,
// one thread then counts this CTA in with release semantics, which cover what it has observed through the barrier.
__device__ __forceinline__ void publish_step(unsigned int* counter, bool elected) {
  asm volatile("bar.sync 1, 128;" ::: "memory");
  if (elected) asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(counter), "r"(1u) : "memory");
}

// mbarrier wait that also gives up when another role or CTA has reported an error
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, int* err, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (*(volatile int*)err != 0) return false;
    if (clock64() - t0 > kWaitCycles) {
      atomicCAS(err, 0, code);
      return false;
    }
  }
}

__device__ __forceinline__ bool wait_bar_warp(uint32_t bar, uint32_t parity, int* err, int code) {
  return __all_sync(0xffffffffu, (int)wait_bar(bar, parity, err, code)) != 0;
}

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 t = __bfloat1622float2(p[k]);
    f[2 * k] = t.x;
    f[2 * k + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
  return u;
}

template <int NI>                        // issuer warps (p.issuers of them have work)
__global__ void __launch_bounds__(block_threads(NI), 1)
lstm_fwd_persistent_kernel(const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_w,
                           const LstmP p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
  __shared__ __align__(8) uint64_t w_bar;
  __shared__ __align__(8) uint64_t acc_bar;
  __shared__ uint32_t tmem_base_holder;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int S = p.num_stages;
  const int kblocks = p.H / kBlockK;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_w = smem0;                                        // kblocks x 4 KiB
  const uint32_t smem_a = smem0 + (uint32_t)kblocks * kWBlockBytes;     // S stages (a multiple of 1024 in)
  const int u0 = blockIdx.x * kUnits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&w_bar), 1);
    mbar_init(smem_u32(&acc_bar), (uint32_t)p.issuers);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_holder)), "r"((uint32_t)(kFwdParts * kCols)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = tmem_base_holder;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      // the W_hh slice: per K-block four boxes of 8 rows (one per gate), 8 rows = one swizzle atom
      mbar_expect_tx(smem_u32(&w_bar), (uint32_t)kblocks * kWBlockBytes);
      for (int kb = 0; kb < kblocks; ++kb)
        for (int g = 0; g < 4; ++g)
          tma_load_2d(smem_w + (uint32_t)kb * kWBlockBytes + (uint32_t)g * 1024u, &map_w, smem_u32(&w_bar), kb * kBlockK,
                      g * p.H + u0);
      uint32_t it = 0;
      bool ok = true;
      for (int t = 1; t < p.T && ok; ++t) {
        // every CTA has published its part of h_{t-1}
        const unsigned int target = (unsigned int)p.G * (unsigned int)t;
        ok = wait_counter(p.counter, target, p.err, 5);
        if (!ok) break;
        asm volatile("fence.proxy.async;" ::: "memory");      // the TMA reads below come after what was just observed
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = (int)(it % (uint32_t)S);
          const uint32_t ph = (it / (uint32_t)S) & 1u;
          if (!wait_bar(smem_u32(&empty_bar[s]), ph ^ 1u, p.err, 1)) { ok = false; break; }
          const uint32_t fb = smem_u32(&full_bar[s]);
          mbar_expect_tx(fb, p.stage_bytes);
          tma_load_2d(smem_a + (uint32_t)s * p.stage_bytes, &map_h, fb, kb * kBlockK, (t - 1) * p.Bt + p.b0);
        }
      }
    }
  } else if (warp == 1 || warp > 5) {
    // ------------------------------- MMA issuers ------------------------------
    const int me = warp == 1 ? 0 : warp - 5;
    if (me < p.issuers) {
      bool ok = wait_bar_warp(smem_u32(&w_bar), 0, p.err, 6);
      // (the whole warp walks the loop, see umma_lo_elect)  Descriptors advance by 32-bit adds on
      // their low words and the ring position is carried along instead of being derived by division.
      const uint64_t da0 = make_desc(smem_a, 0), db0 = make_desc(smem_w, 0);
      const uint32_t a_hi = (uint32_t)(da0 >> 32), b_hi = (uint32_t)(db0 >> 32);
      const uint32_t a_lo0 = (uint32_t)da0, b_lo0 = (uint32_t)db0;
      const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
      const uint32_t idesc = p.idesc, a_step = p.stage_bytes >> 4;
      const int issuers = p.issuers;
      for (int t = 1; t < p.T && ok; ++t) {
        const uint32_t it0 = (uint32_t)(t - 1) * (uint32_t)kblocks + (uint32_t)me;
        uint32_t s = it0 % (uint32_t)S, ph = (it0 / (uint32_t)S) & 1u;
        uint32_t b_lo = b_lo0 + (uint32_t)me * (kWBlockBytes >> 4);
        for (int kb = me; kb < kblocks; kb += issuers) {
          if (!wait_bar_warp(full0 + 8u * s, ph, p.err, 2)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_lo = a_lo0 + s * a_step, acc = tmem_acc + (uint32_t)((kb & (p.parts - 1)) * kCols);
          if (kb < p.parts) umma_lo_elect<1, 0>(acc, a_lo, a_hi, b_lo, b_hi, idesc, 0u);
          else umma_lo_elect<1, 1>(acc, a_lo, a_hi, b_lo, b_hi, idesc, 1u);
#pragma unroll
          for (int kk = 1; kk < kBlockK / 16; ++kk)
            umma_lo_elect<1, 1>(acc, a_lo + kk * 2, a_hi, b_lo + kk * 2, b_hi, idesc, 1u);
          umma_commit_elect(empty0 + 8u * s);
          b_lo += (uint32_t)issuers * (kWBlockBytes >> 4);
          s += (uint32_t)issuers;
          if (s >= (uint32_t)S) { s -= (uint32_t)S; ph ^= 1u; }
        }
        if (ok) umma_commit_elect(smem_u32(&acc_bar));
      }
    }
  } else {
    // ------------------------------ cell epilogue ------------------------------
    const int lg = warp & 3;                       // TMEM lane group of this warp
    const int b = lg * 32 + lane;                  // batch row
    const bool row = b < p.B;
    const int H = p.H;
    float c[kUnits];
#pragma unroll
    for (int j = 0; j < kUnits; ++j) c[j] = 0.f;
    float bias[kCols];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int j = 0; j < kUnits; ++j)
        bias[g * kUnits + j] = p.b_hh != nullptr ? __bfloat162float(p.b_hh[g * H + u0 + j]) : 0.f;
    bool ok = true;
    for (int t = 0; t < p.T && ok; ++t) {
      // input projection of this row: four 16-byte pieces (one per gate), in flight while the MMAs run
      uint4 gxv[4];
      const int64_t row4 = ((int64_t)t * p.Bt + p.b0 + (row ? b : 0)) * 4 * H + u0;
#pragma unroll
      for (int g = 0; g < 4; ++g) gxv[g] = *reinterpret_cast<const uint4*>(p.gx + row4 + (int64_t)g * H);
      uint32_t r[kCols];
      uint4 hold[4];                                 // gate activations of this step, stored after the publish
      if (t > 0) {
        ok = wait_bar(smem_u32(&acc_bar), (uint32_t)(t - 1) & 1u, p.err, 3);
        // one decision for all four epilogue warps (they meet at a named barrier further down)
        unsigned int all_ok;
        asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.and.pred p, 2, 128, q;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(all_ok) : "r"((unsigned int)ok) : "memory");
        ok = all_ok != 0;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_acc + ((uint32_t)(lg * 32) << 16);
        tmem_ld32(acc, r);
        tmem_ld_wait();
        for (int q = 1; q < p.parts; ++q) {
          uint32_t r2[kCols];
          tmem_ld32(acc + (uint32_t)(q * kCols), r2);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kCols; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
        }
      } else {
#pragma unroll
        for (int j = 0; j < kCols; ++j) r[j] = 0u;
      }
      if (row) {
        float pre[kCols];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float f[8];
          unpack8(gxv[g], f);
#pragma unroll
          for (int j = 0; j < kUnits; ++j) {
            float v = f[j];
            if (t > 0) v += __uint_as_float(r[g * kUnits + j]);
            if (p.b_hh != nullptr) v += bias[g * kUnits + j];
            pre[g * kUnits + j] = v;
          }
        }
        float hi[kUnits], ai[kUnits], af[kUnits], ag[kUnits], ao[kUnits];
#pragma unroll
        for (int j = 0; j < kUnits; ++j) {
          ai[j] = sigmoidf_(pre[j]);
          af[j] = sigmoidf_(pre[kUnits + j]);
          ag[j] = tanhf(pre[2 * kUnits + j]);
          ao[j] = sigmoidf_(pre[3 * kUnits + j]);
          c[j] = af[j] * c[j] + ai[j] * ag[j];
          hi[j] = ao[j] * tanhf(c[j]);
        }
        const int64_t rowh = ((int64_t)t * p.Bt + p.b0 + b) * H + u0;
        *reinterpret_cast<uint4*>(p.y + rowh) = pack8(hi);
        hold[0] = pack8(ai); hold[1] = pack8(af); hold[2] = pack8(ag); hold[3] = pack8(ao);
      }
      // publish: the accumulator has been read (the next step may overwrite it) and h_t is written
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      publish_step(p.counter, warp == 2 && lane == 0);
      // what only the backward pass reads goes out after the other CTAs have been let go
      if (row) {
        const int64_t rowh = ((int64_t)t * p.Bt + p.b0 + b) * H + u0;
        float4* cp = reinterpret_cast<float4*>(p.c_all + rowh);
        cp[0] = make_float4(c[0], c[1], c[2], c[3]);
        cp[1] = make_float4(c[4], c[5], c[6], c[7]);
        __nv_bfloat16* ap = p.act + ((int64_t)t * p.Bt + p.b0 + b) * 4 * H + u0;
        *reinterpret_cast<uint4*>(ap) = hold[0];
        *reinterpret_cast<uint4*>(ap + H) = hold[1];
        *reinterpret_cast<uint4*>(ap + 2 * (int64_t)H) = hold[2];
        *reinterpret_cast<uint4*>(ap + 3 * (int64_t)H) = hold[3];
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"((uint32_t)(kFwdParts * kCols)) : "memory");
  }
}


// ------------------------------------------------------------------------------------------------
// Backward recurrence, whole sequence in one cooperative kernel (bf16, B <= 128, H a power of two in
// 128..1024: G = (H/128)^2 CTAs).  Two phases per step, separated by a grid-wide counter:
//   A(t): cell backward.  CTA c owns the U = H/G hidden units from c*U for all rows: dh = dy[t] + dh_acc,
//         dgates[t] from the saved activations and cell states, dh_acc cleared.
//   B(t): dh_acc += dgates[t] . W_hh.  CTA (ns, ks) contracts the K slice [512 ks, 512 ks + 512) of the 4H gate
//         columns into the 128 units of slice ns: its [512 x 128] piece of W_hh sits in shared memory for the
//         whole sequence (MN-major operand, read in place), dgates[t] streams in by TMA, 32 MMAs of
//         128 x 128 x 16 accumulate in tensor memory and the epilogue adds the tile to dh_acc with red.v4.f32.
// ------------------------------------------------------------------------------------------------
constexpr int kBwdMaxStages = 8;
constexpr uint32_t kBwdRing = 64 * 1024;   // stages of dgates: 4 of 128 rows, 8 of 64 rows or fewer
constexpr int kBwdN = 128;               // units per N slice
constexpr int kBwdK = 512;               // gate columns per K slice
constexpr uint32_t kBwdWBytes = kBwdK * kBwdN * 2;       // 128 KiB

struct LstmBwdP {
  int T, B, H, G, NS;
  int num_stages;
  uint32_t stage_bytes;         // as in LstmP
  int Bt, b0;                   // as in LstmP
  const __nv_bfloat16* dy;      // [T, B, H]
  const __nv_bfloat16* act;     // [T, B, 4H]
  const float* c_all;           // [T, B, H]
  __nv_bfloat16* dgates;        // [T, B, 4H]
  float* dh_acc;                // [B, H], zeroed before the launch
  unsigned int* counter;        // zeroed before the launch
  int* err;
  uint32_t idesc;
};

// What a step's cell backward reads for eight units of a row, except dh: nothing here depends on the chain.
struct CellIn {
  uint4 dy, a[4];
  float4 q0, q1;                // c_{t-1}
};
__device__ __forceinline__ void load_cell(CellIn& in, const LstmBwdP& p, int t, int b, int u) {
  const int H = p.H;
  const int64_t e = ((int64_t)t * p.Bt + p.b0 + b) * H + u;         // [T,Bt,H] element
  const int64_t e4 = ((int64_t)t * p.Bt + p.b0 + b) * 4 * H + u;    // [T,Bt,4H] element of gate 0
  in.dy = *reinterpret_cast<const uint4*>(p.dy + e);
#pragma unroll
  for (int g = 0; g < 4; ++g) in.a[g] = *reinterpret_cast<const uint4*>(p.act + e4 + (int64_t)g * H);
  in.q0 = in.q1 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (t > 0) {
    in.q0 = *reinterpret_cast<const float4*>(p.c_all + e - (int64_t)p.Bt * H);
    in.q1 = *(reinterpret_cast<const float4*>(p.c_all + e - (int64_t)p.Bt * H) + 1);
  }
}
// The factors that dh and dc are multiplied with.
struct CellK { float dy[8], dc[8], f[8], ki[8], kf[8], kg[8], ko[8]; };
__device__ __forceinline__ void cell_factors(CellK& k, const CellIn& in, const float* ct) {
  float ai[8], ag[8], ao[8];
  const float cp[8] = {in.q0.x, in.q0.y, in.q0.z, in.q0.w, in.q1.x, in.q1.y, in.q1.z, in.q1.w};
  unpack8(in.dy, k.dy);
  unpack8(in.a[0], ai);
  unpack8(in.a[1], k.f);
  unpack8(in.a[2], ag);
  unpack8(in.a[3], ao);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float tc = tanhf(ct[j]);
    k.dc[j] = ao[j] * (1.f - tc * tc);
    k.ki[j] = ag[j] * ai[j] * (1.f - ai[j]);
    k.kf[j] = cp[j] * k.f[j] * (1.f - k.f[j]);
    k.kg[j] = ai[j] * (1.f - ag[j] * ag[j]);
    k.ko[j] = tc * ao[j] * (1.f - ao[j]);
  }
}
// dh_acc is read and cleared, the gate gradients go out, dc moves on one step.
__device__ __forceinline__ void cell_bwd(const CellK& k, const LstmBwdP& p, int t, int b, int u, float* dc) {
  const int H = p.H;
  float4* dhp = reinterpret_cast<float4*>(p.dh_acc + (int64_t)b * H + u);
  const float4 h0 = __ldcg(dhp), h1 = __ldcg(dhp + 1);
  const float dhv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
  float gi[8], gf[8], gg[8], go[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float dh = k.dy[j] + dhv[j];
    const float dcj = dh * k.dc[j] + dc[j];
    dc[j] = dcj * k.f[j];
    gi[j] = dcj * k.ki[j];
    gf[j] = dcj * k.kf[j];
    gg[j] = dcj * k.kg[j];
    go[j] = dh * k.ko[j];
  }
  __nv_bfloat16* gp = p.dgates + ((int64_t)t * p.Bt + p.b0 + b) * 4 * H + u;
  *reinterpret_cast<uint4*>(gp) = pack8(gi);
  *reinterpret_cast<uint4*>(gp + H) = pack8(gf);
  *reinterpret_cast<uint4*>(gp + 2 * (int64_t)H) = pack8(gg);
  *reinterpret_cast<uint4*>(gp + 3 * (int64_t)H) = pack8(go);
  dhp[0] = make_float4(0.f, 0.f, 0.f, 0.f);
  dhp[1] = make_float4(0.f, 0.f, 0.f, 0.f);
}


// AND of a flag over the 128 epilogue threads (named barrier 2)
__device__ __forceinline__ bool all_epilogue(bool ok) {
  unsigned int r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %1, 0;\nbar.red.and.pred p, 2, 128, q;\nselp.u32 %0, 1, 0, p;\n}"
               : "=r"(r) : "r"((unsigned int)ok) : "memory");
  return r != 0;
}

// UV: groups of eight units that a thread owns (H / G / 8).  It owns the same ones of the same row in every step, so
// dc stays in registers.  At UV = 2 (H = 1024) a step's activations are loaded during the previous step's contraction
// and turned into factors before the wait for dh, which leaves two loads and a few multiplications on the chain.
template <int UV>
__global__ void __launch_bounds__(kBwdThreads, 1)
lstm_bwd_persistent_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_w,
                           const LstmBwdP p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kBwdMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kBwdMaxStages];
  __shared__ __align__(8) uint64_t w_bar;
  __shared__ __align__(8) uint64_t acc_bar;
  __shared__ uint32_t tmem_base_holder;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_w = smem0;                       // 8 K-blocks x 2 atoms x 8 KiB
  const uint32_t smem_a = smem0 + kBwdWBytes;          // S stages
  const int S = p.num_stages;
  const int ns = blockIdx.x % p.NS, ks = blockIdx.x / p.NS;
  constexpr int kKb = kBwdK / kBlockK;                 // 8 K-blocks per step

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&w_bar), 1);
    mbar_init(smem_u32(&acc_bar), kBwdIssuers);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_holder)), "r"((uint32_t)(kBwdIssuers * kBwdN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = tmem_base_holder;

  // step index i = T-1-t; arrivals: after A_i the counter reaches G*(2i+1), after B_i G*(2i+2)
  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(smem_u32(&w_bar), kBwdWBytes);
      for (int kb = 0; kb < kKb; ++kb)
        for (int j = 0; j < 2; ++j)
          tma_load_2d(smem_w + (uint32_t)(kb * 2 + j) * kAtomBytes, &map_w, smem_u32(&w_bar), ns * kBwdN + j * 64,
                      ks * kBwdK + kb * kBlockK);
      uint32_t it = 0;
      bool ok = true;
      for (int i = 0; i + 1 < p.T && ok; ++i) {
        const int t = p.T - 1 - i;
        if (!wait_counter(p.counter, (unsigned int)p.G * (unsigned int)(2 * i + 1), p.err, 5)) break;
        asm volatile("fence.proxy.async;" ::: "memory");
        for (int kb = 0; kb < kKb; ++kb, ++it) {
          const int s = (int)(it % (uint32_t)S);
          const uint32_t ph = (it / (uint32_t)S) & 1u;
          if (!wait_bar(smem_u32(&empty_bar[s]), ph ^ 1u, p.err, 1)) { ok = false; break; }
          const uint32_t fb = smem_u32(&full_bar[s]);
          mbar_expect_tx(fb, p.stage_bytes);
          tma_load_2d(smem_a + (uint32_t)s * p.stage_bytes, &map_g, fb, ks * kBwdK + kb * kBlockK, t * p.Bt + p.b0);
        }
      }
    }
  } else if (warp == 1 || warp > 5) {
    const int me = warp == 1 ? 0 : warp - 5;
    {
      bool ok = wait_bar_warp(smem_u32(&w_bar), 0, p.err, 6);
      // lean issue loop: see the forward kernel
      const uint64_t da0 = make_desc(smem_a, 0), db0 = make_desc(smem_w, 1);
      const uint32_t a_hi = (uint32_t)(da0 >> 32), b_hi = (uint32_t)(db0 >> 32);
      const uint32_t a_lo0 = (uint32_t)da0, b_lo0 = (uint32_t)db0;
      const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
      const uint32_t idesc = p.idesc, acc = tmem_acc + (uint32_t)(me * kBwdN), a_step = p.stage_bytes >> 4;
      for (int i = 0; i + 1 < p.T && ok; ++i) {
        const uint32_t it0 = (uint32_t)(i * kKb + me);
        uint32_t s = it0 % (uint32_t)S, ph = (it0 / (uint32_t)S) & 1u;
        for (int kb = me; kb < kKb; kb += kBwdIssuers) {
          if (!wait_bar_warp(full0 + 8u * s, ph, p.err, 2)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_lo = a_lo0 + s * a_step, b_lo = b_lo0 + (uint32_t)kb * ((2u * kAtomBytes) >> 4);
          if (kb == me) umma_lo_elect<1, 0>(acc, a_lo, a_hi, b_lo, b_hi, idesc, 0u);
          else umma_lo_elect<1, 1>(acc, a_lo, a_hi, b_lo, b_hi, idesc, 1u);
#pragma unroll
          for (int kk = 1; kk < kBlockK / 16; ++kk)
            umma_lo_elect<1, 1>(acc, a_lo + kk * 2, a_hi, b_lo + kk * 128, b_hi, idesc, 1u);
          umma_commit_elect(empty0 + 8u * s);
          s += (uint32_t)kBwdIssuers;
          if (s >= (uint32_t)S) { s -= (uint32_t)S; ph ^= 1u; }
        }
        if (ok) umma_commit_elect(smem_u32(&acc_bar));
      }
    }
  } else {
    const int lg = warp & 3;
    const int b = lg * 32 + lane;
    const bool row = b < p.B;
    const int H = p.H;
    const int ua = blockIdx.x * UV * 8;            // first unit of this CTA's phase-A slice
    bool ok = true;
    float dc[UV][8];
#pragma unroll
    for (int v = 0; v < UV; ++v)
#pragma unroll
      for (int j = 0; j < 8; ++j) dc[v][j] = 0.f;
    CellIn in[2];
    float ct[2][8];                                // cell states of the step at hand
    auto load_ct = [&](float* c, int t, int u) {
      const float4* cq = reinterpret_cast<const float4*>(p.c_all + ((int64_t)t * p.Bt + p.b0 + b) * H + u);
      const float4 c0 = cq[0], c1 = cq[1];
      c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    };
    if (UV == 2 && row) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        load_cell(in[v], p, p.T - 1, b, ua + v * 8);
        load_ct(ct[v], p.T - 1, ua + v * 8);
      }
    }
    for (int i = 0; i < p.T && ok; ++i) {
      const int t = p.T - 1 - i;
      CellK k[2];
      if (UV == 2 && row) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          cell_factors(k[v], in[v], ct[v]);
          const float4 q0 = in[v].q0, q1 = in[v].q1;
          ct[v][0] = q0.x; ct[v][1] = q0.y; ct[v][2] = q0.z; ct[v][3] = q0.w;
          ct[v][4] = q1.x; ct[v][5] = q1.y; ct[v][6] = q1.z; ct[v][7] = q1.w;
        }
      }
      // ---- phase A(t): needs every CTA's B(t+1) contribution to dh_acc
      if (i > 0) {
        bool mine = true;
        if (warp == 2 && lane == 0) mine = wait_counter(p.counter, (unsigned int)p.G * (unsigned int)(2 * i), p.err, 7);
        ok = all_epilogue(mine);
        if (!ok) break;
      }
      if (row) {
#pragma unroll
        for (int v = 0; v < UV; ++v) {
          const int u = ua + v * 8;
          if (UV > 2) {
            load_cell(in[0], p, t, b, u);
            load_ct(ct[0], t, u);
            cell_factors(k[0], in[0], ct[0]);
          }
          cell_bwd(k[UV == 2 ? v : 0], p, t, b, u, dc[v]);
        }
      }
      publish_step(p.counter, warp == 2 && lane == 0);
      if (t == 0) break;
      if (UV == 2 && row) {                        // in flight during the contraction
#pragma unroll
        for (int v = 0; v < 2; ++v) load_cell(in[v], p, t - 1, b, ua + v * 8);
      }
      // ---- phase B(t): add this CTA's tile of dgates[t] . W_hh to dh_acc
      ok = all_epilogue(wait_bar(smem_u32(&acc_bar), (uint32_t)i & 1u, p.err, 3));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int cc = 0; cc < kBwdN; cc += 32) {
        uint32_t r[32], r2[32];
        __syncwarp();
        tmem_ld32(tmem_acc + ((uint32_t)(lg * 32) << 16) + (uint32_t)cc, r);
        tmem_ld32(tmem_acc + ((uint32_t)(lg * 32) << 16) + (uint32_t)(kBwdN + cc), r2);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 32; ++q) r[q] = __float_as_uint(__uint_as_float(r[q]) + __uint_as_float(r2[q]));
        if (row) {
          float* o = p.dh_acc + (int64_t)b * H + ns * kBwdN + cc;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                         ::"l"(o + q * 4), "f"(__uint_as_float(r[q * 4])), "f"(__uint_as_float(r[q * 4 + 1])),
                           "f"(__uint_as_float(r[q * 4 + 2])), "f"(__uint_as_float(r[q * 4 + 3]))
                         : "memory");
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      publish_step(p.counter, warp == 2 && lane == 0);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"((uint32_t)(kBwdIssuers * kBwdN)) : "memory");
  }
}

int g_bwd_state[64][5];   // per device and log2(UV)

std::mutex g_mu;
int g_state[64][2];       // per device and kernel: 0 unknown, 1 usable, -1 not usable

}  // namespace

// Returns PD_OK when the sequence was enqueued, 1 when this path does not apply (the caller then runs the
// per-step path), or an error code.  `counter` must point at 4 bytes of device scratch.
int pd_lstm_fwd_persistent(const void* gx, const void* w_hh, const void* b_hh, int T, int B, int H, void* y, void* act,
                           float* c_all, unsigned int* counter, cudaStream_t s) {
  return pd_lstm_fwd_persistent_rows(gx, w_hh, b_hh, T, B, 0, B, H, y, act, c_all, counter, s);
}

// The same on the batch rows b0 .. b0 + B - 1 of tensors that hold Bt rows per time step.  Two such launches on two
// streams (the halves of a batch) run side by side: with B <= 64 a CTA takes half of an SM's shared memory, so both
// grids are resident at once and each hides the other's waits.
int pd_lstm_fwd_persistent_rows(const void* gx, const void* w_hh, const void* b_hh, int T, int Bt, int b0, int B, int H,
                                void* y, void* act, float* c_all, unsigned int* counter, cudaStream_t s) {
  if (B > 128 || H % kBlockK != 0 || H % kUnits != 0 || T < 2 || b0 < 0 || b0 + B > Bt) return 1;
  const int G = H / kUnits;
  const int kblocks = H / kBlockK;
  const uint32_t w_bytes = (uint32_t)kblocks * kWBlockBytes;
  if (w_bytes > 96u * 1024u) return 1;
  // Only the batch's own rows are staged: every CTA reads all of h_{t-1} from L2 each step, which at 128 rows is 33 MB
  // per step and was what a step at any batch waited for.  An MMA still reads 128 rows from a stage's start: rows beyond
  // the batch come from the next stages (behind the last one lies slack) and land in accumulator rows that nobody reads.
  const int rows = (B + 7) & ~7;
  const uint32_t stage_bytes = (uint32_t)rows * kBlockK * 2;
  const bool half = B <= 64 && B < Bt;       // one of several launches that share the GPU
  const uint32_t budget = (half ? 96u : 200u) * 1024u;           // half: two CTAs (105 KiB each at most) per SM
  if (w_bytes + 2 * stage_bytes > budget) return 1;
  int stages = (int)((budget - w_bytes) / stage_bytes);
  if (stages > kMaxStages) stages = kMaxStages;
  const size_t smem = (size_t)w_bytes + (size_t)stages * stage_bytes + (kStageBytes - stage_bytes) + 1024;
  const void* kernel = half ? (const void*)lstm_fwd_persistent_kernel<1> : (const void*)lstm_fwd_persistent_kernel<kFwdIssuers>;
  const int threads = block_threads(half ? 1 : kFwdIssuers);
  int dev = 0;
  PD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return 1;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_state[dev][half] == 0) {
      int coop = 0, per_sm = 0;
      PD_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
      PD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024));
      PD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 216 * 1024));
      g_state[dev][half] = (coop && per_sm >= 1) ? 1 : -1;
    }
    if (g_state[dev][half] < 0) return 1;
  }
  if (G > pd_num_sms()) return 1;

  LstmP p;
  memset(&p, 0, sizeof(p));
  p.T = T; p.B = B; p.H = H; p.G = G; p.num_stages = stages;
  p.parts = kblocks >= 4 ? 4 : (kblocks >= 2 ? 2 : 1);
  p.issuers = half ? 1 : (kblocks < kFwdIssuers ? kblocks : kFwdIssuers);
  if (p.issuers > stages) p.issuers = stages;
  p.Bt = Bt; p.b0 = b0; p.stage_bytes = stage_bytes;
  p.gx = (const __nv_bfloat16*)gx; p.b_hh = (const __nv_bfloat16*)b_hh;
  p.y = (__nv_bfloat16*)y; p.act = (__nv_bfloat16*)act; p.c_all = c_all; p.counter = counter;
  p.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kCols >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  int rc = pd_gemm_error_word(&p.err);
  if (rc != PD_OK) return rc;
  CUtensorMap mh, mw;
  rc = pd_make_map_2d(&mh, y, (int64_t)T * Bt, H, H, kBlockK, rows);
  if (rc != PD_OK) return rc;
  rc = pd_make_map_2d(&mw, w_hh, 4ll * H, H, H, kBlockK, 8);
  if (rc != PD_OK) return rc;
  PD_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s));
  void* args[] = {(void*)&mh, (void*)&mw, (void*)&p};
  PD_CUDA(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)G), dim3((unsigned)threads), args, smem, s));
  return PD_OK;
}

// Backward recurrence as one cooperative kernel; same return convention as pd_lstm_fwd_persistent.
// dh_ws and dc_ws: fp32 [B, H] scratch each (dc_ws holds the grid counter: like all of a call's scratch it is the
// call's own, also where the call has been recorded and is replayed beside others).
int pd_lstm_bwd_persistent(const void* dy, const void* w_hh, const void* act, const float* c_all, int T, int B, int H,
                           void* dgates, float* dh_ws, float* dc_ws, cudaStream_t s) {
  return pd_lstm_bwd_persistent_rows(dy, w_hh, act, c_all, T, B, 0, B, H, dgates, dh_ws, dc_ws, s);
}

// Batch rows b0 .. b0 + B - 1 of tensors with Bt rows per time step (dh_ws, dc_ws: of this launch alone).  The
// grid is (H / 128)^2 CTAs - 64 at H = 1024 - so the halves of a batch, launched on two streams, run side by side.
int pd_lstm_bwd_persistent_rows(const void* dy, const void* w_hh, const void* act, const float* c_all, int T, int Bt,
                                int b0, int B, int H, void* dgates, float* dh_ws, float* dc_ws, cudaStream_t s) {
  if (B > 128 || H < kBwdN || H > 1024 || (H & (H - 1)) != 0 || b0 < 0 || b0 + B > Bt) return 1;
  const int NS = H / kBwdN, KS = 4 * H / kBwdK;
  const int G = NS * KS;
  if (H % G != 0 || (H / G) % 8 != 0 || G > pd_num_sms()) return 1;
  const void* kernel = nullptr;
  int lg = 0;
  switch (H / G / 8) {
    case 2: kernel = (const void*)lstm_bwd_persistent_kernel<2>; lg = 1; break;
    case 4: kernel = (const void*)lstm_bwd_persistent_kernel<4>; lg = 2; break;
    case 8: kernel = (const void*)lstm_bwd_persistent_kernel<8>; lg = 3; break;
    case 16: kernel = (const void*)lstm_bwd_persistent_kernel<16>; lg = 4; break;
    default: return 1;
  }
  const int rows = (B + 7) & ~7;                       // see the forward kernel's launch
  const uint32_t stage_bytes = (uint32_t)rows * kBlockK * 2;
  int stages = (int)(kBwdRing / stage_bytes);
  if (stages > kBwdMaxStages) stages = kBwdMaxStages;
  const size_t smem = (size_t)kBwdWBytes + (size_t)stages * stage_bytes + (kStageBytes - stage_bytes) + 1024;
  int dev = 0;
  PD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return 1;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_bwd_state[dev][lg] == 0) {
      int coop = 0, per_sm = 0;
      PD_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
      PD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024));
      PD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBwdThreads, 208 * 1024));
      g_bwd_state[dev][lg] = (coop && per_sm >= 1) ? 1 : -1;
    }
    if (g_bwd_state[dev][lg] < 0) return 1;
  }
  unsigned int* counter = reinterpret_cast<unsigned int*>(dc_ws);
  LstmBwdP p;
  memset(&p, 0, sizeof(p));
  p.T = T; p.B = B; p.H = H; p.G = G; p.NS = NS; p.num_stages = stages; p.stage_bytes = stage_bytes;
  p.Bt = Bt; p.b0 = b0;
  p.dy = (const __nv_bfloat16*)dy; p.act = (const __nv_bfloat16*)act; p.c_all = c_all;
  p.dgates = (__nv_bfloat16*)dgates; p.dh_acc = dh_ws; p.counter = counter;
  p.idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(kBwdN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  int rc = pd_gemm_error_word(&p.err);
  if (rc != PD_OK) return rc;
  CUtensorMap mg, mw;
  rc = pd_make_map_2d(&mg, dgates, (int64_t)T * Bt, 4ll * H, 4ll * H, kBlockK, rows);
  if (rc != PD_OK) return rc;
  rc = pd_make_map_2d(&mw, w_hh, 4ll * H, H, H, 64, kBlockK);
  if (rc != PD_OK) return rc;
  PD_CUDA(cudaMemsetAsync(dh_ws, 0, (size_t)B * H * sizeof(float), s));
  PD_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s));
  void* args[] = {(void*)&mg, (void*)&mw, (void*)&p};
  PD_CUDA(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)G), dim3(kBwdThreads), args, smem, s));
  return PD_OK;
}
