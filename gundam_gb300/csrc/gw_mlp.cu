// gw_mlp.cu -- the learned surrogate: a BF16 MLP trained and evaluated with
// hand-written tcgen05 kernels (libgw.so, C ABI gwm_* in include/gw.h).
//
// Every GEMM is C[M x N] = A[M x K] * B[N x K]^T with both operands K-major
// (contiguous along K) in BF16 and FP32 accumulation in tensor memory (TMEM):
//   * one CTA (4 or 8 warps) owns a 128 x BN output tile;
//   * the K loop stages 128 x 64 and BN x 64 BF16 tiles in shared memory by TMA
//     with the 128-byte swizzle, in a ring of S stages;
//   * one elected thread issues tcgen05.mma (M = 128, N = BN, K = 16 each) and
//     tcgen05.commit to an mbarrier per stage; every wait on it is bounded;
//   * the epilogue reads the accumulator with tcgen05.ld (a thread: one row) and
//     fuses bias, SiLU, the SiLU derivative of the backward pass, the training
//     loss and its gradient, and row-major / transposed BF16 or FP32 stores;
//   * TMEM is allocated once per CTA and freed on every exit path.
// Forward: z = W x + b, h = silu(z); backward: dX = dY W (with the SiLU
// derivative fused), dW = dY^T X; Adam on FP32 master weights refreshes the
// BF16 weights and their transposes.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cfloat>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "gw.h"
#include "gw_launch.h"

namespace gwm {
namespace {

typedef __nv_bfloat16 bf16;
using gw::dep_launch;
using gw::dep_wait;

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr uint64_t kWaitNs = 1000000000ull;  // 1 s per MMA commit

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > kWaitNs) return false;
  }
}

// ---- tcgen05 primitives ----
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major with the 128-byte swizzle: rows of
// 64 BF16 (128 bytes), 8-row atoms of 1024 bytes (SBO) whose 16-byte chunks
// are XOR-permuted by the row within the atom (the pattern the TMA unit
// writes with CU_TENSOR_MAP_SWIZZLE_128B into 1024-byte-aligned buffers);
// LBO is unused for this layout.  A K step of 16 elements adds 32 bytes.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;             // LBO (unused)
  d |= (uint64_t)(1024 >> 4) << 32;   // SBO
  d |= (uint64_t)1 << 46;             // descriptor version
  d |= (uint64_t)2 << 61;             // layout: 128-byte swizzle
  return d;
}

// Instruction descriptor, kind::f16: D = F32, A = B = BF16, both K-major.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}


__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + __expf(-z)); }

struct Epilogue {
  const float* bias;    // [N] or null
  int act;              // 1: SiLU
  const float* gate;    // [M x N] pre-activations: multiply by silu'(gate) (backward) or null
  float* out_f32;       // [M x N] value before the activation, or null
  bf16* out_bf16;       // [M x N] after the activation, or null
  bf16* out_bf16_t;     // [N x M] after the activation, or null
  int ld_t;             // leading dimension of out_bf16_t (>= M)
  // mean squared error against rows perm[r] (perm null: r) of target [. x N], or
  // null: the BF16 outputs are then its gradient 2 e * inv, e = value - target,
  // and *loss += scale * inv * sum e^2 (one atomic per tile)
  const float* target;
  const int32_t* perm;
  float* loss;
  float inv, scale;
  int b_ready;          // 1: B was written before the launch chain began (weights, outside training)
};

// 2-D tiled TMA load of box {8 elements, R rows} at (k, row) into shared
// memory, completing on an mbarrier (transaction bytes).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int k, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(k), "r"(row), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// A thread's 32 consecutive values of one row of an FP32 matrix (p: the first,
// 16-byte aligned when `vec`); only the first n are read or written.
__device__ __forceinline__ void row_load(const float* p, int n, bool vec, float (&v)[32]) {
  if (vec && n == 32) {
#pragma unroll
    for (int q = 0; q < 32; q += 4) {
      const float4 f = *reinterpret_cast<const float4*>(p + q);
      v[q] = f.x;
      v[q + 1] = f.y;
      v[q + 2] = f.z;
      v[q + 3] = f.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = q < n ? p[q] : 0.f;
  }
}

__device__ __forceinline__ void row_store(float* p, int n, bool vec, const float (&v)[32]) {
  if (vec && n == 32) {
#pragma unroll
    for (int q = 0; q < 32; q += 4) *reinterpret_cast<float4*>(p + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < 32; ++q)
      if (q < n) p[q] = v[q];
  }
}

__device__ __forceinline__ void row_store(bf16* p, int n, bool vec, const bf16 (&v)[32]) {
  if (vec && n == 32) {
#pragma unroll
    for (int q = 0; q < 32; q += 8) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = (uint32_t)__bfloat16_as_ushort(v[q + 2 * i]) | (uint32_t)__bfloat16_as_ushort(v[q + 2 * i + 1]) << 16;
      *reinterpret_cast<uint4*>(p + q) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 32; ++q)
      if (q < n) p[q] = v[q];
  }
}

// Pipelined GEMM tile, C[128 x BN] = A[128 x K] * B[BN x K]^T.
//   * thread 0 (warp 0) issues the TMA loads of each 64-wide K tile into one
//     of S shared-memory stages (one box of 64 K-elements x rows per operand,
//     128-byte swizzle, 1024-byte-aligned stages); rows beyond M / N and
//     columns beyond K arrive as zeros;
//   * thread 32 (warp 1) waits for a stage, issues its four K = 16 MMAs and
//     commits them to the stage's "empty" barrier, which lets the producer
//     refill it; a final commit signals the epilogue;
//   * all NW warps read the accumulator from TMEM, warp w the rows
//     32 (w % 4) .. + 31 and every (NW / 4)-th group of 32 columns, one row per
//     thread, and load and store that row's 32 values as 16-byte vectors (128
//     contiguous bytes per thread and matrix).  The gate or target values of a
//     thread's first columns are loaded before it waits for the accumulator.
//     A warp that went through 32 dependent loads per gate tile and a
//     shared-memory transpose per output bound every backward product: 44 us
//     (M = 2048, N = K = 512, against 17 us without a gate); now 11 us with or
//     without one.
// Every wait is bounded; on a timeout the tile records the failure in
// *status, drains its own copies (bounded) and frees TMEM.
template <int BN, int S, int NW>
__device__ __forceinline__ void gemm_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, int m0, int n0, int M,
                                          int N, int K, const Epilogue& ep, uint32_t* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int kA = kBM * kBK * 2;  // 16 KB
  constexpr int kB = BN * kBK * 2;
  constexpr int kStage = kA + kB;
  constexpr int kGroups = NW / 4;  // column groups of the epilogue
  static_assert(BN % (32 * kGroups) == 0, "every column group has whole 32-column chunks");
  __shared__ __align__(8) uint64_t full[S], empty[S], done;
  __shared__ float sbias[BN];  // the tile's bias columns, read by every row of the epilogue
  __shared__ float sloss[NW];
  __shared__ uint32_t tmem_base;
  __shared__ volatile int failed;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) tmem_alloc(&tmem_base, BN);
  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const int nk = (K + kBK - 1) / kBK;
  int produced = 0;
  // the kernel before this one may still run: until dep_wait only what it does
  // not write is read, the weights' tiles of the first stages when they are
  // known to be ready
  dep_launch();
  const int early = ep.b_ready ? min(nk, S) : 0;
  if (tid == 0) {
    for (int kt = 0; kt < early; ++kt) {
      mbar_arrive_expect(&full[kt], (uint32_t)kStage);
      tma_load_2d(smem + kt * kStage + kA, &tmB, kt * kBK, n0, &full[kt]);
    }
  }
  dep_wait();
  if (ep.bias) {
    // one coalesced load per column instead of one load per element in the
    // epilogue, where the dependent loads stalled the tile's four warps (read
    // after the barrier that follows the accumulator's completion)
    for (int c = tid; c < BN; c += NW * 32) sbias[c] = (n0 + c < N) ? ep.bias[n0 + c] : 0.f;
  }

  if (tid == 0) {
    // producer
    for (int kt = 0; kt < nk; ++kt) {
      const int st = kt % S;
      if (kt >= S && !mbar_wait_bounded(&empty[st], (uint32_t)(((kt / S) - 1) & 1))) {
        failed = 1;
        break;
      }
      if (failed && kt >= early) break;  // a stage whose weights are on the way is completed, so that it can be drained
      unsigned char* a = smem + st * kStage;
      unsigned char* b = a + kA;
      if (kt >= early) {
        mbar_arrive_expect(&full[st], (uint32_t)kStage);
        tma_load_2d(b, &tmB, kt * kBK, n0, &full[st]);
      }
      tma_load_2d(a, &tmA, kt * kBK, m0, &full[st]);
      produced = kt + 1;
    }
  } else if (tid == 32) {
    // MMA issuer
    constexpr uint32_t idesc = instr_desc(kBM, BN);
    int kt = 0;
    for (; kt < nk; ++kt) {
      const int st = kt % S;
      if (!mbar_wait_bounded(&full[st], (uint32_t)((kt / S) & 1))) {
        failed = 1;
        break;
      }
      if (failed) break;
      tc_fence_after();
      const uint32_t a0 = smem_u32(smem + st * kStage), b0 = a0 + kA;
#pragma unroll
      for (int s16 = 0; s16 < kBK / 16; ++s16) {
        const uint64_t ad = smem_desc_sw128(a0 + s16 * 32);
        const uint64_t bd = smem_desc_sw128(b0 + s16 * 32);
        mma_bf16(tmem, ad, bd, idesc, (kt > 0 || s16 > 0) ? 1u : 0u);
      }
      mma_commit(&empty[st]);
    }
    // covers every MMA issued above (or none)
    mma_commit(&done);
  }
  __syncwarp();

  // this thread's row, and the gate / target values of its first columns
  const int r = m0 + (warp & 3) * 32 + lane;
  const bool row_ok = r < M;
  const bool vec = (N & 7) == 0;  // rows of every operand stay 16-byte aligned
  const float* pre_row = nullptr;
  if (row_ok) {
    if (ep.gate) pre_row = ep.gate + (size_t)r * N;
    else if (ep.target) pre_row = ep.target + (size_t)(ep.perm ? ep.perm[r] : r) * N;
  }
  constexpr int kStep = 32 * kGroups;
  const int cfirst = (warp >> 2) * 32;
  float pre[32];
  auto load_pre = [&](int c0) {
    if (pre_row && n0 + c0 < N) row_load(pre_row + n0 + c0, min(32, N - (n0 + c0)), vec, pre);
  };
  load_pre(cfirst);

  const bool ok = mbar_wait_bounded(&done, 0);
  if (!ok) failed = 1;
  __syncthreads();
  if (failed) {
    if (tid == 0) {
      atomicOr(status, 1u);
      // drain the copies this tile issued (bounded) before the block exits
      for (int kt = produced > S ? produced - S : 0; kt < produced; ++kt)
        mbar_wait_bounded(&full[kt % S], (uint32_t)((kt / S) & 1));
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, BN);
    return;
  }
  tc_fence_after();

  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  float e2 = 0.f;
  for (int c0 = cfirst; c0 < BN; c0 += kStep) {
    if (n0 + c0 >= N) break;
    float v[32];
    tmem_ld32(lane_addr + (uint32_t)c0, v);
    if (row_ok) {
      const int ncol = min(32, N - (n0 + c0));
      const size_t o = (size_t)r * N + n0 + c0;
      if (ep.gate) {
#pragma unroll
        for (int q = 0; q < 32; ++q) {
          const float g = pre[q];
          const float sg = sigmoidf_(g);
          v[q] *= sg * (1.f + g * (1.f - sg));
        }
      }
      if (ep.bias) {
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] += sbias[c0 + q];
      }
      if (ep.out_f32) row_store(ep.out_f32 + o, ncol, vec, v);
      if (ep.target) {
#pragma unroll
        for (int q = 0; q < 32; ++q) {
          const float e = v[q] - pre[q];
          if (q < ncol) e2 += e * e;
          v[q] = 2.f * e * ep.inv;
        }
      }
      load_pre(c0 + kStep);
      if (ep.out_bf16 || ep.out_bf16_t) {
        bf16 h[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) h[q] = __float2bfloat16((ep.act == 1) ? v[q] * sigmoidf_(v[q]) : v[q]);
        if (ep.out_bf16) row_store(ep.out_bf16 + o, ncol, vec, h);
        if (ep.out_bf16_t) {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (q < ncol) ep.out_bf16_t[(size_t)(n0 + c0 + q) * ep.ld_t + r] = h[q];
        }
      }
    }
    __syncwarp();
  }
  if (ep.target) {
    for (int o = 16; o; o >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
    if (lane == 0) sloss[warp] = e2;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, BN);
  if (ep.target && tid == 0) {
    float t = 0.f;
    for (int w = 0; w < NW; ++w) t += sloss[w];
    atomicAdd(ep.loss, t * ep.inv * ep.scale);
  }
}

template <int BN, int S, int NW>
__global__ void __launch_bounds__(NW * 32) k_gemm(const __grid_constant__ CUtensorMap tmA,
                                                  const __grid_constant__ CUtensorMap tmB, int M, int N, int K,
                                                  Epilogue ep, uint32_t* status) {
  gemm_tile<BN, S, NW>(tmA, tmB, blockIdx.y * kBM, blockIdx.x * BN, M, N, K, ep, status);
}

// Products of one K that do not depend on one another, in one launch: the tiles
// of product i are the blocks [tile0[i], tile0[i + 1]).  The weight gradients
// are such a set once the output gradients of all layers are there.  One after
// another they left most of the chip idle: of 2048 rows the hidden layers' 512 x
// 512 products are 64 tiles each and the launches took 15 + 15 + 15 + 18 us;
// together they take 17 us.
constexpr int kMaxGroup = 8;
struct GemmGroup {
  CUtensorMap a[kMaxGroup], b[kMaxGroup];
  float* out[kMaxGroup];  // [M x N]
  int M[kMaxGroup], N[kMaxGroup], tile0[kMaxGroup + 1];
  int n, K;
};

template <int BN, int S, int NW>
__global__ void __launch_bounds__(NW * 32) k_gemm_group(const __grid_constant__ GemmGroup g, uint32_t* status) {
  int i = 0;
  while (i + 1 < g.n && (int)blockIdx.x >= g.tile0[i + 1]) ++i;
  const int N = g.N[i], t = blockIdx.x - g.tile0[i], cols = (N + BN - 1) / BN;
  Epilogue ep{};
  ep.out_f32 = g.out[i];
  gemm_tile<BN, S, NW>(g.a[i], g.b[i], t / cols * kBM, t % cols * BN, g.M[i], N, g.K, ep, status);
}

// ---- small kernels ----
// Rows of a row-major FP32 matrix to BF16, row-major and transposed.  Row r
// of the output is row perm[r] of x (perm null: row r).  32 x 32 tiles go
// through shared memory so both stores are coalesced; block (32, 8).
__global__ void k_rows_to_bf16(const float* x, const int32_t* perm, int rows, int cols, bf16* y, bf16* yt, int ld_t) {
  dep_launch();
  dep_wait();
  __shared__ bf16 tile[32][34];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int i = ty; i < 32; i += 8) {
    const int r = r0 + i, c = c0 + tx;
    bf16 v = __float2bfloat16(0.f);
    if (r < rows && c < cols) {
      const size_t src = perm ? (size_t)perm[r] : (size_t)r;
      v = __float2bfloat16(x[src * cols + c]);
      y[(size_t)r * cols + c] = v;
    }
    tile[i][tx] = v;
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int c = c0 + i, r = r0 + tx;
    if (c < cols && r < rows) yt[(size_t)c * ld_t + r] = tile[tx][i];
  }
}

// Bias gradient of one output unit by 16 lanes: the FP32 sum of its BF16 row
// dzt [B].  Lane q adds the elements q, q + 16, ... in order, then the 16 parts
// are added in lane order; the sum on every lane of the half-warp.
__device__ __forceinline__ float bias_grad(const bf16* dzt, int B) {
  const int q = threadIdx.x & 15;
  float s = 0.f;
  int i = q;
  for (; i + 15 * 16 < B; i += 256) {
    bf16 u[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) u[j] = dzt[i + 16 * j];
#pragma unroll
    for (int j = 0; j < 16; ++j) s += __bfloat162float(u[j]);
  }
  for (; i < B; i += 16) s += __bfloat162float(dzt[i]);
  __syncwarp();
  float t = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) t += __shfl_sync(0xffffffffu, s, j, 16);
  return t;
}

// Bias gradients of one layer, a half-warp per unit (gwm_gradients).
__global__ void __launch_bounds__(256) k_bias_grad(const bf16* dzt, int rows, int B, float* out) {
  dep_launch();
  dep_wait();
  const int r = blockIdx.x * 16 + (threadIdx.x >> 4);
  const float g = bias_grad(dzt + (size_t)min(r, rows - 1) * B, B);  // whole warps stay in the shuffles
  if (r < rows && (threadIdx.x & 15) == 0) out[r] = g;
}

__device__ __forceinline__ float adam_value(float w, float g, float& m, float& v, float lr, float c1, float c2) {
  constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  return w - lr * (m / c1) / (sqrtf(v / c2) + eps);
}

constexpr int kMaxLayers = 16;
struct AdamLayer {
  float *w, *m, *v, *b, *mb, *vb;
  const float* g;
  bf16 *wb, *wt;
  const bf16* dzt;  // [rows x batch] output gradients, for the biases (null: biases stay)
  int rows, cols;
  int tile0, bias0;  // first weight tile and first bias block of the layer
};
struct AdamArgs {
  AdamLayer l[kMaxLayers];
  int n_layers, n_tiles, batch;
  float lr, c1, c2;
};

// Adam on the FP32 master weights and biases of every layer in one launch.
// The last n_tiles blocks: 32 x 32 weight tiles, whose BF16 copy and its
// transpose are both stored coalesced (the transpose through shared memory);
// the blocks before them: 16 biases each, whose gradient is formed here from
// the layer's transposed output gradients (chains of loads, so they start first).  A launch per weight and bias array
// with a scattered transpose, and a column-sum launch per layer, took 99 us of a
// 440 us step at 200 -> 512 -> 512 -> 512 -> 3000 and batch 2048; this launch
// takes 22 us (24 with the biases last).  The bound is the 32 bytes per weight that w, g, m, v and the BF16
// copies move (69 MB, mostly from L2).
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ AdamArgs a) {
  dep_launch();
  dep_wait();
  const int tid = threadIdx.x;
  const int n_bias = (int)gridDim.x - a.n_tiles;
  int blk = (int)blockIdx.x - n_bias, li = 0;
  if (blk >= 0) {
    while (li + 1 < a.n_layers && blk >= a.l[li + 1].tile0) ++li;
    const AdamLayer& L = a.l[li];
    const int t = blk - L.tile0, tc = (L.cols + 31) / 32;
    const int r0 = (t / tc) * 32, c0 = (t % tc) * 32;
    const int tx = tid & 31, ty = tid >> 5;
    __shared__ bf16 tile[32][34];
    const int c = c0 + tx;
    float w[4], g[4], m[4], v[4];
    size_t at[4];
    bool in[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = r0 + ty + 8 * j;
      in[j] = r < L.rows && c < L.cols;
      at[j] = (size_t)r * L.cols + c;
      if (in[j]) {
        w[j] = L.w[at[j]];
        g[j] = L.g[at[j]];
        m[j] = L.m[at[j]];
        v[j] = L.v[at[j]];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!in[j]) continue;
      w[j] = adam_value(w[j], g[j], m[j], v[j], a.lr, a.c1, a.c2);
      L.w[at[j]] = w[j];
      L.m[at[j]] = m[j];
      L.v[at[j]] = v[j];
      const bf16 b = __float2bfloat16(w[j]);
      L.wb[at[j]] = b;
      tile[ty + 8 * j][tx] = b;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = c0 + ty + 8 * j, r = r0 + tx;
      if (cc < L.cols && r < L.rows) L.wt[(size_t)cc * L.rows + r] = tile[tx][ty + 8 * j];
    }
    return;
  }
  blk = blockIdx.x;
  while (li + 1 < a.n_layers && blk >= a.l[li + 1].bias0) ++li;
  const AdamLayer& L = a.l[li];
  const int r = (blk - L.bias0) * 16 + (tid >> 4);
  const float g = bias_grad(L.dzt + (size_t)min(r, L.rows - 1) * a.batch, a.batch);
  if (r < L.rows && (tid & 15) == 0) {
    float m = L.mb[r], v = L.vb[r];
    L.b[r] = adam_value(L.b[r], g, m, v, a.lr, a.c1, a.c2);
    L.mb[r] = m;
    L.vb[r] = v;
  }
}

// Standardised inputs: x = (theta - mean) / scale, FP32, and (h0 set) the BF16
// rows of the first GEMM.
__global__ void k_standardize(const double* __restrict__ theta, int rows, int cols, const float* __restrict__ mean,
                              const float* __restrict__ scale, float* x, bf16* h0) {
  dep_launch();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)rows * cols) return;
  const int c = (int)(i % cols);
  const float z = (float)((theta[i] - (double)mean[c]) / (double)scale[c]);
  x[i] = z;
  if (h0) h0[i] = __float2bfloat16(z);
}

// Surrogate head (device pointers).  The predicted log rate of a bin is
//   base(x) + mu + sd * mlp(x)
// with x the standardised parameters and base either affine (nodes == 0:
// b0 + sum_k x_k tab[k][bin]) or additive piecewise-linear (nodes >= 2:
// b0 + sum_k interp_k(x_k), interp_k linear between `nodes` equally spaced
// values tab[k][0..nodes-1][bin] over x_k in [-lim, lim], constant outside).
// Sum w^2 is modelled as exp(r_b + sum_k x_k r_w[k][bin]) * rate (r_w optional).
struct Head {
  int din, nb, nodes;
  float lim;
  const float* tab;
  const float* b0;
  const float* mu;
  const float* sd;
  const float* r_w;
  const float* r_b;
};

__device__ __forceinline__ float head_base(const Head& h, const float* __restrict__ x, int bin) {
  float acc = h.b0[bin];
  if (h.nodes >= 2) {
    const float inv_w = (float)(h.nodes - 1) / (2.f * h.lim);
    for (int k = 0; k < h.din; ++k) {
      const float xc = fminf(fmaxf(x[k], -h.lim), h.lim);
      const float u = (xc + h.lim) * inv_w;
      const int i = min((int)u, h.nodes - 2);
      const float t = u - (float)i;
      const float* T = h.tab + ((size_t)k * h.nodes + i) * h.nb + bin;
      acc += fmaf(t, T[h.nb] - T[0], T[0]);
    }
  } else {
    for (int k = 0; k < h.din; ++k) acc = fmaf(x[k], h.tab[(size_t)k * h.nb + bin], acc);
  }
  return acc;
}


// log(data / mc) for data, mc > 0: log1p((data - mc) / mc) near 1, where
// log(data) - log(mc) would cancel in FP32, and the difference of logs away
// from it, where the ratio itself can underflow or overflow.
__device__ __forceinline__ float log_ratio_f(float data, float mc) {
  const float r = (data - mc) / mc;
  return fabsf(r) < 0.5f ? log1pf(r) : logf(data) - logf(mc);
}

// Per-bin likelihood term of the surrogate in FP32 (stage 1 only; the exact
// engine keeps its FP64 path).  Same formulas as the engine's FP64 ones:
// Poisson (PoissonLogLikelihood.h:19-53) and Barlow-Beeston OA2021
// (BarlowBeestonBanff2022.h:150-294), with log(data / mc) from log_ratio_f.
// The one sum of two products that the compiler could fuse either way is fused
// explicitly, so that every kernel gives a point the same value.
__device__ __forceinline__ float llh_term_f(int type, float data, float pred, float sumw2) {
  if (type == GW_LLH_POISSON) {
    if (pred <= 0.f) return INFINITY;
    if (data <= 0.f) return 2.f * pred;
    return 2.f * ((pred - data) + data * log_ratio_f(data, pred));
  }
  if (type != GW_LLH_BARLOW_BEESTON_OA2021) return 0.f;
  if (pred <= -1.f) return (pred <= 0.f && data > 0.f) ? INFINITY : 0.f;
  float newmc = pred, penalty = 0.f;
  if (sumw2 > 0.f) {
    const float f2 = sumw2 / (pred * pred);
    const float temp = sumw2 / pred - 1.f;
    const float temp2 = __fmaf_rn(__fmul_rn(4.f, data), f2, __fmul_rn(temp, temp));
    if (temp2 < 0.f) return INFINITY;
    const float beta = 0.5f * (sqrtf(temp2) - temp);
    newmc = fmaxf(pred * beta, FLT_MIN);
    penalty = (beta - 1.f) * (beta - 1.f) / (2.f * f2);
  }
  newmc = fmaxf(newmc, FLT_MIN);
  float stat;
  if (data <= FLT_EPSILON) stat = newmc;
  else stat = (newmc - data) + data * log_ratio_f(data, newmc);
  return 2.f * stat + 2.f * penalty;
}

// Derivatives of the FP32 per-bin term with respect to log(rate) and to
// log(sum w^2):
//   Poisson: dL/dlog mu = 2 (mu - n), dL/dlog s2 = 0;
//   Barlow-Beeston OA2021: beta minimises the bin's joint likelihood (its
//   quadratic is the stationarity condition), so by the envelope theorem the
//   derivatives are the partials at fixed beta of
//   L = 2 (beta mu - n + n log(n / (beta mu))) + (beta - 1)^2 mu^2 / s2:
//     dL/dlog mu = 2 (beta mu - n) + 2 (beta - 1)^2 / f2,
//     dL/dlog s2 = -(beta - 1)^2 / f2,  f2 = s2 / mu^2.
__device__ __forceinline__ void llh_term_grad_f(int type, float data, float pred, float sumw2, float& gmu,
                                                float& gs2) {
  gmu = 0.f;
  gs2 = 0.f;
  if (type == GW_LLH_POISSON) {
    if (pred > 0.f) gmu = 2.f * (pred - data);
    return;
  }
  if (type != GW_LLH_BARLOW_BEESTON_OA2021 || !(pred > 0.f)) return;
  if (sumw2 > 0.f) {
    const float f2 = sumw2 / (pred * pred);
    const float temp = sumw2 / pred - 1.f;
    const float temp2 = __fmaf_rn(temp, temp, __fmul_rn(__fmul_rn(4.f, data), f2));
    if (temp2 < 0.f) return;
    const float beta = 0.5f * (sqrtf(temp2) - temp);
    const float pen = (beta - 1.f) * (beta - 1.f) / f2;
    gmu = 2.f * (beta * pred - data) + 2.f * pen;
    gs2 = -pen;
  } else {
    gmu = 2.f * (pred - data);
  }
}

// Where the head's results go.  sums, sums2 (FP64) and logr are optional.  With
// G set (value and gradient): per (point, bin), G = dL/dlog mu + dL/dlog s2
// (the derivative with respect to the log rate, the modelled sum of w^2 moving
// with it), S = dL/dlog s2, and dY = G * sd (the derivative with respect to the
// network output) as BF16.
struct HeadOut {
  double *part, *sums, *sums2, *logr;
  float *G, *S;
  bf16* dy;
};

// The network's output at (point m, bin), loaded before any output is stored.
__device__ __forceinline__ float head_mlp(const Head& h, const float* mlp, int C, int m, int bin) {
  return bin < h.nb && m < C ? mlp[(size_t)m * h.nb + bin] : 0.f;
}

// Likelihood term of one (point m, bin) from the base `acc`, the log ratio `racc`
// and the network's output y, with its optional outputs.
template <bool GRAD>
__device__ __forceinline__ double head_term(const Head& h, float y, int C, int m, int bin,
                                            const double* __restrict__ data, int llh_type, float acc, float racc,
                                            const HeadOut& out) {
  if (bin >= h.nb || m >= C) return 0.0;
  const size_t o = (size_t)m * h.nb + bin;
  const float lr = acc + h.mu[bin] + h.sd[bin] * y;
  const float mu = expf(lr), s2 = expf(lr + racc);
  if (out.sums) out.sums[o] = (double)mu;
  if (out.sums2) out.sums2[o] = (double)s2;
  if (out.logr) out.logr[o] = (double)lr;
  if constexpr (GRAD) {
    float gmu, gs2;
    llh_term_grad_f(llh_type, (float)data[bin], mu, s2, gmu, gs2);
    const float G = gmu + gs2;
    out.G[o] = G;
    out.S[o] = gs2;
    out.dy[o] = __float2bfloat16(G * h.sd[bin]);
  }
  return (double)llh_term_f(llh_type, (float)data[bin], mu, s2);
}

// The warp's sum of t by a fixed shuffle tree, into part[m][blockIdx.x] (FP64).
__device__ __forceinline__ void head_part(double t, int C, int m, double* part) {
  for (int off = 16; off; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
  if ((threadIdx.x & 31) == 0 && m < C) part[(size_t)m * gridDim.x + blockIdx.x] = t;
}

// Head and likelihood terms, fused, for a base of few nodes: block of 128
// threads, 64 bins (a lane: two neighbours, in packed FP32) x 8 points (warp v
// the points v and v + 4).  The parameters go by in chunks of kHeadK: one TMA
// box brings the chunk's table rows (every node) and one its r_w rows into a
// ring of kHeadStages stages (zeros beyond the bins and the parameters); 64
// threads form the interval and weight of each point and parameter one chunk
// ahead.  A (point, parameter) step of 64 bins is then three shared-memory loads
// (five wavefronts, which is what bounds it) and four packed operations.  Reading the table from L1 / L2 in the loop made
// it a chain of L2 latencies: 67 us for 64 points, 200 parameters and 3000 bins.
// Staging through registers (32 bins per warp) took 51 us, 27 instructions per
// step of 32 bins, issue 62 %; this form takes 31 us (256-thread blocks of 16
// points: 40 us, two of 188 blocks on 36 of the SMs).
// The base is summed over the parameters in order, as k_head_llh does.
constexpr int kHeadK = 8;       // parameters per chunk (network widths are multiples of 8)
constexpr int kHeadNodes = 8;   // nodes a chunk has room for
constexpr int kHeadStages = 3;
constexpr int kHeadBins = 64, kHeadPts = 8, kHeadThreads = 128;
constexpr int kHeadStage = kHeadK * (kHeadNodes + 1) * kHeadBins;  // floats

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(f32x2 r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

template <bool GRAD>
__global__ void __launch_bounds__(kHeadThreads, 3) k_head_staged(const __grid_constant__ CUtensorMap tm_tab,
                                                        const __grid_constant__ CUtensorMap tm_rw, Head h,
                                                        const float* x, const float* mlp, int C,
                                                        const double* __restrict__ data, int llh_type, HeadOut out,
                                                        uint32_t* status) {
  dep_launch();
  extern __shared__ __align__(128) float sh_h[];  // [kHeadStages][kHeadStage]
  __shared__ float4 s_pt[2][kHeadK][kHeadPts];  // (weight, input, staged row of the interval * kHeadBins, 0)
  __shared__ __align__(8) uint64_t bar[kHeadStages];
  const int din = h.din, nb = h.nb, nodes = h.nodes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mb = blockIdx.y * kHeadPts, b0 = blockIdx.x * kHeadBins;
  const float inv_w = (float)(nodes - 1) / (2.f * h.lim);
  const int nchunk = din / kHeadK;
  const bool has_rw = h.r_w != nullptr;
  const uint32_t bytes = (uint32_t)(kHeadK * nodes + (has_rw ? kHeadK : 0)) * kHeadBins * 4u;
  auto issue = [&](int c) {
    float* st = sh_h + (c % kHeadStages) * kHeadStage;
    mbar_arrive_expect(&bar[c % kHeadStages], bytes);
    tma_load_2d(st, &tm_tab, b0, c * kHeadK * nodes, &bar[c % kHeadStages]);
    if (has_rw) tma_load_2d(st + kHeadK * kHeadNodes * kHeadBins, &tm_rw, b0, c * kHeadK, &bar[c % kHeadStages]);
  };
  if (tid == 0) {
    for (int i = 0; i < kHeadStages; ++i) mbar_init(&bar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int c = 0; c < min(nchunk, kHeadStages); ++c) issue(c);  // the tables: constant
  }
  dep_wait();
  // one (parameter, point) of each chunk per thread of the first two warps
  const int sk = tid / kHeadPts, sm = tid % kHeadPts;
  float z = 0.f;
  auto fetch = [&](int c) {
    if (sk < kHeadK) {
      const int k = c * kHeadK + sk;
      z = mb + sm < C ? x[(size_t)(mb + sm) * din + k] : 0.f;
    }
  };
  auto store = [&](int buf) {
    if (sk < kHeadK) {
      const float xc = fminf(fmaxf(z, -h.lim), h.lim);
      const float u = (xc + h.lim) * inv_w;
      const int i = min((int)u, nodes - 2);
      const float t = u - (float)i;
      s_pt[buf][sk][sm] = make_float4(t, z, __int_as_float((sk * nodes + i) * kHeadBins), 0.f);
    }
  };
  const int bin = b0 + 2 * lane;
  f32x2 acc[2], racc[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    acc[j] = pk2(bin < nb ? h.b0[bin] : 0.f, bin + 1 < nb ? h.b0[bin + 1] : 0.f);
    racc[j] = pk2(bin < nb ? h.r_b[bin] : 0.f, bin + 1 < nb ? h.r_b[bin + 1] : 0.f);
  }
  fetch(0);
  store(0);
  if (nchunk > 1) fetch(1);
  __syncthreads();
  for (int c = 0; c < nchunk; ++c) {
    const int buf = c & 1, st = c % kHeadStages;
    const bool ok = mbar_wait_bounded(&bar[st], (uint32_t)((c / kHeadStages) & 1));
    if (c + 1 < nchunk) store(buf ^ 1);  // its readers passed the barrier at the end of chunk c - 1
    if (c + 2 < nchunk) fetch(c + 2);
    const float* tab = sh_h + st * kHeadStage + 2 * lane;
    if (ok) {
      auto step = [&](int kk) {
        const f32x2 w = has_rw ? *reinterpret_cast<const f32x2*>(tab + (kHeadK * kHeadNodes + kk) * kHeadBins) : 0ull;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 pt = s_pt[buf][kk][warp + 4 * j];
          const float* row = tab + __float_as_int(pt.z);
          const f32x2 lo = *reinterpret_cast<const f32x2*>(row);
          const f32x2 hi = *reinterpret_cast<const f32x2*>(row + kHeadBins);
          acc[j] = add2(acc[j], fma2(pk2(pt.x, pt.x), sub2(hi, lo), lo));
          racc[j] = fma2(pk2(pt.y, pt.y), w, racc[j]);
        }
      };
#pragma unroll
      for (int kk = 0; kk < kHeadK; ++kk) step(kk);  // din is a multiple of kHeadK (gwm_create)
    }
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicOr(status, 1u);
        // the copies still in flight land before the block exits (bounded)
        for (int i = c; i < min(nchunk, c + kHeadStages); ++i)
          mbar_wait_bounded(&bar[i % kHeadStages], (uint32_t)((i / kHeadStages) & 1));
      }
      return;
    }
    if (tid == 0 && c + kHeadStages < nchunk) issue(c + kHeadStages);
  }
  float y[2][2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) y[j][i] = head_mlp(h, mlp, C, mb + warp + 4 * j, bin + i);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    float a0, a1, r0, r1;
    upk2(acc[j], a0, a1);
    upk2(racc[j], r0, r1);
    const int m = mb + warp + 4 * j;
    const double t0 = head_term<GRAD>(h, y[j][0], C, m, bin, data, llh_type, a0, r0, out);
    const double t1 = head_term<GRAD>(h, y[j][1], C, m, bin + 1, data, llh_type, a1, r1, out);
    head_part(t0 + t1, C, m, out.part);
  }
}

// The same for an affine base or one of more nodes than k_head_staged holds.
// Block (32 bins, 8 point rows); thread (x, y) of block (bx, by) handles bin
// 32 bx + x and the PPT points by * 8 PPT + y + 8 j.  The block first stages,
// for each of its points and parameters, the input x and (additive base) the
// table offset of the interpolation interval and its weight in shared memory;
// the inner loop is then two coalesced table loads and two FMAs per point and
// parameter, with the table lines of a bin shared through L1 across the
// block's points.  Four parameters' loads are issued before the first is used:
// left to the compiler, the form without gradients came to 40 registers, fewer
// loads in flight and a sixth block per SM that took the L1 from the others (200
// parameters, 16 nodes, 3000 bins, 2048 points: a call 1312 us, 1077 with 48
// registers, 998 now; 64 points 164 -> 130).
template <int PPT, bool GRAD>
__global__ void __launch_bounds__(256) k_head_llh(Head h, const float* x, const float* mlp, int C,
                                                  const double* __restrict__ data, int llh_type, HeadOut out) {
  dep_launch();
  dep_wait();
  extern __shared__ unsigned char sh_raw[];
  constexpr int NP = 8 * PPT;  // points per block
  const int din = h.din;
  float* s_z = reinterpret_cast<float*>(sh_raw);          // [NP][din]
  float* s_t = s_z + NP * din;                            // [NP][din]
  int* s_off = reinterpret_cast<int*>(s_t + NP * din);    // [NP][din]
  const int mb = blockIdx.y * NP;
  const int tid = threadIdx.y * 32 + threadIdx.x;
  const bool additive = h.nodes >= 2;
  const float inv_w = additive ? (float)(h.nodes - 1) / (2.f * h.lim) : 0.f;
  const float* xb = x + (size_t)mb * din;
  const int rows = min(C - mb, NP) * din;
  for (int e0 = tid; e0 < NP * din; e0 += 4 * 256) {
    float z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) z[q] = e0 + q * 256 < rows ? xb[e0 + q * 256] : 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = e0 + q * 256, k = e % din;
      if (e >= NP * din) break;
      s_z[e] = z[q];
      if (additive) {
        const float xc = fminf(fmaxf(z[q], -h.lim), h.lim);
        const float u = (xc + h.lim) * inv_w;
        const int i = min((int)u, h.nodes - 2);
        s_t[e] = u - (float)i;
        s_off[e] = (k * h.nodes + i) * h.nb;
      } else {
        s_t[e] = z[q];
        s_off[e] = k * h.nb;
      }
    }
  }
  __syncthreads();
  const int bin = blockIdx.x * 32 + threadIdx.x;
  const bool bin_ok = bin < h.nb;
  float acc[PPT], racc[PPT];
#pragma unroll
  for (int j = 0; j < PPT; ++j) {
    acc[j] = bin_ok ? h.b0[bin] : 0.f;
    racc[j] = bin_ok ? h.r_b[bin] : 0.f;
  }
  if (bin_ok) {
    const float* __restrict__ tab = h.tab + bin;
    const float* __restrict__ rw = h.r_w ? h.r_w + bin : nullptr;
    const int nb = h.nb;
    // four parameters' table rows on the way at a time (din is a multiple of 8)
    constexpr int U = 4;
    for (int k = 0; k < din; k += U) {
      float w[U], lo[U][PPT], hi[U][PPT];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        w[u] = rw ? __ldg(rw + (size_t)(k + u) * nb) : 0.f;
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
          const int off = s_off[(threadIdx.y + 8 * j) * din + k + u];
          lo[u][j] = __ldg(tab + off);
          hi[u][j] = additive ? __ldg(tab + off + nb) : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
          const int e = (threadIdx.y + 8 * j) * din + k + u;
          const float t = s_t[e];
          if (additive) acc[j] += fmaf(t, hi[u][j] - lo[u][j], lo[u][j]);
          else acc[j] = fmaf(t, lo[u][j], acc[j]);
          racc[j] = fmaf(s_z[e], w[u], racc[j]);
        }
    }
  }
  float y[PPT];
#pragma unroll
  for (int j = 0; j < PPT; ++j) y[j] = head_mlp(h, mlp, C, mb + threadIdx.y + 8 * j, bin);
#pragma unroll
  for (int j = 0; j < PPT; ++j) {
    const int m = mb + threadIdx.y + 8 * j;
    head_part(head_term<GRAD>(h, y[j], C, m, bin, data, llh_type, acc[j], racc[j], out), C, m, out.part);
  }
}

// llh[m] = sum over blocks of part[m][*], one warp per point, fixed order.
__global__ void k_llh_finish(const double* part, int nblk, int C, double* llh) {
  dep_launch();
  dep_wait();
  const int m = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (m >= C) return;
  double s = 0.0;
  for (int b = lane; b < nblk; b += 32) s += part[(size_t)m * nblk + b];
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) llh[m] = s;
}

// Gradient of the likelihood through the base and the sum-of-w^2 model, for
// point m = blockIdx.x and parameters k = blockIdx.y * 8 + (0..7):
//   gz[m][k] = sum_b G[m][b] * d base_b / d x_k + S[m][b] * r_w[k][b]
// (d base / d x_k: the slope of the interpolation interval of x_k, zero
// outside [-lim, lim]; affine base: tab[k][b]).  The point's G and S rows are
// staged in shared memory; fixed-order block reduction: the 8 warps' parts of a
// (point, parameter) go to gz[m][k][0..7], which k_grad_finish adds in order.
// The general form, for an affine base or one of more nodes than
// k_base_grad_staged holds.
__global__ void __launch_bounds__(256) k_base_grad(Head h, const float* x, const float* G, const float* S, float* gz) {
  dep_launch();
  dep_wait();
  extern __shared__ float shg[];
  float* g = shg;            // [nb]
  float* sg = shg + h.nb;    // [nb]
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float *Gm = G + (size_t)m * h.nb, *Sm = S + (size_t)m * h.nb;
  for (int b0 = tid; b0 < h.nb; b0 += 4 * 256) {  // four of each on the way
    float vg[4], vs[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int b = min(b0 + q * 256, h.nb - 1);
      vg[q] = Gm[b];
      vs[q] = Sm[b];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (b0 + q * 256 < h.nb) {
        g[b0 + q * 256] = vg[q];
        sg[b0 + q * 256] = vs[q];
      }
  }
  __syncthreads();
  const bool additive = h.nodes >= 2;
  const float inv_w = additive ? (float)(h.nodes - 1) / (2.f * h.lim) : 0.f;
  for (int q = 0; q < 8; ++q) {
    const int k = blockIdx.y * 8 + q;
    if (k >= h.din) break;
    const float z = x[(size_t)m * h.din + k];
    const float* lo;
    float scale_ = 1.f;
    if (additive) {
      const float xc = fminf(fmaxf(z, -h.lim), h.lim);
      const float u = (xc + h.lim) * inv_w;
      const int i = min((int)u, h.nodes - 2);
      lo = h.tab + ((size_t)k * h.nodes + i) * h.nb;
      scale_ = (z > -h.lim && z < h.lim) ? inv_w : 0.f;
    } else {
      lo = h.tab + (size_t)k * h.nb;
    }
    const float* rw = h.r_w ? h.r_w + (size_t)k * h.nb : nullptr;
    float acc = 0.f;
    for (int b = tid; b < h.nb; b += 256) {
      const float slope = additive ? (lo[b + h.nb] - lo[b]) * scale_ : lo[b];
      acc = fmaf(g[b], slope, acc);
      if (rw) acc = fmaf(sg[b], rw[b], acc);
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) gz[((size_t)m * h.din + k) * 8 + warp] = acc;
  }
}

// The same for a base of few nodes, all points of a tile sharing the table.
// Block (w, bk): the bins 32 w + lane + 256 j (j = 0, 1, ...), those of warp w
// of k_base_grad, and the parameters [bk, bk + 1) * kGradK; warp v the points
// 8 v .. 8 v + 7 of each 64-point tile.  Per j, one TMA box brings the kGradK * nodes
// table rows of the 32 bins and one the r_w rows (zeros beyond the bins and the
// parameters), kGradStages j ahead, so that the table is read once per 64 points
// instead of twice per (point, parameter), and no load of it is waited for:
// 64 points, 200 parameters and 3000 bins took 108 us, bound by the latency of
// the 460 MB that went through L2; this form takes 33 us (39 us with
// kGradK = 4).  Each lane's sum over j and the shuffle tree
// are those of k_base_grad.
constexpr int kGradK = 8, kGradM = 8, kGradStages = 8;
constexpr int kGradRows = kGradK * kHeadNodes;
__global__ void __launch_bounds__(256, 2) k_base_grad_staged(const __grid_constant__ CUtensorMap tm_tab,
                                                             const __grid_constant__ CUtensorMap tm_rw, Head h,
                                                             const float* x, const float* G, const float* S, int C,
                                                             float* gz, uint32_t* status) {
  dep_launch();
  extern __shared__ __align__(128) float sh_g[];  // [kGradStages][kGradRows + kGradK][32]
  constexpr int kStage = (kGradRows + kGradK) * 32;
  __shared__ int2 s_iv[kGradK][8 * kGradM];  // (staged row of the interval * 32, slope scale)
  __shared__ __align__(8) uint64_t bar[kGradStages];
  const int w = blockIdx.x, k0 = blockIdx.y * kGradK, m0 = blockIdx.z * 8 * kGradM;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = h.nb, nodes = h.nodes;
  const int b0 = 32 * w;
  const int nj = b0 < nb ? (nb - b0 + 255) / 256 : 0;
  const bool has_rw = h.r_w != nullptr;
  const uint32_t bytes = (uint32_t)(kGradK * nodes + (has_rw ? kGradK : 0)) * 128u;
  auto issue = [&](int j) {
    float* st = sh_g + (j % kGradStages) * kStage;
    mbar_arrive_expect(&bar[j % kGradStages], bytes);
    tma_load_2d(st, &tm_tab, b0 + 256 * j, k0 * nodes, &bar[j % kGradStages]);
    if (has_rw) tma_load_2d(st + kGradRows * 32, &tm_rw, b0 + 256 * j, k0, &bar[j % kGradStages]);
  };
  if (tid == 0) {
    for (int i = 0; i < kGradStages; ++i) mbar_init(&bar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int j = 0; j < min(nj, kGradStages); ++j) issue(j);  // the tables: constant
  }
  dep_wait();
  const float inv_w = (float)(nodes - 1) / (2.f * h.lim);
  for (int e = tid; e < kGradK * 8 * kGradM; e += 256) {
    const int q = e / (8 * kGradM), mm = e % (8 * kGradM);
    const int k = min(k0 + q, h.din - 1), m = min(m0 + mm, C - 1);
    const float z = x[(size_t)m * h.din + k];
    const float xc = fminf(fmaxf(z, -h.lim), h.lim);
    const float u = (xc + h.lim) * inv_w;
    const int i = min((int)u, nodes - 2);
    s_iv[q][mm] = make_int2((q * nodes + i) * 32, __float_as_int((z > -h.lim && z < h.lim) ? inv_w : 0.f));
  }
  float acc[kGradK][kGradM];
#pragma unroll
  for (int q = 0; q < kGradK; ++q)
#pragma unroll
    for (int j = 0; j < kGradM; ++j) acc[q][j] = 0.f;
  const int mw = m0 + warp * kGradM;  // this warp's first point
  float g[kGradM], sg[kGradM];
  auto load_gs = [&](int j) {
    const int b = b0 + 256 * j + lane;
#pragma unroll
    for (int i = 0; i < kGradM; ++i) {
      const bool in = b < nb && mw + i < C;
      const size_t o = (size_t)(mw + i) * nb + b;
      g[i] = in ? G[o] : 0.f;
      sg[i] = in ? S[o] : 0.f;
    }
  };
  if (nj > 0) load_gs(0);
  bool failed = false;
  __syncthreads();
  for (int j = 0; j < nj; ++j) {
    const int st = j % kGradStages;
    const bool ok = mbar_wait_bounded(&bar[st], (uint32_t)((j / kGradStages) & 1));
    if (__syncthreads_or(!ok)) {
      failed = true;
      if (tid == 0) {
        atomicOr(status, 1u);
        // the copies still in flight land before the block exits (bounded)
        for (int i = j; i < min(nj, j + kGradStages); ++i)
          mbar_wait_bounded(&bar[i % kGradStages], (uint32_t)((i / kGradStages) & 1));
      }
      break;
    }
    const float* tab = sh_g + st * kStage + lane;
    float cg[kGradM], cs[kGradM];
#pragma unroll
    for (int i = 0; i < kGradM; ++i) {
      cg[i] = g[i];
      cs[i] = sg[i];
    }
    if (j + 1 < nj) load_gs(j + 1);
    if (b0 + 256 * j + lane < nb) {
#pragma unroll
      for (int q = 0; q < kGradK; ++q) {
        const float rw = has_rw ? tab[(kGradRows + q) * 32] : 0.f;
#pragma unroll
        for (int i = 0; i < kGradM; ++i) {
          const int2 iv = s_iv[q][warp * kGradM + i];
          const float lo = tab[iv.x], hi = tab[iv.x + 32];
          const float slope = (hi - lo) * __int_as_float(iv.y);
          acc[q][i] = fmaf(cg[i], slope, acc[q][i]);
          if (has_rw) acc[q][i] = fmaf(cs[i], rw, acc[q][i]);
        }
      }
    }
    __syncthreads();
    if (tid == 0 && j + kGradStages < nj) issue(j + kGradStages);
  }
  if (failed) return;
#pragma unroll
  for (int q = 0; q < kGradK; ++q)
#pragma unroll
    for (int i = 0; i < kGradM; ++i) {
      float t = acc[q][i];
      for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0 && k0 + q < h.din && mw + i < C) gz[((size_t)(mw + i) * h.din + k0 + q) * 8 + w] = t;
    }
}

// Columns [k0, k1) of a mat-vec by one thread: sum_k A[k][p] d[k] with A
// [. x P] row-major, N partial sums in turn, sixteen loads in flight (a load at
// a time made the penalty and the proposal chains of L2 latencies: 27 us per
// launch at P = 200, now 10-14 us).
template <int N>
__device__ __forceinline__ void column_sum(const float* __restrict__ A, int P, int p, const float* __restrict__ d,
                                           int k0, int k1, float (&u)[N]) {
#pragma unroll
  for (int q = 0; q < N; ++q) u[q] = 0.f;
  int k = k0;
  for (; k + 16 <= k1; k += 16) {
    float c[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) c[q] = __ldg(A + (size_t)(k + q) * P + p);
#pragma unroll
    for (int q = 0; q < 16; ++q) u[q % N] = fmaf(c[q], d[k + q], u[q % N]);
  }
  for (; k + N <= k1; k += N)
#pragma unroll
    for (int q = 0; q < N; ++q) u[q] = fmaf(__ldg(A + (size_t)(k + q) * P + p), d[k + q], u[q]);
  for (; k < k1; ++k) u[0] = fmaf(__ldg(A + (size_t)k * P + p), d[k], u[0]);
}

// Sum of red [n] in FP64 by one warp, a fixed order; the result on every lane.
__device__ __forceinline__ double warp_sum(const float* red, int n) {
  double t = 0.0;
  for (int i = threadIdx.x & 31; i < n; i += 32) t += (double)red[i];
  for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Per point (block), G groups of P32 threads as k_finish_accept: the value
// f = llh + penalty and the gradient with respect to the parameters,
// (gz + dx) / scale + 2 C^-1 (theta - mean) (prior optional).
__global__ void k_grad_finish(const double* part, int nblk, const double* theta, int P,
                              const float* __restrict__ scale, const float* gz, const float* dx,
                              const double* __restrict__ m, const float* __restrict__ icov, double* f, double* grad) {
  dep_launch();
  dep_wait();
  extern __shared__ float shf2[];
  const int P32 = (P + 31) & ~31, Gn = blockDim.x / P32;
  float* d = shf2;              // [P32]
  float* up = shf2 + P32;       // [Gn][P32]
  float* red = up + Gn * P32;   // [P32]
  __shared__ double s_llh;
  const int c = blockIdx.x, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int b = lane; b < nblk; b += 32) t += part[(size_t)c * nblk + b];
    for (int off = 16; off; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) s_llh = t;
  }
  const int g = threadIdx.x / P32, p = threadIdx.x - g * P32;
  if (m) {
    if (g == 0) d[p] = p < P ? (float)(theta[(size_t)c * P + p] - m[p]) : 0.f;
    __syncthreads();
    const int ks = (P + Gn - 1) / Gn;
    if (p < P) {
      float u[2];
      column_sum<2>(icov, P, p, d, g * ks, min(P, (g + 1) * ks), u);
      up[g * P32 + p] = u[0] + u[1];
    }
    __syncthreads();
  }
  if (g == 0) {
    float u = 0.f;
    if (m)
      for (int q = 0; q < Gn; ++q) u += (p < P) ? up[q * P32 + p] : 0.f;
    red[p] = m ? d[p] * u : 0.f;
    if (p < P) {
      const size_t o = (size_t)c * P + p;
      float gs = 0.f;  // the parts of k_base_grad, in order
#pragma unroll
      for (int w = 0; w < 8; ++w) gs += gz[o * 8 + w];
      grad[o] = (double)((gs + dx[o]) / scale[p]) + (m ? 2.0 * (double)u : 0.0);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double pen = m ? warp_sum(red, P32) : 0.0;
    if (lane == 0) f[c] = s_llh + pen;
  }
}

// Training target of a reweighted point, one thread per (point, bin):
//   t = (log(sum of weights) - base(x) - mu) / sd
// with the same FP32 base as k_head, so that k_head inverts it.
__global__ void k_target(Head h, const float* __restrict__ x, const double* __restrict__ sums,
                         float* __restrict__ t) {
  const int bin = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = blockIdx.y;
  if (bin >= h.nb) return;
  const float* xm = x + (size_t)m * h.din;
  const double sv = sums[(size_t)m * h.nb + bin];
  const double lr = log(sv > 1e-300 ? sv : 1e-300);
  t[(size_t)m * h.nb + bin] = (float)((lr - (double)head_base(h, xm, bin) - (double)h.mu[bin]) / (double)h.sd[bin]);
}

}  // namespace
}  // namespace gwm

// ---------------------------------------------------------------------------
// Host side: the network object and the C ABI.
// ---------------------------------------------------------------------------
using gw::launch_dependent;
using gwm::bf16;

struct gwm_chain_state;
static void chain_free(gwm_chain_state* s);

struct gwm_net {
  gwm_chain_state* chain = nullptr;  // device state of the surrogate sub-chains (gwm_set_chain)
  int n_layers = 0;
  std::vector<int> dims;  // dims[0] = inputs, dims[L] = outputs
  int batch_max = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  // the base's gradient beside the network's (gwm_value_grad), made on first use
  cudaStream_t side = nullptr;
  cudaEvent_t side_go = nullptr, side_done = nullptr;
  std::vector<void*> allocs;
  const void* opened[24] = {};  // kernels whose shared-memory limit this network has raised (open_shared)
  int n_opened = 0;
  // per layer l (0..L-1): weights [dims[l+1] x dims[l]]
  std::vector<float*> w, b, gw_, gb, mw, vw, mb, vb;
  std::vector<bf16*> wb, wt;
  // activations: x0 (input), then per layer z (f32), h (bf16) and h^T (bf16)
  std::vector<bf16*> h, ht;   // h[0] = input
  std::vector<float*> z;      // z[l] = pre-activation of layer l
  std::vector<bf16*> dz, dzt; // gradients of pre-activations
  float* xin = nullptr;       // staging of the FP32 input
  float* target = nullptr;
  float* loss = nullptr;
  uint32_t* status = nullptr;
  int64_t step = 0;
  std::string err;
  // surrogate head (gwm_set_head / gwm_predict)
  bool has_head = false;
  int h_nodes = 0;
  float h_lim = 0.f;
  size_t h_tab_elems = 0;
  bool h_has_rw = false;
  float *h_mean = nullptr, *h_scale = nullptr, *h_tab = nullptr, *h_b0 = nullptr, *h_mu = nullptr, *h_sd = nullptr,
        *h_rb = nullptr, *h_rw = nullptr;
  double *h_data = nullptr, *h_theta = nullptr, *h_sums = nullptr, *h_sums2 = nullptr, *h_llh = nullptr,
         *h_logr = nullptr, *h_part = nullptr;
  // gradient buffers (gwm_value_grad), allocated on first use
  float *g_G = nullptr, *g_S = nullptr, *g_gz = nullptr, *g_dx = nullptr;
  double *g_f = nullptr, *g_grad = nullptr;
  // training set on the device (gwm_train_reserve / gwm_train_append*):
  // standardised inputs [train_max x dims[0]] and targets [train_max x dims[L]]
  float *train_x = nullptr, *train_t = nullptr;
  int64_t train_n = 0, train_max = 0;
};

static thread_local std::string g_gwm_err;

static int gwm_fail(gwm_net* n, int code, const char* msg) {
  if (n) n->err = msg;
  else g_gwm_err = msg;
  return code;
}

#define GWM_CUDA(n, call)                                             \
  do {                                                                \
    cudaError_t _e = (call);                                          \
    if (_e != cudaSuccess) return gwm_fail((n), GW_ERR_CUDA, cudaGetErrorString(_e)); \
  } while (0)

// Clears and uploads go through the network's stream, which does not wait for the
// legacy default stream: there a memset returns before it is done, and so may a
// copy from pageable memory.
template <typename T>
static int gwm_alloc(gwm_net* n, T** p, size_t count) {
  void* q = nullptr;
  const size_t bytes = sizeof(T) * (count ? count : 1);
  if (cudaMalloc(&q, bytes) == cudaSuccess) n->allocs.push_back(q);
  if (!q || cudaMemsetAsync(q, 0, bytes, n->stream) != cudaSuccess) {
    cudaGetLastError();
    return gwm_fail(n, GW_ERR_NOMEM, "cudaMalloc failed");
  }
  *p = (T*)q;
  return GW_OK;
}

// The host array belongs to the copy until the stream is synchronised.
template <typename T>
static int gwm_upload(gwm_net* n, T* dst, const T* src, size_t count) {
  GWM_CUDA(n, cudaMemcpyAsync(dst, src, sizeof(T) * count, cudaMemcpyHostToDevice, n->stream));
  return GW_OK;
}

// Raises the kernel's limit of dynamic shared memory (48 KB by default) to
// `bytes`, the same for every call with this kernel, on the network's device.  The
// limit belongs to a device, so each network sees to its own.
template <typename... P>
static int open_shared(gwm_net* n, void (*kernel)(P...), size_t bytes) {
  const void* fn = (const void*)kernel;
  for (int i = 0; i < n->n_opened; ++i)
    if (n->opened[i] == fn) return GW_OK;
  const cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (r != cudaSuccess) {
    cudaGetLastError();
    return gwm_fail(n, GW_ERR_CUDA, cudaGetErrorString(r));
  }
  if (n->n_opened < (int)(sizeof(n->opened) / sizeof(n->opened[0]))) n->opened[n->n_opened++] = fn;
  return GW_OK;
}

static size_t gemm_smem(int bn, int stages) {
  return (size_t)stages * (gwm::kBM * gwm::kBK * 2 + bn * gwm::kBK * 2) + 1024;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
    else
      cudaGetLastError();
  });
  return fn;
}

// Tensor map of a row-major BF16 matrix [rows x K] (K % 8 == 0, 16-byte
// aligned rows) read in boxes of 64 K-elements (128 bytes) x box_rows rows
// with the 128-byte swizzle, zero fill.
static int make_map(gwm_net* n, CUtensorMap* map, const bf16* p, int rows, int K, int box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return gwm_fail(n, GW_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  if (((uintptr_t)p & 15) != 0) return gwm_fail(n, GW_ERR_ARG, "GEMM operand not 16-byte aligned");
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)gwm::kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)p, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return gwm_fail(n, GW_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return GW_OK;
}

// Tensor map of a row-major FP32 matrix [rows x cols] (cols % 4 == 0) read in
// boxes of box_cols x box_rows, zero fill.
static int make_map_f32(gwm_net* n, CUtensorMap* map, const float* p, int rows, int cols, int box_cols, int box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return gwm_fail(n, GW_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 4};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)p, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return gwm_fail(n, GW_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return GW_OK;
}

template <int BN, int S, int NW>
static int launch_gemm(gwm_net* n, const bf16* A, const bf16* B, int M, int N, int K, const gwm::Epilogue& ep) {
  CUtensorMap ma, mb;
  int rc = make_map(n, &ma, A, M, K, gwm::kBM);
  if (!rc) rc = make_map(n, &mb, B, N, K, BN);
  if (rc) return rc;
  const size_t smem = gemm_smem(BN, S);
  if ((rc = open_shared(n, gwm::k_gemm<BN, S, NW>, smem))) return rc;
  dim3 grid((N + BN - 1) / BN, (M + gwm::kBM - 1) / gwm::kBM);
  launch_dependent(gwm::k_gemm<BN, S, NW>, grid, NW * 32, smem, n->stream,
                   ma, mb, M, N, K, ep, n->status);
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

struct Product {
  const bf16 *A, *B;
  float* out;
  int M, N;
};

template <int BN, int S, int NW>
static int launch_group(gwm_net* n, const Product* p, int cnt, int K) {
  gwm::GemmGroup g;
  g.n = cnt;
  g.K = K;
  g.tile0[0] = 0;
  for (int i = 0; i < cnt; ++i) {
    int rc = make_map(n, &g.a[i], p[i].A, p[i].M, K, gwm::kBM);
    if (!rc) rc = make_map(n, &g.b[i], p[i].B, p[i].N, K, BN);
    if (rc) return rc;
    g.out[i] = p[i].out;
    g.M[i] = p[i].M;
    g.N[i] = p[i].N;
    g.tile0[i + 1] = g.tile0[i] + ((p[i].N + BN - 1) / BN) * ((p[i].M + gwm::kBM - 1) / gwm::kBM);
  }
  const size_t smem = gemm_smem(BN, S);
  const int rc = open_shared(n, gwm::k_gemm_group<BN, S, NW>, smem);
  if (rc) return rc;
  launch_dependent(gwm::k_gemm_group<BN, S, NW>, g.tile0[cnt], NW * 32, smem, n->stream, g, n->status);
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

constexpr int kWave = 148;  // tiles that give (nearly) each of GB300's 152 SMs one

static int tiles(int M, int N, int BN) { return ((M + gwm::kBM - 1) / gwm::kBM) * ((N + BN - 1) / BN); }

// C[M x N] = A[M x K] * B[N x K]^T with the given epilogue.  The widest tile
// that still gives one CTA per SM or more (148 of GB300's 152): at the
// network's sizes a launch is one wave, and a tile runs few K steps, so more
// CTAs, not wider tiles, keep the chip busy.
//   * 128 x 256 tiles take a ring of two stages, so that two CTAs (and their
//     accumulators, 256 TMEM columns each) share an SM and one's epilogue
//     overlaps the other's MMAs.
//   * With the loss in the epilogue and up to three such tiles per SM, 64-column
//     tiles instead: a thread then has the targets of all its columns on the way
//     before it waits for the accumulator, and the last wave is finer (3000
//     outputs, K = 512, a whole training step: 2048 rows 159 -> 155 us, 4096
//     rows 253 -> 239; 8192 rows 461 -> 465, and 128-column tiles at 1024 rows
//     122 -> 125, which therefore stay).
//   * 64-column tiles that share no SM take eight stages: the K steps are a chain
//     of L2 latencies over the ring's depth (K = 3000, M = 2048, N = 512: 24 ->
//     11 us), and four only where a second tile shares the SM.
//   * Where even 64-column tiles leave half of the SMs idle (few rows),
//     32-column tiles with a ring of eight stages (64 rows, N = K = 512: 17 us
//     with 64-column tiles and four stages, 9 us now; 3000 columns: 10.4 -> 8 us).
// The tile shape does not change the order of any accumulation.
static int gemm(gwm_net* n, const bf16* A, const bf16* B, int M, int N, int K, const gwm::Epilogue& ep) {
  if (K % 8 != 0) return gwm_fail(n, GW_ERR_ARG, "GEMM K must be a multiple of 8");
  const int t256 = tiles(M, N, 256), t64 = tiles(M, N, 64);
  if (N > 128 && t256 >= kWave && !(ep.target && t256 < 3 * kWave))
    return launch_gemm<256, 2, 8>(n, A, B, M, N, K, ep);
  if (N > 64 && t256 < kWave && tiles(M, N, 128) >= kWave) return launch_gemm<128, 4, 8>(n, A, B, M, N, K, ep);
  if (N > 32 && t64 > 152) return launch_gemm<64, 4, 8>(n, A, B, M, N, K, ep);
  if (N > 32 && t64 >= kWave / 2) return launch_gemm<64, 8, 8>(n, A, B, M, N, K, ep);
  return launch_gemm<32, 8, 4>(n, A, B, M, N, K, ep);
}

// The products p[0..cnt), all of depth K, in launches of kMaxGroup.  The widest
// tiles that give half of the SMs one each, with rings as deep as one tile per
// SM allows.  2048 rows of 200-512-512-512-3000 (136 tiles of 128 columns, 272
// of 64 in rings of four, two to an SM, or in rings of eight): a training step
// takes 155, 157 and 168 us, and 190 us with 32-column tiles; 256 rows: 97, 98,
// 100 and 106.
static int gemm_set(gwm_net* n, const Product* p, int cnt, int K) {
  if (K % 8 != 0) return gwm_fail(n, GW_ERR_ARG, "GEMM K must be a multiple of 8");
  for (; cnt > 0; p += gwm::kMaxGroup, cnt -= gwm::kMaxGroup) {
    const int c = cnt < gwm::kMaxGroup ? cnt : gwm::kMaxGroup;
    int t128 = 0, t64 = 0;
    for (int i = 0; i < c; ++i) {
      t128 += tiles(p[i].M, p[i].N, 128);
      t64 += tiles(p[i].M, p[i].N, 64);
    }
    int rc;
    if (t128 >= kWave / 2) rc = launch_group<128, 6, 8>(n, p, c, K);
    else if (t64 >= kWave / 2) rc = launch_group<64, 8, 8>(n, p, c, K);
    else rc = launch_group<32, 8, 4>(n, p, c, K);
    if (rc) return rc;
  }
  return GW_OK;
}

static int check_status(gwm_net* n) {
  uint32_t h = 0;
  GWM_CUDA(n, cudaMemcpyAsync(&h, n->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, n->stream));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  if (h) {
    cudaMemsetAsync(n->status, 0, sizeof(uint32_t), n->stream);
    return gwm_fail(n, GW_ERR_DEVICE_TIMEOUT, "a bounded wait on a tensor-core commit gave up");
  }
  return GW_OK;
}

extern "C" int gwm_create(const int32_t* dims, int32_t n_layers, int32_t batch_max, int32_t device, gwm_net** out) {
  if (!dims || !out || n_layers < 1 || n_layers > 16 || batch_max < 1 || batch_max % 8)
    return gwm_fail(nullptr, GW_ERR_ARG, "gwm_create: bad arguments (batch_max must be a multiple of 8)");
  for (int l = 0; l <= n_layers; ++l)
    if (dims[l] < 8 || dims[l] % 8) return gwm_fail(nullptr, GW_ERR_ARG, "gwm_create: widths must be multiples of 8");
  gwm_net* n = new gwm_net();
  n->n_layers = n_layers;
  n->dims.assign(dims, dims + n_layers + 1);
  n->batch_max = batch_max;
  n->device = device;
  if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    delete n;
    return gwm_fail(nullptr, GW_ERR_CUDA, "gwm_create: no usable CUDA device");
  }
  const int L = n_layers, Bm = batch_max;
  n->w.resize(L); n->b.resize(L); n->gw_.resize(L); n->gb.resize(L); n->mw.resize(L); n->vw.resize(L);
  n->mb.resize(L); n->vb.resize(L); n->wb.resize(L); n->wt.resize(L);
  n->h.resize(L); n->ht.resize(L); n->z.resize(L); n->dz.resize(L); n->dzt.resize(L);
  int rc = GW_OK;
  for (int l = 0; l < L && rc == GW_OK; ++l) {
    const size_t nw = (size_t)dims[l + 1] * dims[l];
    rc |= gwm_alloc(n, &n->w[l], nw) | gwm_alloc(n, &n->gw_[l], nw) | gwm_alloc(n, &n->mw[l], nw) |
          gwm_alloc(n, &n->vw[l], nw) | gwm_alloc(n, &n->wb[l], nw) | gwm_alloc(n, &n->wt[l], nw);
    rc |= gwm_alloc(n, &n->b[l], dims[l + 1]) | gwm_alloc(n, &n->gb[l], dims[l + 1]) |
          gwm_alloc(n, &n->mb[l], dims[l + 1]) | gwm_alloc(n, &n->vb[l], dims[l + 1]);
    rc |= gwm_alloc(n, &n->h[l], (size_t)Bm * dims[l]) | gwm_alloc(n, &n->ht[l], (size_t)Bm * dims[l]);
    rc |= gwm_alloc(n, &n->z[l], (size_t)Bm * dims[l + 1]);
    rc |= gwm_alloc(n, &n->dz[l], (size_t)Bm * dims[l + 1]) | gwm_alloc(n, &n->dzt[l], (size_t)Bm * dims[l + 1]);
  }
  rc |= gwm_alloc(n, &n->xin, (size_t)Bm * dims[0]) | gwm_alloc(n, &n->target, (size_t)Bm * dims[L]) |
        gwm_alloc(n, &n->loss, 1) | gwm_alloc(n, &n->status, 1);
  if (rc != GW_OK) {
    g_gwm_err = n->err;
    for (void* p : n->allocs) cudaFree(p);
    delete n;
    return GW_ERR_NOMEM;
  }
  *out = n;
  return GW_OK;
}

extern "C" int gwm_destroy(gwm_net* n) {
  if (!n) return GW_ERR_ARG;
  cudaSetDevice(n->device);
  cudaStreamSynchronize(n->stream);
  if (n->side) {
    cudaStreamSynchronize(n->side);
    cudaStreamDestroy(n->side);
  }
  if (n->side_go) cudaEventDestroy(n->side_go);
  if (n->side_done) cudaEventDestroy(n->side_done);
  for (void* p : n->allocs) cudaFree(p);
  cudaFree(n->train_x);
  cudaFree(n->train_t);
  cudaFree(n->h_tab);
  chain_free(n->chain);
  cudaStreamDestroy(n->stream);
  delete n;
  return GW_OK;
}

extern "C" int gwm_last_error(const gwm_net* n, char* buf, size_t len) {
  if (!buf || !len) return GW_ERR_ARG;
  snprintf(buf, len, "%s", n ? n->err.c_str() : g_gwm_err.c_str());
  return GW_OK;
}

// Appends layer l to the arguments of k_adam; batch: the rows of the layer's
// transposed output gradients (biases).  Returns the bias blocks so far.
static int adam_layer(gwm_net* n, int l, gwm::AdamArgs* a, int batch, int bias_blocks = 0) {
  gwm::AdamLayer& L = a->l[a->n_layers++];
  L.w = n->w[l];
  L.m = n->mw[l];
  L.v = n->vw[l];
  L.b = n->b[l];
  L.mb = n->mb[l];
  L.vb = n->vb[l];
  L.g = n->gw_[l];
  L.wb = n->wb[l];
  L.wt = n->wt[l];
  L.dzt = n->dzt[l];
  L.rows = n->dims[l + 1];
  L.cols = n->dims[l];
  L.tile0 = a->n_tiles;
  L.bias0 = bias_blocks;
  a->n_tiles += ((L.rows + 31) / 32) * ((L.cols + 31) / 32);
  a->batch = batch;
  return bias_blocks + (L.rows + 15) / 16;
}

// Weights of layer l: w [dims[l+1] x dims[l]] row-major, b [dims[l+1]] (host, FP32).
extern "C" int gwm_set_layer(gwm_net* n, int32_t l, const float* w, const float* b) {
  if (!n || !w || !b || l < 0 || l >= n->n_layers) return GW_ERR_ARG;
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int rows = n->dims[l + 1], cols = n->dims[l];
  const size_t nw = (size_t)rows * cols;
  const int rc = gwm_upload(n, n->w[l], w, nw) | gwm_upload(n, n->b[l], b, rows);
  if (rc) return rc;
  // BF16 copies through a zero-learning-rate Adam pass (also clears the moments)
  GWM_CUDA(n, cudaMemsetAsync(n->gw_[l], 0, sizeof(float) * nw, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(n->mw[l], 0, sizeof(float) * nw, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(n->vw[l], 0, sizeof(float) * nw, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(n->mb[l], 0, sizeof(float) * rows, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(n->vb[l], 0, sizeof(float) * rows, n->stream));
  gwm::AdamArgs aa{};
  adam_layer(n, l, &aa, 1);
  aa.lr = 0.f;
  aa.c1 = aa.c2 = 1.f;
  launch_dependent(gwm::k_adam, aa.n_tiles, 256, 0, n->stream,
                   aa);
  GWM_CUDA(n, cudaGetLastError());
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  n->step = 0;
  return GW_OK;
}

extern "C" int gwm_get_layer(gwm_net* n, int32_t l, float* w, float* b) {
  if (!n || !w || !b || l < 0 || l >= n->n_layers) return GW_ERR_ARG;
  GWM_CUDA(n, cudaSetDevice(n->device));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  const size_t nw = (size_t)n->dims[l + 1] * n->dims[l];
  GWM_CUDA(n, cudaMemcpy(w, n->w[l], sizeof(float) * nw, cudaMemcpyDeviceToHost));
  GWM_CUDA(n, cudaMemcpy(b, n->b[l], sizeof(float) * n->dims[l + 1], cudaMemcpyDeviceToHost));
  return GW_OK;
}

// What a forward pass leaves behind besides the output z[L-1].
enum Keep : int {
  kKeepNone = 0,  // inference
  kKeepZ = 1,     // the hidden pre-activations, for the input gradient
  kKeepAll = 2    // and the transposed activations, for the weight gradients
};

// The training loss at the output: targets (rows perm[r] when perm is set),
// *loss += scale * mean squared error.  The output z[L-1] itself is not stored.
struct Loss {
  const float* target;
  const int32_t* perm;
  float* loss;
  float scale;
};

// Forward pass of the B rows in h[0].  With a loss, the output layer's tiles
// form its gradient dz[L-1] (and the transpose) in their epilogue, so that the
// B x dims[L] output is neither written nor read back.
static int forward(gwm_net* n, int B, Keep keep, const Loss* loss = nullptr) {
  const int L = n->n_layers;
  for (int l = 0; l < L; ++l) {
    gwm::Epilogue ep{};
    ep.bias = n->b[l];
    ep.b_ready = keep != kKeepAll;
    if (l + 1 < L) {
      ep.act = 1;
      if (keep != kKeepNone) ep.out_f32 = n->z[l];
      ep.out_bf16 = n->h[l + 1];
      if (keep == kKeepAll) ep.out_bf16_t = n->ht[l + 1];
      ep.ld_t = B;
    } else if (loss) {
      ep.target = loss->target;
      ep.perm = loss->perm;
      ep.loss = loss->loss;
      ep.inv = 1.f / ((float)B * (float)n->dims[L]);
      ep.scale = loss->scale;
      ep.out_bf16 = n->dz[l];
      ep.out_bf16_t = n->dzt[l];
      ep.ld_t = B;
    } else {
      ep.out_f32 = n->z[l];
    }
    int rc = gemm(n, n->h[l], n->wb[l], B, n->dims[l + 1], n->dims[l], ep);
    if (rc) return rc;
  }
  return GW_OK;
}

static dim3 tiles32(int rows, int cols) { return dim3((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32)); }

// Input rows to BF16 (and transposed) for the first GEMM; row r is perm[r] of x (perm null: r).
// The transposed copy feeds the weight gradient of the first layer.
static int stage_input(gwm_net* n, const float* x, const int32_t* perm, int B) {
  launch_dependent(gwm::k_rows_to_bf16, tiles32(B, n->dims[0]), dim3(32, 8), 0, n->stream,
                   x, perm, B, n->dims[0], n->h[0], n->ht[0], B);
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

static int load_input(gwm_net* n, const float* x, int B, bool device_ptr) {
  const size_t cnt = (size_t)B * n->dims[0];
  GWM_CUDA(n, cudaMemcpyAsync(n->xin, x, sizeof(float) * cnt,
                              device_ptr ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, n->stream));
  return stage_input(n, n->xin, nullptr, B);
}

// Forward pass of B inputs x [B x dims[0]] (FP32, host or device) into
// y [B x dims[L]] (FP32, same side as x).
extern "C" int gwm_forward(gwm_net* n, const float* x, int32_t B, float* y, int32_t device_ptrs) {
  if (!n || !x || !y || B < 1 || B > n->batch_max || B % 8) return gwm_fail(n, GW_ERR_ARG, "gwm_forward: bad batch");
  GWM_CUDA(n, cudaSetDevice(n->device));
  int rc = load_input(n, x, B, device_ptrs != 0);
  if (!rc) rc = forward(n, B, kKeepNone);
  if (rc) return rc;
  const int L = n->n_layers;
  GWM_CUDA(n, cudaMemcpyAsync(y, n->z[L - 1], sizeof(float) * (size_t)B * n->dims[L],
                              device_ptrs ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, n->stream));
  return check_status(n);
}

static int backward(gwm_net* n, int B) {
  const int L = n->n_layers;
  // dz[L-1] (and its transpose) was written by the forward pass's loss epilogue;
  // the bias gradients follow from the dzt (k_adam, k_bias_grad)
  for (int l = L - 1; l > 0; --l) {
    // dz_{l-1} = (dz_l W_l) * silu'(z_{l-1}) : [B x dims[l]], K = dims[l+1]
    gwm::Epilogue ep{};
    ep.gate = n->z[l - 1];
    ep.out_bf16 = n->dz[l - 1];
    ep.out_bf16_t = n->dzt[l - 1];
    ep.ld_t = B;
    int rc = gemm(n, n->dz[l], n->wt[l], B, n->dims[l], n->dims[l + 1], ep);
    if (rc) return rc;
  }
  // dW_l = dz_l^T h_l : [dims[l+1] x dims[l]], K = B
  std::vector<Product> dw(L);
  for (int l = 0; l < L; ++l) dw[l] = {n->dzt[l], n->ht[l], n->gw_[l], n->dims[l + 1], n->dims[l]};
  return gemm_set(n, dw.data(), L, B);
}

// Forward pass with the loss against host or device targets t [B x dims[L]] in *n->loss.
static int forward_loss(gwm_net* n, const float* t, int B, bool device_ptr) {
  const size_t cnt = (size_t)B * n->dims[n->n_layers];
  GWM_CUDA(n, cudaMemcpyAsync(n->target, t, sizeof(float) * cnt,
                              device_ptr ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(n->loss, 0, sizeof(float), n->stream));
  const Loss ls{n->target, nullptr, n->loss, 1.f};
  return forward(n, B, kKeepAll, &ls);
}

// One Adam update of every layer with learning rate lr after a backward pass of B rows.
static int adam_all(gwm_net* n, int B, float lr) {
  n->step += 1;
  gwm::AdamArgs a{};
  int bias_blocks = 0;
  for (int l = 0; l < n->n_layers; ++l) bias_blocks = adam_layer(n, l, &a, B, bias_blocks);
  a.lr = lr;
  a.c1 = 1.f - powf(0.9f, (float)n->step);
  a.c2 = 1.f - powf(0.999f, (float)n->step);
  launch_dependent(gwm::k_adam, a.n_tiles + bias_blocks, 256, 0, n->stream,
                   a);
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

// Gradients of the mean squared error for a batch (no update): copied to
// the host, layer by layer, gw[l] [dims[l+1] x dims[l]], gb[l] [dims[l+1]].
extern "C" int gwm_gradients(gwm_net* n, const float* x, const float* t, int32_t B, float* const* gw,
                             float* const* gb, float* loss) {
  if (!n || !x || !t || !gw || !gb || B < 8 || B > n->batch_max || B % 8)
    return gwm_fail(n, GW_ERR_ARG, "gwm_gradients: bad batch");
  GWM_CUDA(n, cudaSetDevice(n->device));
  int rc = load_input(n, x, B, false);
  if (!rc) rc = forward_loss(n, t, B, false);
  if (!rc) rc = backward(n, B);
  if (rc) return rc;
  for (int l = 0; l < n->n_layers; ++l)
    launch_dependent(gwm::k_bias_grad, (n->dims[l + 1] + 15) / 16, 256, 0, n->stream,
                     n->dzt[l], n->dims[l + 1], B, n->gb[l]);
  GWM_CUDA(n, cudaGetLastError());
  rc = check_status(n);
  if (rc) return rc;
  for (int l = 0; l < n->n_layers; ++l) {
    GWM_CUDA(n, cudaMemcpy(gw[l], n->gw_[l], sizeof(float) * (size_t)n->dims[l + 1] * n->dims[l],
                           cudaMemcpyDeviceToHost));
    GWM_CUDA(n, cudaMemcpy(gb[l], n->gb[l], sizeof(float) * n->dims[l + 1], cudaMemcpyDeviceToHost));
  }
  if (loss) GWM_CUDA(n, cudaMemcpy(loss, n->loss, sizeof(float), cudaMemcpyDeviceToHost));
  return GW_OK;
}

// One Adam step on a batch (x, t on the device when device_ptrs != 0).
extern "C" int gwm_train_step(gwm_net* n, const float* x, const float* t, int32_t B, float lr, int32_t device_ptrs,
                              float* loss) {
  if (!n || !x || !t || B < 8 || B > n->batch_max || B % 8) return gwm_fail(n, GW_ERR_ARG, "gwm_train_step: bad batch");
  GWM_CUDA(n, cudaSetDevice(n->device));
  int rc = load_input(n, x, B, device_ptrs != 0);
  if (!rc) rc = forward_loss(n, t, B, device_ptrs != 0);
  if (!rc) rc = backward(n, B);
  if (!rc) rc = adam_all(n, B, lr);
  if (rc) return rc;
  if (loss) {
    GWM_CUDA(n, cudaMemcpyAsync(loss, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
  }
  return check_status(n);
}

// Plain GEMM through the same kernel (tests): C[M x N] = A[M x K] B[N x K]^T,
// BF16 inputs, FP32 output, all host arrays.
extern "C" int gwm_gemm_test(const uint16_t* A, const uint16_t* B, int32_t M, int32_t N, int32_t K, float* C) {
  if (!A || !B || !C || M < 1 || N < 1 || K < 8 || K % 8) return gwm_fail(nullptr, GW_ERR_ARG, "gwm_gemm_test: bad sizes");
  gwm_net tmp;
  if (cudaStreamCreate(&tmp.stream) != cudaSuccess) return gwm_fail(nullptr, GW_ERR_CUDA, "no stream");
  bf16 *dA = nullptr, *dB = nullptr;
  float* dC = nullptr;
  int rc = gwm_alloc(&tmp, &dA, (size_t)M * K) | gwm_alloc(&tmp, &dB, (size_t)N * K) |
           gwm_alloc(&tmp, &dC, (size_t)M * N) | gwm_alloc(&tmp, &tmp.status, 1);
  if (rc == GW_OK) {
    cudaMemcpy(dA, A, sizeof(uint16_t) * (size_t)M * K, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, B, sizeof(uint16_t) * (size_t)N * K, cudaMemcpyHostToDevice);
    gwm::Epilogue ep{};
    ep.out_f32 = dC;
    rc = gemm(&tmp, dA, dB, M, N, K, ep);
    if (rc == GW_OK) rc = check_status(&tmp);
    if (rc == GW_OK && cudaMemcpy(C, dC, sizeof(float) * (size_t)M * N, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = GW_ERR_CUDA;
  }
  if (rc != GW_OK) g_gwm_err = tmp.err;
  for (void* p : tmp.allocs) cudaFree(p);
  cudaStreamDestroy(tmp.stream);
  return rc;
}

// ---------------------------------------------------------------------------
// Surrogate head: standardisation, affine base, output scaling, rate -> LLH.
// ---------------------------------------------------------------------------
static gwm::Head head_view(const gwm_net* n) {
  gwm::Head h{};
  h.din = n->dims[0];
  h.nb = n->dims[n->n_layers];
  h.nodes = n->h_nodes;
  h.lim = n->h_lim;
  h.tab = n->h_tab;
  h.b0 = n->h_b0;
  h.mu = n->h_mu;
  h.sd = n->h_sd;
  h.r_w = n->h_has_rw ? n->h_rw : nullptr;
  h.r_b = n->h_rb;
  return h;
}

// Buffers of the head and of gwm_predict; the base table is (re)sized to tab_elems.
static int head_alloc(gwm_net* n, size_t tab_elems) {
  const int din = n->dims[0], nb = n->dims[n->n_layers], Bm = n->batch_max;
  if (!n->has_head) {
    int rc = gwm_alloc(n, &n->h_mean, din) | gwm_alloc(n, &n->h_scale, din) | gwm_alloc(n, &n->h_b0, nb) |
             gwm_alloc(n, &n->h_mu, nb) | gwm_alloc(n, &n->h_sd, nb) | gwm_alloc(n, &n->h_rb, nb) |
             gwm_alloc(n, &n->h_rw, (size_t)din * nb) | gwm_alloc(n, &n->h_data, nb) |
             gwm_alloc(n, &n->h_theta, (size_t)Bm * din) | gwm_alloc(n, &n->h_sums, (size_t)Bm * nb) |
             gwm_alloc(n, &n->h_sums2, (size_t)Bm * nb) | gwm_alloc(n, &n->h_llh, Bm) |
             gwm_alloc(n, &n->h_logr, (size_t)Bm * nb) | gwm_alloc(n, &n->h_part, (size_t)Bm * ((nb + 31) / 32));
    if (rc) return rc;
    n->has_head = true;
  }
  if (n->h_tab_elems != tab_elems) {
    GWM_CUDA(n, cudaStreamSynchronize(n->stream));
    cudaFree(n->h_tab);
    n->h_tab = nullptr;
    n->h_tab_elems = 0;
    if (cudaMalloc(&n->h_tab, sizeof(float) * tab_elems) != cudaSuccess) {
      cudaGetLastError();
      n->h_tab = nullptr;
      return gwm_fail(n, GW_ERR_NOMEM, "cudaMalloc failed (head table)");
    }
    n->h_tab_elems = tab_elems;
  }
  return GW_OK;
}

// Uploads the parts shared by both head forms; ends with the stream's work done.
static int head_common(gwm_net* n, const float* in_mean, const float* in_scale, const float* base_b,
                       const float* out_mu, const float* out_sd, const float* ratio_w, const double* data) {
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  std::vector<float> rt;
  n->h_has_rw = ratio_w != nullptr;
  if (ratio_w) {
    // [nb x din] -> [din x nb]
    rt.resize((size_t)din * nb);
    for (int b = 0; b < nb; ++b)
      for (int k = 0; k < din; ++k) rt[(size_t)k * nb + b] = ratio_w[(size_t)b * din + k];
  }
  const int rc = gwm_upload(n, n->h_mean, in_mean, din) | gwm_upload(n, n->h_scale, in_scale, din) |
                 gwm_upload(n, n->h_b0, base_b, nb) | gwm_upload(n, n->h_mu, out_mu, nb) |
                 gwm_upload(n, n->h_sd, out_sd, nb) | gwm_upload(n, n->h_data, data, nb) |
                 (rt.empty() ? GW_OK : gwm_upload(n, n->h_rw, rt.data(), rt.size()));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  return rc;
}

extern "C" int gwm_set_head(gwm_net* n, const float* in_mean, const float* in_scale, const float* base_w,
                            const float* base_b, const float* out_mu, const float* out_sd, const float* ratio,
                            const double* data) {
  if (!n || !in_mean || !in_scale || !base_w || !base_b || !out_mu || !out_sd || !ratio || !data) return GW_ERR_ARG;
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  int rc = head_alloc(n, (size_t)din * nb);
  if (rc) return rc;
  // base_w arrives as [nb x din]; stored transposed [din x nb] for the head kernel
  std::vector<float> wt((size_t)din * nb), lr(nb);
  for (int b = 0; b < nb; ++b)
    for (int k = 0; k < din; ++k) wt[(size_t)k * nb + b] = base_w[(size_t)b * din + k];
  for (int b = 0; b < nb; ++b) lr[b] = ratio[b] > 0.f ? logf(ratio[b]) : -1e30f;
  rc = gwm_upload(n, n->h_tab, wt.data(), wt.size()) | gwm_upload(n, n->h_rb, lr.data(), nb);
  n->h_nodes = 0;
  n->h_lim = 0.f;
  return rc | head_common(n, in_mean, in_scale, base_b, out_mu, out_sd, nullptr, data);
}

extern "C" int gwm_set_head_additive(gwm_net* n, const float* in_mean, const float* in_scale, int32_t nodes,
                                     float lim, const float* base_tab, const float* base_b, const float* out_mu,
                                     const float* out_sd, const float* ratio_w, const float* ratio_b,
                                     const double* data) {
  if (!n || !in_mean || !in_scale || !base_tab || !base_b || !out_mu || !out_sd || !ratio_b || !data || nodes < 2 ||
      nodes > 4096 || !(lim > 0.f))
    return gwm_fail(n, GW_ERR_ARG, "gwm_set_head_additive: bad arguments");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  const size_t te = (size_t)din * nodes * nb;
  int rc = head_alloc(n, te);
  if (rc) return rc;
  rc = gwm_upload(n, n->h_tab, base_tab, te) | gwm_upload(n, n->h_rb, ratio_b, nb);
  n->h_nodes = nodes;
  n->h_lim = lim;
  return rc | head_common(n, in_mean, in_scale, base_b, out_mu, out_sd, ratio_w, data);
}

// Tensor maps of the base table and of r_w in boxes of box_cols bins x
// box_params parameters.
static int head_maps(gwm_net* n, CUtensorMap* tab, CUtensorMap* rw, int box_cols, int box_params) {
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  const int rc = make_map_f32(n, tab, n->h_tab, din * n->h_nodes, nb, box_cols, box_params * n->h_nodes);
  return rc ? rc : make_map_f32(n, rw, n->h_rw, din, nb, box_cols, box_params);
}

// A base whose tables the staged kernels hold (k_head_staged, k_base_grad_staged).
static bool head_staged(const gwm_net* n) { return n->h_nodes >= 2 && n->h_nodes <= gwm::kHeadNodes; }

// Likelihood partials per point: one per block of bins.
static int head_parts(const gwm_net* n) {
  const int nb = n->dims[n->n_layers], w = head_staged(n) ? gwm::kHeadBins : 32;
  return (nb + w - 1) / w;
}

template <bool GRAD>
static int launch_head(gwm_net* n, int C, int llh_type, const gwm::HeadOut& out) {
  const int L = n->n_layers;
  constexpr int kPPT = 2;
  const size_t shm = (size_t)8 * kPPT * n->dims[0] * 12;
  if (shm > 200 * 1024) return gwm_fail(n, GW_ERR_LIMIT, "surrogate head: too many inputs");
  if (head_staged(n)) {
    CUtensorMap tab, rw;
    int rc = head_maps(n, &tab, &rw, gwm::kHeadBins, gwm::kHeadK);
    if (rc) return rc;
    constexpr int kShm = gwm::kHeadStages * gwm::kHeadStage * 4;
    if ((rc = open_shared(n, gwm::k_head_staged<GRAD>, kShm))) return rc;
    const dim3 grid(head_parts(n), (C + gwm::kHeadPts - 1) / gwm::kHeadPts);
    launch_dependent(gwm::k_head_staged<GRAD>, grid, gwm::kHeadThreads, kShm, n->stream,
                     tab, rw, head_view(n), n->xin, n->z[L - 1], C, n->h_data, llh_type, out, n->status);
  } else {
    if (shm > 48 * 1024) {
      const int rc = open_shared(n, gwm::k_head_llh<kPPT, GRAD>, 200 * 1024);
      if (rc) return rc;
    }
    const dim3 grid(head_parts(n), (C + 8 * kPPT - 1) / (8 * kPPT));
    launch_dependent(gwm::k_head_llh<kPPT, GRAD>, grid, dim3(32, 8), shm, n->stream,
                     head_view(n), n->xin, n->z[L - 1], C, n->h_data, llh_type, out);
  }
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

// The base's part of the input gradient, eight parts per (point, parameter) in g_gz.
static int launch_base_grad(gwm_net* n, int C, cudaStream_t stream) {
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  const size_t shb = sizeof(float) * 2 * (size_t)nb;
  if (shb > 200 * 1024) return gwm_fail(n, GW_ERR_LIMIT, "gwm_value_grad: too many bins");
  if (head_staged(n)) {
    CUtensorMap tab, rw;
    int rc = head_maps(n, &tab, &rw, 32, gwm::kGradK);
    if (rc) return rc;
    constexpr int kShm = gwm::kGradStages * (gwm::kGradRows + gwm::kGradK) * 32 * 4;
    if ((rc = open_shared(n, gwm::k_base_grad_staged, kShm))) return rc;
    constexpr int kTile = 8 * gwm::kGradM;
    const dim3 grid(8, (din + gwm::kGradK - 1) / gwm::kGradK, (C + kTile - 1) / kTile);
    launch_dependent(gwm::k_base_grad_staged, grid, 256, kShm, stream,
                     tab, rw, head_view(n), n->xin, n->g_G, n->g_S, C, n->g_gz, n->status);
  } else {
    if (shb > 48 * 1024) {
      const int rc = open_shared(n, gwm::k_base_grad, 200 * 1024);
      if (rc) return rc;
    }
    launch_dependent(gwm::k_base_grad, dim3(C, (din + 7) / 8), 256, shb, stream,
                     head_view(n), n->xin, n->g_G, n->g_S, n->g_gz);
  }
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

// Fused head + likelihood of the first C rows of the network's output (xin
// holds their standardised inputs): h_llh [C]; with `outputs`, h_sums,
// h_sums2 and h_logr too.
static int head_llh(gwm_net* n, int C, int llh_type, bool outputs, bool finish = true) {
  gwm::HeadOut out{};
  out.part = n->h_part;
  if (outputs) {
    out.sums = n->h_sums;
    out.sums2 = n->h_sums2;
    out.logr = n->h_logr;
  }
  const int rc = launch_head<false>(n, C, llh_type, out);
  if (rc) return rc;
  const int nbx = head_parts(n);
  if (finish) launch_dependent(gwm::k_llh_finish, (C + 7) / 8, 256, 0, n->stream,
                     n->h_part, nbx, C, n->h_llh);
  GWM_CUDA(n, cudaGetLastError());
  return GW_OK;
}

// Surrogate statistical likelihood of B parameter points theta [B x din]
// (host FP64): llh [B]; log_rates [B x nb] optional.  llh_type as gw_eval.
extern "C" int gwm_predict(gwm_net* n, const double* theta, int32_t B, int32_t llh_type, double* llh,
                           double* log_rates) {
  if (!n || !theta || !llh || B < 1 || B > n->batch_max) return gwm_fail(n, GW_ERR_ARG, "gwm_predict: bad batch");
  if (!n->has_head) return gwm_fail(n, GW_ERR_STATE, "gwm_predict: gwm_set_head has not been called");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  const int Bp = ((B + 7) / 8) * 8;  // GEMM rows in multiples of 8; the extra rows are zeros
  if (Bp > n->batch_max) return gwm_fail(n, GW_ERR_ARG, "gwm_predict: batch above batch_max after padding");
  if (Bp > B) GWM_CUDA(n, cudaMemsetAsync(n->h_theta, 0, sizeof(double) * (size_t)Bp * din, n->stream));
  GWM_CUDA(n, cudaMemcpyAsync(n->h_theta, theta, sizeof(double) * (size_t)B * din, cudaMemcpyHostToDevice, n->stream));
  gwm::k_standardize<<<(unsigned)(((size_t)Bp * din + 255) / 256), 256, 0, n->stream>>>(
      n->h_theta, Bp, din, n->h_mean, n->h_scale, n->xin, n->h[0]);
  GWM_CUDA(n, cudaGetLastError());
  int rc = forward(n, Bp, kKeepNone);
  if (rc) return rc;
  rc = head_llh(n, B, llh_type, log_rates != nullptr);
  if (rc) return rc;
  GWM_CUDA(n, cudaMemcpyAsync(llh, n->h_llh, sizeof(double) * B, cudaMemcpyDeviceToHost, n->stream));
  if (log_rates)
    GWM_CUDA(n, cudaMemcpyAsync(log_rates, n->h_logr, sizeof(double) * (size_t)B * nb, cudaMemcpyDeviceToHost,
                                n->stream));
  return check_status(n);
}

// ---------------------------------------------------------------------------
// Training set on the device and the training loop.
// ---------------------------------------------------------------------------
extern "C" int gwm_train_reserve(gwm_net* n, int64_t n_max) {
  if (!n || n_max < 8) return gwm_fail(n, GW_ERR_ARG, "gwm_train_reserve: n_max must be >= 8");
  GWM_CUDA(n, cudaSetDevice(n->device));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  cudaFree(n->train_x);
  cudaFree(n->train_t);
  n->train_x = n->train_t = nullptr;
  n->train_n = n->train_max = 0;
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  if (cudaMalloc(&n->train_x, sizeof(float) * (size_t)n_max * din) != cudaSuccess ||
      cudaMalloc(&n->train_t, sizeof(float) * (size_t)n_max * nb) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(n->train_x);
    cudaFree(n->train_t);
    n->train_x = n->train_t = nullptr;
    return gwm_fail(n, GW_ERR_NOMEM, "gwm_train_reserve: cudaMalloc failed");
  }
  n->train_max = n_max;
  return GW_OK;
}

extern "C" int gwm_train_size(gwm_net* n, int64_t* count) {
  if (!n || !count) return GW_ERR_ARG;
  *count = n->train_n;
  return GW_OK;
}

// Standardises h_theta rows and turns h_sums rows into targets at the end of
// the training set (the head must be set).
static int append_rows(gwm_net* n, int K) {
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  float* x = n->train_x + (size_t)n->train_n * din;
  gwm::k_standardize<<<(unsigned)(((size_t)K * din + 255) / 256), 256, 0, n->stream>>>(
      n->h_theta, K, din, n->h_mean, n->h_scale, x, nullptr);
  gwm::k_target<<<dim3((nb + 255) / 256, K), 256, 0, n->stream>>>(head_view(n), x, n->h_sums,
                                                                  n->train_t + (size_t)n->train_n * nb);
  GWM_CUDA(n, cudaGetLastError());
  n->train_n += K;
  return GW_OK;
}

static int append_check(gwm_net* n, const double* theta, int K, const char* who) {
  if (!n || !theta || K < 1 || K > n->batch_max) return gwm_fail(n, GW_ERR_ARG, who);
  if (!n->has_head) return gwm_fail(n, GW_ERR_STATE, "training targets need the head (gwm_set_head) first");
  if (n->train_n + K > n->train_max) return gwm_fail(n, GW_ERR_LIMIT, "training set full (gwm_train_reserve)");
  return GW_OK;
}

// Appends K points theta [K x dims[0]] (host FP64) with their bin sums
// [K x dims[L]] (FP64, host, or device memory when sums_on_device != 0).
extern "C" int gwm_train_append(gwm_net* n, const double* theta, const double* sums, int32_t K,
                                int32_t sums_on_device) {
  int rc = append_check(n, theta, K, "gwm_train_append: bad arguments");
  if (rc) return rc;
  if (!sums) return gwm_fail(n, GW_ERR_ARG, "gwm_train_append: sums missing");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  GWM_CUDA(n, cudaMemcpyAsync(n->h_theta, theta, sizeof(double) * (size_t)K * din, cudaMemcpyHostToDevice, n->stream));
  GWM_CUDA(n, cudaMemcpyAsync(n->h_sums, sums, sizeof(double) * (size_t)K * nb,
                              sums_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, n->stream));
  rc = append_rows(n, K);
  if (rc) return rc;
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  return GW_OK;
}

// Appends K points theta [K x dims[0]] (host FP64) reweighted exactly by the
// engine e on the network's stream; nothing leaves the device.  The engine's
// parameter count must equal dims[0], its bin count dims[L], and K <= its k_max.
extern "C" int gwm_train_append_eval(gwm_net* n, gw_engine* e, const double* theta, int32_t K) {
  int rc = append_check(n, theta, K, "gwm_train_append_eval: bad arguments");
  if (rc) return rc;
  if (!e) return gwm_fail(n, GW_ERR_ARG, "gwm_train_append_eval: no engine");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0];
  GWM_CUDA(n, cudaMemcpyAsync(n->h_theta, theta, sizeof(double) * (size_t)K * din, cudaMemcpyHostToDevice, n->stream));
  rc = gw_eval_device(e, n->h_theta, K, n->h_sums, n->h_sums2, nullptr, nullptr, (void*)n->stream);
  if (rc) {
    char buf[256];
    gw_last_error(e, buf, sizeof(buf));
    n->err = std::string("gwm_train_append_eval: engine: ") + buf;
    return rc;
  }
  return append_rows(n, K);
}

// Trains on the device-resident set: `epochs` passes of floor(count / batch)
// Adam steps over a seeded permutation per epoch, learning rate cosine-decayed
// from lr0 to lr_min over all steps.  No host synchronisation between steps;
// losses[e] = mean training loss of epoch e (optional).
extern "C" int gwm_train_epochs(gwm_net* n, int32_t epochs, int32_t batch, float lr0, float lr_min, uint64_t seed,
                                float* losses) {
  if (!n || epochs < 1 || batch < 8 || batch % 8 || batch > n->batch_max)
    return gwm_fail(n, GW_ERR_ARG, "gwm_train_epochs: bad epochs or batch");
  if (n->train_n < batch) return gwm_fail(n, GW_ERR_STATE, "gwm_train_epochs: fewer training points than one batch");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int64_t N = n->train_n;
  const int64_t spe = N / batch, total = (int64_t)epochs * spe;
  // permutations of all epochs, drawn on the host (splitmix64 + Fisher-Yates)
  std::vector<int32_t> perm((size_t)epochs * N);
  uint64_t st = seed;
  auto next = [&st]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  for (int e = 0; e < epochs; ++e) {
    int32_t* p = perm.data() + (size_t)e * N;
    for (int64_t i = 0; i < N; ++i) p[i] = (int32_t)i;
    for (int64_t i = N - 1; i > 0; --i) {
      const int64_t j = (int64_t)(next() % (uint64_t)(i + 1));
      std::swap(p[i], p[j]);
    }
  }
  int32_t* d_perm = nullptr;
  float* d_loss = nullptr;
  if (cudaMalloc(&d_perm, sizeof(int32_t) * perm.size()) != cudaSuccess ||
      cudaMalloc(&d_loss, sizeof(float) * epochs) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(d_perm);
    return gwm_fail(n, GW_ERR_NOMEM, "gwm_train_epochs: cudaMalloc failed");
  }
  int rc = GW_OK;
  if (cudaMemcpyAsync(d_perm, perm.data(), sizeof(int32_t) * perm.size(), cudaMemcpyHostToDevice, n->stream) !=
          cudaSuccess ||
      cudaMemsetAsync(d_loss, 0, sizeof(float) * epochs, n->stream) != cudaSuccess)
    rc = gwm_fail(n, GW_ERR_CUDA, "gwm_train_epochs: copy failed");
  const float inv_spe = 1.f / (float)spe;
  for (int64_t s = 0; s < total && rc == GW_OK; ++s) {
    const int64_t e = s / spe, j = s % spe;
    const int32_t* p = d_perm + e * N + j * batch;
    const double c = std::cos(M_PI * (double)s / (double)total);
    const float lr = (float)(lr_min + 0.5 * (lr0 - lr_min) * (1.0 + c));
    rc = stage_input(n, n->train_x, p, batch);
    const Loss ls{n->train_t, p, d_loss + e, inv_spe};
    if (!rc) rc = forward(n, batch, kKeepAll, &ls);
    if (!rc) rc = backward(n, batch);
    if (!rc) rc = adam_all(n, batch, lr);
  }
  if (rc == GW_OK) rc = check_status(n);
  if (rc == GW_OK && losses &&
      cudaMemcpy(losses, d_loss, sizeof(float) * epochs, cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = gwm_fail(n, GW_ERR_CUDA, "gwm_train_epochs: loss copy failed");
  cudaStreamSynchronize(n->stream);
  cudaFree(d_perm);
  cudaFree(d_loss);
  return rc;
}

// Copies rows [first, first + count) of the training set to the host:
// x [count x dims[0]] standardised inputs, t [count x dims[L]] targets.
extern "C" int gwm_train_read(gwm_net* n, int64_t first, int32_t count, float* x, float* t) {
  if (!n || first < 0 || count < 0 || first + count > n->train_n) return gwm_fail(n, GW_ERR_ARG, "gwm_train_read: range");
  GWM_CUDA(n, cudaSetDevice(n->device));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  const int din = n->dims[0], nb = n->dims[n->n_layers];
  if (x && count)
    GWM_CUDA(n, cudaMemcpy(x, n->train_x + (size_t)first * din, sizeof(float) * (size_t)count * din,
                           cudaMemcpyDeviceToHost));
  if (t && count)
    GWM_CUDA(n, cudaMemcpy(t, n->train_t + (size_t)first * nb, sizeof(float) * (size_t)count * nb,
                           cudaMemcpyDeviceToHost));
  return GW_OK;
}

// ---------------------------------------------------------------------------
// Surrogate random-walk Metropolis sub-chains on the device: stage 1 of the
// delayed-acceptance sampler.  Per chain c and sub-step s:
//   prop = phi + L n,  n ~ N(0, I) (counter-based hash of (seed, s, c, k));
//   f(prop) = surrogate statistical LLH + (prop - m)^T C^-1 (prop - m);
//   accept when log u < -(f(prop) - f(phi)) / 2, u from the same hash.
// The surrogate of a point depends on that point alone (row-independent GEMM
// tiles, fixed-order reductions), so f is a fixed function of the point.
// ---------------------------------------------------------------------------
namespace gwm {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t hash4(uint64_t seed, uint64_t step, uint64_t chain, uint64_t k) {
  uint64_t h = mix64(seed + 0x9E3779B97F4A7C15ull);
  h = mix64(h ^ (step * 0xD1B54A32D192ED03ull));
  h = mix64(h ^ (chain * 0xABC98388FB8FAC03ull));
  return mix64(h ^ (k * 0x8CB92BA72F3D8DD7ull));
}

// uniform in (0, 1), 53 bits
__device__ __forceinline__ double u01(uint64_t h) { return ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0); }

// First step of a sub-step, block per chain: standard normals n[k]
// (Box-Muller on hash pairs, FP32), the proposal prop = phi + L n with the
// increment in FP32 (Lt = L transposed, so that thread p reads column p
// coalesced; the increment depends on n alone, so the proposal is
// symmetric), written in FP64, and its standardised inputs
// x = (prop - mean) / scale (FP32, as k_standardize) with the BF16 row of the
// first GEMM (as k_rows_to_bf16).
__global__ void k_propose_stage(const double* phi, int P, const float* __restrict__ Lt, uint64_t seed,
                                uint64_t step, double* prop, const float* __restrict__ mean,
                                const float* __restrict__ scale, float* x, bf16* h0) {
  dep_launch();
  dep_wait();
  // blockDim.x = G * P32: group g of the column's partial sums covers the
  // k-range [g*ks, (g+1)*ks); the groups are combined in a fixed order
  extern __shared__ float shp[];
  const int P32 = (P + 31) & ~31, G = blockDim.x / P32;
  float* nrm = shp;            // [P + 1]
  float* part = shp + P + 1;   // [G][P32]
  const int c = blockIdx.x;
  for (int k2 = threadIdx.x; 2 * k2 < P; k2 += blockDim.x) {
    const float u1 = (float)u01(hash4(seed, step, c, 2 * k2));
    const float u2 = (float)u01(hash4(seed, step, c, 2 * k2 + 1));
    const float r = sqrtf(-2.f * logf(u1));
    float sn, cs;
    sincospif(2.f * u2, &sn, &cs);
    nrm[2 * k2] = r * cs;
    if (2 * k2 + 1 < P) nrm[2 * k2 + 1] = r * sn;
  }
  __syncthreads();
  const int g = threadIdx.x / P32, p = threadIdx.x - g * P32;
  const int ks = (P + G - 1) / G;
  if (p < P) {
    float a[4];
    column_sum<4>(Lt, P, p, nrm, g * ks, min(min(P, (g + 1) * ks), p + 1), a);
    part[g * P32 + p] = (a[0] + a[1]) + (a[2] + a[3]);
  }
  __syncthreads();
  if (g == 0 && p < P) {
    float inc = 0.f;
    for (int q = 0; q < G; ++q) inc += part[q * P32 + p];
    const size_t o = (size_t)c * P + p;
    const double v = phi[o] + (double)inc;
    prop[o] = v;
    const float z = (float)((v - (double)mean[p]) / (double)scale[p]);
    x[o] = z;
    h0[o] = __float2bfloat16(z);
  }
}

// Last step of a sub-step, block per chain: the surrogate LLH of the proposal
// from the per-block partials (the order of k_llh_finish), its prior penalty
// d^T C^-1 d, d = prop - m (FP32, C^-1 read by columns, fixed-order
// reduction; skipped when m is null), and the Metropolis decision on
// f = llh + penalty: accept when log u < -(f - f_current) / 2 with u from the
// hash of (seed, step, chain); NaN proposals are rejected.  first != 0 takes
// the value unconditionally (the initial evaluation).
__global__ void k_finish_accept(const double* part, int nblk, const double* prop, int P,
                                const double* __restrict__ m, const float* __restrict__ icov, uint64_t seed,
                                uint64_t step, int first, double* phi, double* f, int32_t* n_acc) {
  dep_launch();
  dep_wait();
  // blockDim.x = G * P32 as k_propose_stage
  extern __shared__ float shf[];
  const int P32 = (P + 31) & ~31, G = blockDim.x / P32;
  float* d = shf;              // [P32]
  float* up = shf + P32;       // [G][P32]
  float* red = up + G * P32;   // [P32]
  __shared__ double s_llh;
  __shared__ int s_take;
  const int c = blockIdx.x, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int b = lane; b < nblk; b += 32) t += part[(size_t)c * nblk + b];
    for (int off = 16; off; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) s_llh = t;
  }
  const int g = threadIdx.x / P32, p = threadIdx.x - g * P32;
  if (m) {
    if (g == 0) d[p] = p < P ? (float)(prop[(size_t)c * P + p] - m[p]) : 0.f;
    __syncthreads();
    const int ks = (P + G - 1) / G;
    if (p < P) {
      float u[4];
      column_sum<4>(icov, P, p, d, g * ks, min(P, (g + 1) * ks), u);
      up[g * P32 + p] = (u[0] + u[1]) + (u[2] + u[3]);
    }
    __syncthreads();
    if (g == 0) {
      float u = 0.f;
      for (int q = 0; q < G; ++q) u += (p < P) ? up[q * P32 + p] : 0.f;
      red[p] = d[p] * u;
    }
  }
  __syncthreads();
  double pen = 0.0;
  if (m && threadIdx.x < 32) pen = warp_sum(red, P32);
  if (threadIdx.x == 0) {
    const double fn = s_llh + pen;
    int take;
    if (first) {
      f[c] = fn;
      take = 0;
    } else {
      const double u = u01(hash4(seed, step, c, 0xFFFFFFFFull));
      take = log(u) < -(fn - f[c]) * 0.5;  // NaN proposals are rejected
      if (take) {
        f[c] = fn;
        n_acc[c] += 1;
      }
    }
    s_take = take;
  }
  __syncthreads();
  if (s_take)
    for (int q = threadIdx.x; q < P; q += blockDim.x) phi[(size_t)c * P + q] = prop[(size_t)c * P + q];
}

}  // namespace
}  // namespace gwm

// Chain state on the device (sized at gwm_set_chain).
struct gwm_chain_state {
  int P = 0;
  bool prior = false;
  float *Lt = nullptr, *icov = nullptr;
  double *m = nullptr, *phi = nullptr, *f = nullptr;
  int32_t* nacc = nullptr;
};

static void chain_free(gwm_chain_state* s) {
  if (!s) return;
  cudaFree(s->Lt);
  cudaFree(s->m);
  cudaFree(s->icov);
  cudaFree(s->phi);
  cudaFree(s->f);
  cudaFree(s->nacc);
  delete s;
}

// Evaluates the surrogate of the first C rows of h_theta (device) up to the
// per-block likelihood partials h_part.  Rows C..roundup(C, 8) of h_theta must
// be finite.
static int surrogate_llh_device(gwm_net* n, int C, int llh_type) {
  const int din = n->dims[0];
  const int Bp = ((C + 7) / 8) * 8;
  gwm::k_standardize<<<(unsigned)(((size_t)Bp * din + 255) / 256), 256, 0, n->stream>>>(
      n->h_theta, Bp, din, n->h_mean, n->h_scale, n->xin, n->h[0]);
  GWM_CUDA(n, cudaGetLastError());
  const int rc = forward(n, Bp, kKeepNone);
  if (rc) return rc;
  return head_llh(n, C, llh_type, false, false);
}

// Proposal Cholesky factor L [P x P] (lower, row-major, host FP64) and the
// Gaussian prior (mean [P], inverse covariance [P x P]; both null for none)
// of the sub-chains; P == dims[0].  Room for up to batch_max chains.
extern "C" int gwm_set_chain(gwm_net* n, const double* prop_chol, const double* prior_mean,
                             const double* prior_icov) {
  if (!n || !prop_chol || ((prior_mean == nullptr) != (prior_icov == nullptr)))
    return gwm_fail(n, GW_ERR_ARG, "gwm_set_chain: bad arguments");
  if (!n->has_head) return gwm_fail(n, GW_ERR_STATE, "gwm_set_chain: gwm_set_head first");
  if (n->dims[0] > 1024) return gwm_fail(n, GW_ERR_LIMIT, "gwm_set_chain: at most 1024 parameters");
  GWM_CUDA(n, cudaSetDevice(n->device));
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  const int P = n->dims[0], Cm = n->batch_max;
  gwm_chain_state* s = n->chain;
  if (!s) {
    s = new gwm_chain_state();
    s->P = P;
    bool ok = cudaMalloc(&s->Lt, sizeof(float) * P * P) == cudaSuccess &&
              cudaMalloc(&s->m, sizeof(double) * P) == cudaSuccess &&
              cudaMalloc(&s->icov, sizeof(float) * P * P) == cudaSuccess &&
              cudaMalloc(&s->phi, sizeof(double) * (size_t)Cm * P) == cudaSuccess &&
              cudaMalloc(&s->f, sizeof(double) * Cm) == cudaSuccess &&
              cudaMalloc(&s->nacc, sizeof(int32_t) * Cm) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      chain_free(s);
      return gwm_fail(n, GW_ERR_NOMEM, "gwm_set_chain: cudaMalloc failed");
    }
    n->chain = s;
  }
  std::vector<float> lt((size_t)P * P), icov;
  for (int p = 0; p < P; ++p)
    for (int k = 0; k < P; ++k) lt[(size_t)k * P + p] = (float)prop_chol[(size_t)p * P + k];
  int rc = gwm_upload(n, s->Lt, lt.data(), lt.size());
  s->prior = prior_mean != nullptr;
  if (s->prior) {
    // symmetric: C^-1 [k][p] read as column p; symmetrised in FP64 first
    icov.resize((size_t)P * P);
    for (int p = 0; p < P; ++p)
      for (int k = 0; k < P; ++k)
        icov[(size_t)k * P + p] = (float)(0.5 * (prior_icov[(size_t)k * P + p] + prior_icov[(size_t)p * P + k]));
    rc |= gwm_upload(n, s->m, prior_mean, P) | gwm_upload(n, s->icov, icov.data(), icov.size());
  }
  GWM_CUDA(n, cudaStreamSynchronize(n->stream));
  return rc;
}

// Runs n_sub surrogate Metropolis steps for C chains from theta0 [C x P]
// (host FP64) with surrogate values f0 [C] (stat LLH + prior penalty, host;
// null: computed first, on the device).  Writes the end points phi [C x P],
// their surrogate values fphi [C] and the accepted sub-steps n_acc [C].
// n_sub == 0 with f0 == null evaluates the surrogate at theta0.
extern "C" int gwm_substeps(gwm_net* n, const double* theta0, const double* f0, int32_t C, int32_t n_sub,
                            int32_t llh_type, uint64_t seed, double* phi, double* fphi, int32_t* n_acc) {
  if (!n || !theta0 || !phi || !fphi || C < 1 || C > n->batch_max || n_sub < 0)
    return gwm_fail(n, GW_ERR_ARG, "gwm_substeps: bad arguments");
  gwm_chain_state* s = n->chain;
  if (!s || !n->has_head) return gwm_fail(n, GW_ERR_STATE, "gwm_substeps: gwm_set_chain first");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int P = s->P;
  const int Bp = ((C + 7) / 8) * 8;
  // G thread groups of P32 threads per chain split the k-range of the
  // proposal and penalty mat-vecs
  const int P32 = (P + 31) & ~31;
  const int G = std::max(1, std::min(4, 1024 / P32));
  const unsigned thr = (unsigned)(G * P32);
  const bool prior = s->prior;
  const size_t sh_prop = sizeof(float) * ((size_t)P + 1 + (size_t)G * P32);
  GWM_CUDA(n, cudaMemcpyAsync(s->phi, theta0, sizeof(double) * (size_t)C * P, cudaMemcpyHostToDevice, n->stream));
  GWM_CUDA(n, cudaMemsetAsync(s->nacc, 0, sizeof(int32_t) * C, n->stream));
  // rows C..Bp of the staging buffer stay finite (zeros)
  if (Bp > C)
    GWM_CUDA(n, cudaMemsetAsync(n->h_theta + (size_t)C * P, 0, sizeof(double) * (size_t)(Bp - C) * P, n->stream));
  int rc = GW_OK;
  const int nbx = head_parts(n);
  const size_t sh_fin = sizeof(float) * ((size_t)P32 * (G + 2));
  if (f0) {
    GWM_CUDA(n, cudaMemcpyAsync(s->f, f0, sizeof(double) * C, cudaMemcpyHostToDevice, n->stream));
  } else {
    GWM_CUDA(n, cudaMemcpyAsync(n->h_theta, s->phi, sizeof(double) * (size_t)C * P, cudaMemcpyDeviceToDevice,
                                n->stream));
    rc = surrogate_llh_device(n, C, llh_type);
    if (rc) return rc;
    launch_dependent(gwm::k_finish_accept, C, thr, sh_fin, n->stream,
                     n->h_part, nbx, s->phi, P, prior ? s->m : nullptr, s->icov, seed, 0, 1, s->phi, s->f, s->nacc);
    GWM_CUDA(n, cudaGetLastError());
  }
  // rows C..Bp of the first GEMM's input stay zero through the sub-steps
  if (Bp > C) GWM_CUDA(n, cudaMemsetAsync(n->h[0] + (size_t)C * P, 0, sizeof(bf16) * (size_t)(Bp - C) * P, n->stream));
  for (int st = 0; st < n_sub && rc == GW_OK; ++st) {
    launch_dependent(gwm::k_propose_stage, C, thr, sh_prop, n->stream,
                     s->phi, P, s->Lt, seed, (uint64_t)st + 1, n->h_theta, n->h_mean, n->h_scale, n->xin, n->h[0]);
    GWM_CUDA(n, cudaGetLastError());
    rc = forward(n, Bp, kKeepNone);
    if (!rc) rc = head_llh(n, C, llh_type, false, false);
    if (rc) break;
    launch_dependent(gwm::k_finish_accept, C, thr, sh_fin, n->stream,
                     n->h_part, nbx, n->h_theta, P, prior ? s->m : nullptr, s->icov, seed, (uint64_t)st + 1, 0, s->phi,
                     s->f, s->nacc);
    GWM_CUDA(n, cudaGetLastError());
  }
  if (rc) return rc;
  GWM_CUDA(n, cudaMemcpyAsync(phi, s->phi, sizeof(double) * (size_t)C * P, cudaMemcpyDeviceToHost, n->stream));
  GWM_CUDA(n, cudaMemcpyAsync(fphi, s->f, sizeof(double) * C, cudaMemcpyDeviceToHost, n->stream));
  if (n_acc) GWM_CUDA(n, cudaMemcpyAsync(n_acc, s->nacc, sizeof(int32_t) * C, cudaMemcpyDeviceToHost, n->stream));
  return check_status(n);
}

// ---------------------------------------------------------------------------
// Gradient of the surrogate -2 log L (plus the chain's prior penalty, when
// gwm_set_chain gave one) with respect to the parameters.
// ---------------------------------------------------------------------------
// dX of the network for dY in dz[L-1]: the backward GEMMs without the weight
// gradients; the input gradient lands in g_dx (FP32).
static int backward_dx(gwm_net* n, int B) {
  const int L = n->n_layers;
  for (int l = L - 1; l >= 1; --l) {
    gwm::Epilogue e{};
    e.gate = n->z[l - 1];
    e.out_bf16 = n->dz[l - 1];
    e.b_ready = 1;
    int rc = gemm(n, n->dz[l], n->wt[l], B, n->dims[l], n->dims[l + 1], e);
    if (rc) return rc;
  }
  gwm::Epilogue e0{};
  e0.out_f32 = n->g_dx;
  e0.b_ready = 1;
  return gemm(n, n->dz[0], n->wt[0], B, n->dims[0], n->dims[1], e0);
}

extern "C" int gwm_value_grad(gwm_net* n, const double* theta, int32_t C, int32_t llh_type, double* f, double* grad) {
  if (!n || !theta || !f || !grad || C < 1 || C > n->batch_max) return gwm_fail(n, GW_ERR_ARG, "gwm_value_grad: bad batch");
  if (!n->has_head) return gwm_fail(n, GW_ERR_STATE, "gwm_value_grad: gwm_set_head first");
  if (n->dims[0] > 1024) return gwm_fail(n, GW_ERR_LIMIT, "gwm_value_grad: at most 1024 parameters");
  GWM_CUDA(n, cudaSetDevice(n->device));
  const int din = n->dims[0], nb = n->dims[n->n_layers], L = n->n_layers, Bm = n->batch_max;
  const int Bp = ((C + 7) / 8) * 8;
  if (Bp > Bm) return gwm_fail(n, GW_ERR_ARG, "gwm_value_grad: batch above batch_max after padding");
  if (!n->g_G) {
    int rc = gwm_alloc(n, &n->g_G, (size_t)Bm * nb) | gwm_alloc(n, &n->g_S, (size_t)Bm * nb) |
             gwm_alloc(n, &n->g_gz, (size_t)Bm * din * 8) | gwm_alloc(n, &n->g_dx, (size_t)Bm * din) |
             gwm_alloc(n, &n->g_f, Bm) | gwm_alloc(n, &n->g_grad, (size_t)Bm * din);
    if (rc) return rc;
  }
  if (!n->side) GWM_CUDA(n, cudaStreamCreateWithFlags(&n->side, cudaStreamNonBlocking));
  if (!n->side_go) GWM_CUDA(n, cudaEventCreateWithFlags(&n->side_go, cudaEventDisableTiming));
  if (!n->side_done) GWM_CUDA(n, cudaEventCreateWithFlags(&n->side_done, cudaEventDisableTiming));
  if (Bp > C) GWM_CUDA(n, cudaMemsetAsync(n->h_theta, 0, sizeof(double) * (size_t)Bp * din, n->stream));
  GWM_CUDA(n, cudaMemcpyAsync(n->h_theta, theta, sizeof(double) * (size_t)C * din, cudaMemcpyHostToDevice, n->stream));
  gwm::k_standardize<<<(unsigned)(((size_t)Bp * din + 255) / 256), 256, 0, n->stream>>>(
      n->h_theta, Bp, din, n->h_mean, n->h_scale, n->xin, n->h[0]);
  GWM_CUDA(n, cudaGetLastError());
  int rc = forward(n, Bp, kKeepZ);
  if (rc) return rc;
  // the head: likelihood partials, G, S and dY (rows C..Bp of dY are zero)
  if (Bp > C)
    GWM_CUDA(n, cudaMemsetAsync(n->dz[L - 1] + (size_t)C * nb, 0, sizeof(bf16) * (size_t)(Bp - C) * nb, n->stream));
  const int nbx = head_parts(n);
  gwm::HeadOut out{};
  out.part = n->h_part;
  out.G = n->g_G;
  out.S = n->g_S;
  out.dy = n->dz[L - 1];
  rc = launch_head<true>(n, C, llh_type, out);
  if (rc) return rc;
  // The base's gradient and the network's input gradient need only the head's
  // results: the first bounds 152 SMs by shared-memory reads (33 us at 64 points,
  // 200 parameters, 3000 bins), the second is a chain of four latency-bound
  // products on 7 to 16 SMs (27 us), so they run side by side (a call 215 -> 195
  // us; 16 parameters, 200 bins, one point: 117 either way).  Whatever fails, the
  // network's stream goes on only after both.
  GWM_CUDA(n, cudaEventRecord(n->side_go, n->stream));
  GWM_CUDA(n, cudaStreamWaitEvent(n->side, n->side_go, 0));
  rc = launch_base_grad(n, C, n->side);
  const cudaError_t rec = cudaEventRecord(n->side_done, n->side);
  const int rc2 = rc ? rc : backward_dx(n, Bp);
  GWM_CUDA(n, rec);
  GWM_CUDA(n, cudaStreamWaitEvent(n->stream, n->side_done, 0));
  if (rc2) return rc2;
  const int P32 = (din + 31) & ~31;
  const int Gn = std::max(1, std::min(4, 1024 / P32));
  const bool prior = n->chain && n->chain->prior;
  launch_dependent(gwm::k_grad_finish, C, (unsigned)(Gn * P32), sizeof(float) * (size_t)P32 * (Gn + 2), n->stream,
                   n->h_part, nbx, n->h_theta, din, n->h_scale, n->g_gz, n->g_dx, prior ? n->chain->m : nullptr,
                   prior ? n->chain->icov : nullptr, n->g_f, n->g_grad);
  GWM_CUDA(n, cudaGetLastError());
  GWM_CUDA(n, cudaMemcpyAsync(f, n->g_f, sizeof(double) * C, cudaMemcpyDeviceToHost, n->stream));
  GWM_CUDA(n, cudaMemcpyAsync(grad, n->g_grad, sizeof(double) * (size_t)C * din, cudaMemcpyDeviceToHost, n->stream));
  return check_status(n);
}
