// mlp.cu — the surrogate network: 4 -> 128 -> 128 -> 128 -> 3, BF16 weights
// and activations, FP32 accumulation and FP32 master weights (Adam).
//
// Outputs: y0 = sigmoid(z0) (EAD probability), y1 = z1 (normalised APD90
// mean), y2 = softplus(z2) (normalised APD90 variance).  Loss per sample:
// BCE(y0, p) + (y1 - m)^2 + (y2 - s)^2, averaged over the batch.
//
// One kernel, mlp_rows, runs a whole pass: each CTA keeps the network's
// weights in shared memory and takes tiles of 128 samples through every layer
// (and, in training, back through every layer and into the weight gradients)
// with the products on Blackwell's 5th-generation tensor cores (tcgen05.mma,
// BF16 x BF16 -> FP32 accumulators in tensor memory).  Nothing but inputs,
// outputs and gradients touches global memory.  A second kernel,
// mlp_finish, adds the CTAs' gradients in order and takes the Adam step.
// gemm_tc and gemm_bf16 are general strided GEMMs on tcgen05 and mma.sync,
// each other's check (rh_mlp_gemm_check).
// Padded shapes: layer 1 K = 16 (4 inputs + zeros), layer 4 N = 8 (3
// outputs + zeros; the tcgen05 MMA pads N to 16).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <string>

#include "../../include/rh_mlp.h"

namespace {

constexpr int H = 128;   // hidden width
constexpr int KIN = 16;  // padded input width
constexpr int NOUT = 8;  // padded output width

// C[M,N] (f32, row-major, ldc) = sum_k A(m,k) B(k,n); A(m,k) = A[m*sam + k*sak],
// B(k,n) = Bm[k*sbk + n*sbn]; out-of-range elements read as zero.
// One warp per 16 x 8 output tile.
__global__ void gemm_bf16(const __nv_bfloat16* __restrict__ A, int sam, int sak,
                          const __nv_bfloat16* __restrict__ Bm, int sbk, int sbn, float* C, int ldc,
                          int M, int N, int K, int accumulate) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles_n = (N + 7) / 8;
  const int tm = warp / tiles_n, tn = warp % tiles_n;
  if (tm * 16 >= M) return;
  const int g = lane >> 2, tq = lane & 3;
  const int m0 = tm * 16, n0 = tn * 8;
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  auto ldA = [&](int m, int k) -> __nv_bfloat16 {
    return (m < M && k < K) ? A[(int64_t)m * sam + (int64_t)k * sak] : __float2bfloat16(0.f);
  };
  auto ldB = [&](int k, int n) -> __nv_bfloat16 {
    return (k < K && n < N) ? Bm[(int64_t)k * sbk + (int64_t)n * sbn] : __float2bfloat16(0.f);
  };
  auto pack = [](__nv_bfloat16 lo, __nv_bfloat16 hi) -> uint32_t {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
  };
  for (int k0 = 0; k0 < K; k0 += 16) {
    const int ka = k0 + tq * 2;
    uint32_t a0 = pack(ldA(m0 + g, ka), ldA(m0 + g, ka + 1));
    uint32_t a1 = pack(ldA(m0 + g + 8, ka), ldA(m0 + g + 8, ka + 1));
    uint32_t a2 = pack(ldA(m0 + g, ka + 8), ldA(m0 + g, ka + 9));
    uint32_t a3 = pack(ldA(m0 + g + 8, ka + 8), ldA(m0 + g + 8, ka + 9));
    uint32_t b0 = pack(ldB(ka, n0 + g), ldB(ka + 1, n0 + g));
    uint32_t b1 = pack(ldB(ka + 8, n0 + g), ldB(ka + 9, n0 + g));
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
  const int r0 = m0 + g, r1 = m0 + g + 8, cc = n0 + tq * 2;
  float* out[4] = {C + (int64_t)r0 * ldc + cc, C + (int64_t)r0 * ldc + cc + 1,
                   C + (int64_t)r1 * ldc + cc, C + (int64_t)r1 * ldc + cc + 1};
  const bool ok[4] = {r0 < M && cc < N, r0 < M && cc + 1 < N, r1 < M && cc < N,
                      r1 < M && cc + 1 < N};
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (ok[q]) *out[q] = accumulate ? *out[q] + c[q] : c[q];
}

// ---- the same GEMM on the 5th-generation tensor cores (tcgen05) ----
//
// One CTA of 128 threads per 128-row tile of C, every column of C (N <= 256).
// K is staged in chunks of 128 elements: the threads copy A (128 x 128) and
// B (N x 128, as the MMA's N x K operand) from global memory into shared
// memory in the canonical K-major layout without swizzle (core matrices of 8
// rows x 16 bytes), one elected thread issues eight tcgen05.mma (M = 128,
// N = the padded width, K = 16 each) into an FP32 accumulator in tensor
// memory and commits them to an mbarrier, and the next chunk is staged once
// they have read shared memory.  Each warp then reads its 32 accumulator
// rows with tcgen05.ld and writes C.  Out-of-range elements read as zero.
// Every wait on the mbarrier is bounded: on expiry the CTA sets *err, skips
// the rest of its MMAs, waits once more (bounded again) for those in flight and
// frees its tensor memory.
namespace tc {

constexpr int kM = 128;   // rows per CTA = tensor-memory lanes
constexpr int kKc = 128;  // K elements per staged chunk
constexpr int kNmax = 128;
constexpr int kSmemA = kM * kKc * 2;      // bytes
constexpr int kSmemB = kNmax * kKc * 2;
// Polls of an mbarrier before a wait gives up: the hardware holds a poll for up
// to 3.75 us while nothing arrives (2^22 of them took 15.7 s), so 1 s in all.
constexpr int kWaitLimit = 1 << 18;

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor of tcgen05: start address, the byte
// distance between core matrices adjacent along K (lbo) and along M or N
// (sbo), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// Byte offset of element (row, k) of a staged operand with `rows` rows
// (a multiple of 8): core matrix (row / 8, k / 8) at ((k/8) * rows/8 +
// row/8) * 128, row % 8 at 16-byte steps, k % 8 at 2-byte steps.
__device__ __forceinline__ uint32_t core_off(int row, int k, int rows) {
  return (uint32_t)(((k >> 3) * (rows >> 3) + (row >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int it = 0; it < kWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace tc

// C[M,N] (f32, row-major, ldc) = sum_k A(m,k) B(k,n) (+ C when accumulate),
// with A and B addressed as in gemm_bf16; N <= 128.  The general form of the
// products mlp_rows takes on its own tiles, reached through rh_mlp_gemm_check.
__global__ void __launch_bounds__(128, 1)
    gemm_tc(const __nv_bfloat16* __restrict__ A, int sam, int sak,
            const __nv_bfloat16* __restrict__ Bm, int sbk, int sbn, float* C, int ldc, int M,
            int N, int K, int accumulate, int* err) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_base;
  unsigned char* sA = smem;
  unsigned char* sB = smem + tc::kSmemA;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * tc::kM;
  const int Nm = (N + 15) & ~15;                 // MMA width: a multiple of 16
  const uint32_t ncols = Nm <= 32 ? 32u : (Nm <= 64 ? 64u : 128u);  // power of two >= 32
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc::saddr(&bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::saddr(&tmem_base)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = tc::instr_desc(tc::kM, Nm);
  bool ok = true;
  const int nchunks = (K + tc::kKc - 1) / tc::kKc;
  int ch = 0;
  for (; ch < nchunks && ok; ++ch) {
    const int k0 = ch * tc::kKc;
    // stage A (128 x 128) and B (Nm x 128) as 16-byte core-matrix rows
    for (int c = tid; c < tc::kM * (tc::kKc / 8); c += blockDim.x) {
      const int r = c % tc::kM, kg = c / tc::kM;
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat16 lo = __float2bfloat16(0.f), hi = lo;
        const int m = m0 + r, k = k0 + kg * 8 + 2 * j;
        if (m < M && k < K) lo = A[(int64_t)m * sam + (int64_t)k * sak];
        if (m < M && k + 1 < K) hi = A[(int64_t)m * sam + (int64_t)(k + 1) * sak];
        w[j] = (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
      }
      *reinterpret_cast<uint4*>(sA + tc::core_off(r, kg * 8, tc::kM)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    for (int c = tid; c < Nm * (tc::kKc / 8); c += blockDim.x) {
      const int n = c % Nm, kg = c / Nm;
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat16 lo = __float2bfloat16(0.f), hi = lo;
        const int k = k0 + kg * 8 + 2 * j;
        if (n < N && k < K) lo = Bm[(int64_t)k * sbk + (int64_t)n * sbn];
        if (n < N && k + 1 < K) hi = Bm[(int64_t)(k + 1) * sbk + (int64_t)n * sbn];
        w[j] = (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
      }
      *reinterpret_cast<uint4*>(sB + tc::core_off(n, kg * 8, Nm)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    // the staged operands become visible to the tensor core's (async) proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a0 = tc::saddr(sA), b0 = tc::saddr(sB);
      // K-adjacent core matrices are rows/8 * 128 bytes apart, M/N-adjacent 128
      const uint32_t lbo_a = (tc::kM / 8) * 128, lbo_b = (uint32_t)(Nm / 8) * 128;
#pragma unroll
      for (int s = 0; s < tc::kKc / 16; ++s) {
        const uint64_t ad = tc::smem_desc(a0 + (uint32_t)s * 2 * lbo_a, lbo_a, 128);
        const uint64_t bd = tc::smem_desc(b0 + (uint32_t)s * 2 * lbo_b, lbo_b, 128);
        const uint32_t acc = (ch > 0 || s > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              tc::saddr(&bar))
          : "memory");
    }
    // every thread saw the MMAs finish (or the wait give up) before the next
    // chunk is staged; the outcome is the same in every thread
    ok = __syncthreads_and(tc::mbar_wait(tc::saddr(&bar), (uint32_t)(ch & 1)) ? 1 : 0) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (!ok) {
    if (tid == 0) atomicOr(err, 1);
    tc::mbar_wait(tc::saddr(&bar), (uint32_t)((ch - 1) & 1));  // the last commit's phase
  } else {
    // epilogue: warp w reads accumulator rows 32w..32w+31 (its tensor-memory lanes)
    const int row = m0 + warp * 32 + lane;
    for (int c0 = 0; c0 < Nm; c0 += 16) {
      uint32_t v[16];
      const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
          "%14,%15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
            "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
            "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(ta)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (row < M) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = c0 + j;
          if (col < N) {
            float* o = C + (int64_t)row * ldc + col;
            const float x = __uint_as_float(v[j]);
            *o = accumulate ? *o + x : x;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// ---- the parameter vector (rh_mlp.h) and its BF16 image ----
constexpr int kW1 = 0, kB1 = kW1 + H * KIN, kW2 = kB1 + H, kB2 = kW2 + H * H, kW3 = kB2 + H,
              kB3 = kW3 + H * H, kW4 = kB3 + H, kB4 = kW4 + NOUT * H, kNPar = kB4 + NOUT;
constexpr int NPAD = 16;  // output rows of the MMA
// The image holds the four weight matrices as the MMA's operands: element
// (row, k) of a matrix of `rows` rows at tc::core_off(row, k, rows), so that
// a CTA's copy is one contiguous bulk copy.
constexpr int kImg1 = 0, kImg2 = kImg1 + H * KIN * 2, kImg3 = kImg2 + H * H * 2,
              kImg4 = kImg3 + H * H * 2, kImgBytes = kImg4 + NPAD * H * 2;

// Layer of parameter i, and for a weight its row, column and image offset.
struct ParamPlace {
  int img;      // byte offset in the image, -1 for a bias
  bool padded;  // a padding weight: always zero
};
__device__ __forceinline__ ParamPlace place_of(int i) {
  if (i < kB1) {
    const int r = i / KIN, k = i % KIN;
    return {kImg1 + (int)tc::core_off(r, k, H), k >= RH_MLP_IN};
  }
  if (i >= kW2 && i < kB2) {
    const int j = i - kW2;
    return {kImg2 + (int)tc::core_off(j / H, j % H, H), false};
  }
  if (i >= kW3 && i < kB3) {
    const int j = i - kW3;
    return {kImg3 + (int)tc::core_off(j / H, j % H, H), false};
  }
  if (i >= kW4 && i < kB4) {
    const int j = i - kW4;
    return {kImg4 + (int)tc::core_off(j / H, j % H, NPAD), j / H >= RH_MLP_OUT};
  }
  return {-1, false};
}

constexpr int kRowThreads = 512;  // of a mlp_rows CTA
// A forward pass with held outputs (HELD below) is one cluster.
constexpr int kHeldCtas = 8;  // the largest cluster every device takes
constexpr int kHeldTiles = RH_MLP_NOALLOC_MAX_BATCH / 128 / kHeldCtas;
static_assert(kHeldTiles * kHeldCtas * 128 == RH_MLP_NOALLOC_MAX_BATCH, "whole tiles");

// ---- shared memory of mlp_rows ----
struct RowsSmem {
  static constexpr int kW = 0;                       // the image
  static constexpr int kX0 = kW + kImgBytes;         // packed inputs, 128 x 16
  static constexpr int kA = kX0 + 128 * KIN * 2;     // activations, 128 x 128 each
  static constexpr int kTile = 128 * H * 2;
  // forward only: one activation tile, overwritten layer by layer
  static constexpr int kBiasF = kA + kTile;
  // training: three activation tiles, the dZ tile, dZ4, the column sums
  static constexpr int kD = kA + 3 * kTile;
  static constexpr int kD4 = kD + kTile;
  static constexpr int kRed = kD4 + 128 * NPAD * 2;  // float[3][4][128]
  static constexpr int kBiasT = kRed + 3 * 4 * H * 4;
  static constexpr int kBiasBytes = (3 * H + NOUT) * 4;
  // forward with held outputs: those of the CTA's tiles, float[kHeldTiles][128][3]
  static constexpr int kHeld = kBiasF + kBiasBytes;
  static constexpr int bytes(bool train) { return (train ? kBiasT : kBiasF) + kBiasBytes; }
  static constexpr int bytes_held() { return kHeld + kHeldTiles * 128 * RH_MLP_OUT * 4; }
};
static_assert(RowsSmem::bytes(true) <= 227 * 1024, "shared memory of a CTA");

struct RowsArgs {
  const unsigned char* img;  // BF16 image; nullptr: converted from params in the kernel
  const float* params;       // FP32 vector
  const float* x;            // n x 4
  const float* target;       // n x 3 (training)
  float* y;                  // n x 3 (forward)
  float* loss;               // n loss terms (training)
  float* part;               // [gridDim.x][kNPar] gradients (training)
  int n;
  int* err;                  // set when a wait gave up; nullptr: y becomes NaN
  int* failed;               // the same for mlp_finish, in device memory (training)
};

// One MMA chain: K = 16 ksteps, descriptors advancing by da and db bytes.
__device__ __forceinline__ void mma_chain(uint32_t acc, uint32_t a, uint32_t a_lbo, uint32_t a_sbo,
                                          uint32_t da, uint32_t b, uint32_t b_lbo, uint32_t b_sbo,
                                          uint32_t db, uint32_t idesc, int ksteps, bool add) {
  for (int s = 0; s < ksteps; ++s) {
    const uint64_t ad = tc::smem_desc(a + s * da, a_lbo, a_sbo);
    const uint64_t bd = tc::smem_desc(b + s * db, b_lbo, b_sbo);
    const uint32_t on = (add || s > 0) ? 1u : 0u;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc),
        "l"(ad), "l"(bd), "r"(idesc), "r"(on)
        : "memory");
  }
}

__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                 "=r"(v[6]), "=r"(v[7])
               : "r"(addr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16(lo)) |
         ((uint32_t)__bfloat16_as_ushort(__float2bfloat16(hi)) << 16);
}

// 32 values of one row, columns col.., to BF16 in an operand tile of 128 rows.
__device__ __forceinline__ void store_row32(unsigned char* tile, int row, int col,
                                            const float (&v)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 w;
    w.x = pack_bf16(v[8 * q], v[8 * q + 1]);
    w.y = pack_bf16(v[8 * q + 2], v[8 * q + 3]);
    w.z = pack_bf16(v[8 * q + 4], v[8 * q + 5]);
    w.w = pack_bf16(v[8 * q + 6], v[8 * q + 7]);
    *reinterpret_cast<uint4*>(tile + tc::core_off(row, col + 8 * q, 128)) = w;
  }
}

// Sum over the warp's lanes of each of 32 values: lane i returns the sum of
// v[i] (a halving exchange, 31 shuffles).
__device__ __forceinline__ float column_sums(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      const float give = up ? v[i] : v[i + off];
      const float keep = up ? v[i + off] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  return v[0];
}

// The caller's FP32 weights as the BF16 image (what mlp_load writes), eight
// weights of a row at a time; a warp takes 16 rows of two neighbouring groups
// of eight, whose loads fill 64-byte segments and whose stores conflict twice.
__device__ __forceinline__ void image_from_params(const float* params, unsigned char* img,
                                                  int tid) {
  const bool aligned = (reinterpret_cast<uintptr_t>(params) & 15) == 0;
  for (int i = tid; i < kImgBytes / 16; i += kRowThreads) {
    int row, k, src, rows = H, rvalid = H, kvalid = H, base;
    if (i < kImg2 / 16) {
      row = i >> 1;
      k = (i & 1) * 8;
      src = kW1 + row * KIN + k;
      kvalid = RH_MLP_IN;
      base = kImg1;
    } else if (i < kImg4 / 16) {
      const int j = (i - kImg2 / 16) & 2047, l = (i - kImg2 / 16) >> 11;
      row = ((j >> 1) & 15) | ((j >> 8) << 4);
      k = ((j & 1) | (((j >> 5) & 7) << 1)) * 8;
      src = (l == 0 ? kW2 : kW3) + row * H + k;
      base = l == 0 ? kImg2 : kImg3;
    } else {
      const int j = i - kImg4 / 16;
      row = j >> 4;
      k = (j & 15) * 8;
      src = kW4 + row * H + k;
      rows = NPAD;
      rvalid = RH_MLP_OUT;
      base = kImg4;
    }
    float v[8];
    if (row >= rvalid) {  // padding rows; those past the vector's are not read
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = 0.f;
    } else if (aligned) {
      const float4 lo = *reinterpret_cast<const float4*>(params + src);
      const float4 hi = *reinterpret_cast<const float4*>(params + src + 4);
      v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w;
      v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = params[src + q];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (k + q >= kvalid) v[q] = 0.f;
    *reinterpret_cast<uint4*>(img + base + tc::core_off(row, k, rows)) =
        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                   pack_bf16(v[6], v[7]));
  }
}

// The network on tiles of 128 samples: CTA c takes tiles c, c + gridDim.x, ...
// with 512 threads; thread (row, quarter) owns one sample (a tensor-memory
// lane) and 32 of its 128 columns.
//
// What bounds it: a tile's arithmetic is a few microseconds of one SM's tensor
// cores, so a pass is the latency of its layers, one after the other: an MMA
// chain, a round trip to an mbarrier and an epilogue each (11 us forward, 13 us
// a tile in training, plus 14 us for the weights and the gradients).  So the
// layers run in one CTA with the activations in shared memory.  One launch per
// product, bias and activation, as before, cost 24 us of strided staging per
// product (500 us for a dW over 4,096 samples in one CTA) and ten to 25
// launches.  Whole calls, before and now: 65,536 predictions 2.20 ms and 94 us,
// an epoch of twelve 256-sample steps 5.50 and 0.83 ms, gradients of 4,096
// samples 2.04 ms and 55 us, the no-allocation forward of 1,000 samples 61 and
// 12 us.  256 threads (64 columns each) were slower: 44 us against 38 for two
// training tiles.
//
// Operands: every tile in shared memory is the no-swizzle core-matrix layout
// of 8 rows x 16 bytes, rows along samples (or output units).  Read K-major it
// is the forward operand (samples x features); the same bytes read MN-major
// (the instruction descriptor's transpose bits, with the two strides
// exchanged) are the transposed operands of dW = dZ^T A and dA = dZ W, so
// nothing is transposed or stored twice.
//
// HELD (forward, one cluster of CTAs): y may overlap x or the parameters.  The
// outputs stay in shared memory until every CTA has read its inputs, which a
// cluster barrier tells; without it a CTA's outputs could replace the inputs of
// one that has not started (4,096 samples 24.6 us; 12.3 with memory apart).
template <bool TRAIN, bool HELD = false>
__global__ void __launch_bounds__(kRowThreads, 1) mlp_rows(const RowsArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t bars[2];  // MMAs done; weights landed
  __shared__ uint32_t tmem_base;
  using S = RowsSmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp >> 2, row = (warp & 3) * 32 + lane, col = quarter * 32;
  float* bias = reinterpret_cast<float*>(sm + (TRAIN ? S::kBiasT : S::kBiasF));
  float* held = reinterpret_cast<float*>(sm + S::kHeld);  // HELD only
  constexpr uint32_t kCols = TRAIN ? 512u : 128u;
  const uint32_t mma_bar = tc::saddr(&bars[0]), w_bar = tc::saddr(&bars[1]);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mma_bar) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(w_bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (a.img) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_bar),
                   "r"((uint32_t)kImgBytes)
                   : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
              "r"(tc::saddr(sm + S::kW)),
          "l"(a.img), "r"((uint32_t)kImgBytes), "r"(w_bar)
          : "memory");
    }
  }
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::saddr(&tmem_base)),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = tid; i < 3 * H + NOUT; i += kRowThreads) {
    const int l = i / H, j = i % H;
    bias[i] = a.params[(l == 0 ? kB1 : l == 1 ? kB2 : l == 2 ? kB3 : kB4) + j];
  }
  if (!a.img) image_from_params(a.params, sm + S::kW, tid);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  bool ok = !a.img || tc::mbar_wait(w_bar, 0);
  // accumulators in tensor memory: the layer's product, then (training) dW2,
  // dW3, dW1 and dW4 (transposed: 128 inputs x 16 outputs)
  constexpr uint32_t kDW2 = 128, kDW3 = 256, kDW1 = 384, kDW4 = 400;
  constexpr uint32_t kTA = 1u << 15, kTB = 1u << 16;  // MN-major A, B
  const uint32_t id128 = tc::instr_desc(128, H), id16 = tc::instr_desc(128, NPAD);
  const uint32_t sw = tc::saddr(sm + S::kW), sx = tc::saddr(sm + S::kX0);
  const uint32_t w1 = sw + kImg1, w2 = sw + kImg2, w3 = sw + kImg3, w4 = sw + kImg4;
  // K-major operand of 128 rows: lbo 2048 (next 8 of K), sbo 128 (next 8
  // rows), 4096 a K step; MN-major: lbo 128, sbo 2048, 256 a K step
  constexpr uint32_t kL = 2048, kS = 128, kStep = 4096, kStepT = 256;
  uint32_t phase = 0;
  // makes the CTA's shared-memory writes visible to the tensor cores, then
  // thread 0 issues `mmas` and every thread waits for them; false (in every
  // thread, before any MMA of this call) once a wait has given up
  auto run_mmas = [&](auto mmas) -> bool {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!__syncthreads_and(ok ? 1 : 0)) return false;
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      mmas();
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              mma_bar)
          : "memory");
    }
    ok = tc::mbar_wait(mma_bar, phase);
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return true;
  };
  const bool x16 = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;
  const float inv_n = 1.f / (float)a.n;
  float db[4] = {0.f, 0.f, 0.f, 0.f};  // thread j < 128: column j of db1..3; db4 of thread j < 3
  const int tiles = (a.n + 127) / 128;
  bool first = true;
  auto one_tile = [&](int t) -> bool {
    const int r = t * 128 + row;
    const bool valid = r < a.n;
    if (quarter == 0) {  // inputs to BF16, zero-padded to 16
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (valid) {
        if (x16) {
          x = reinterpret_cast<const float4*>(a.x)[r];
        } else {
          const float* p = a.x + (size_t)r * RH_MLP_IN;
          x = make_float4(p[0], p[1], p[2], p[3]);
        }
      }
      const uint4 w = make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), 0u, 0u);
      *reinterpret_cast<uint4*>(sm + S::kX0 + tc::core_off(row, 0, 128)) = w;
      *reinterpret_cast<uint4*>(sm + S::kX0 + tc::core_off(row, 8, 128)) = make_uint4(0, 0, 0, 0);
    }
    uint32_t mask[3];  // z > 0 of this thread's columns
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      unsigned char* out = sm + S::kA + (TRAIN ? l : 0) * S::kTile;
      const uint32_t in = l == 0 ? sx : tc::saddr(sm + S::kA + (TRAIN ? l - 1 : 0) * S::kTile);
      const uint32_t w = l == 0 ? w1 : l == 1 ? w2 : w3;
      if (!run_mmas([&] {
            mma_chain(tmem, in, kL, kS, kStep, w, kL, kS, kStep, id128, l == 0 ? 1 : H / 16, false);
          }))
        return false;
      uint32_t raw[32];
      tmem_load32(lanes + col, raw);
      float v[32];
      uint32_t m = 0u;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float z = __uint_as_float(raw[j]) + bias[l * H + col + j];
        if (z > 0.f) m |= 1u << j;
        v[j] = z > 0.f ? z : 0.f;
      }
      mask[l] = m;
      store_row32(out, row, col, v);
    }
    // output layer
    const uint32_t a3 = tc::saddr(sm + S::kA + (TRAIN ? 2 : 0) * S::kTile);
    if (!run_mmas([&] {
          mma_chain(tmem, a3, kL, kS, kStep, w4, 256, kS, 512, id16, H / 16, false);
        }))
      return false;
    if (quarter == 0) {
      uint32_t raw[8];
      tmem_load8(lanes, raw);
      const float* b4 = bias + 3 * H;
      const float z0 = __uint_as_float(raw[0]) + b4[0], z1 = __uint_as_float(raw[1]) + b4[1],
                  z2 = __uint_as_float(raw[2]) + b4[2];
      const float y0 = sigmoidf_(z0), y1 = z1, y2 = softplusf_(z2);
      if constexpr (!TRAIN) {
        if (valid && ok) {
          float* y = HELD ? held + ((t / gridDim.x) * 128 + row) * RH_MLP_OUT
                          : a.y + (size_t)r * RH_MLP_OUT;
          y[0] = y0;
          y[1] = y1;
          y[2] = y2;
        }
      } else {
        float g0 = 0.f, g1 = 0.f, g2 = 0.f;  // dZ4, scaled by 1/n
        if (valid) {
          const float* tg = a.target + (size_t)r * RH_MLP_OUT;
          const float p = tg[0], m = tg[1], s = tg[2];
          const float e = 1e-7f;
          a.loss[r] = -(p * logf(fmaxf(y0, e)) + (1.f - p) * logf(fmaxf(1.f - y0, e))) +
                      (y1 - m) * (y1 - m) + (y2 - s) * (y2 - s);
          g0 = (y0 - p) * inv_n;
          g1 = 2.f * (y1 - m) * inv_n;
          g2 = 2.f * (y2 - s) * sigmoidf_(z2) * inv_n;
        }
        const uint4 w = make_uint4(pack_bf16(g0, g1), pack_bf16(g2, 0.f), 0u, 0u);
        *reinterpret_cast<uint4*>(sm + S::kD4 + tc::core_off(row, 0, 128)) = w;
        *reinterpret_cast<uint4*>(sm + S::kD4 + tc::core_off(row, 8, 128)) =
            make_uint4(0, 0, 0, 0);
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = j == 0 ? g0 : j == 1 ? g1 : j == 2 ? g2 : 0.f;
        const float s = column_sums(v, lane);
        db[3] += s;  // lane j < 3 of each of the four row groups; added up at the end
      }
    }
    if constexpr (TRAIN) {
      float* red = reinterpret_cast<float*>(sm + S::kRed);
      const uint32_t d4 = tc::saddr(sm + S::kD4), dd = tc::saddr(sm + S::kD);
      const uint32_t act[3] = {tc::saddr(sm + S::kA), tc::saddr(sm + S::kA + S::kTile),
                               tc::saddr(sm + S::kA + 2 * S::kTile)};
#pragma unroll
      for (int l = 2; l >= 0; --l) {
        // dW of the layer above (over the tile's 128 samples) and dA of this one
        if (!run_mmas([&] {
              if (l == 2) {
                mma_chain(tmem + kDW4, act[2], kS, kL, kStepT, d4, kS, kL, kStepT, id16 | kTA | kTB,
                          8, !first);
                mma_chain(tmem, d4, kL, kS, 0, w4, kS, 256, 0, id128 | kTB, 1, false);
              } else {
                mma_chain(tmem + (l == 1 ? kDW3 : kDW2), dd, kS, kL, kStepT, act[l], kS, kL, kStepT,
                          id128 | kTA | kTB, 8, !first);
                mma_chain(tmem, dd, kL, kS, kStep, l == 1 ? w3 : w2, kS, kL, kStepT, id128 | kTB, 8,
                          false);
              }
            }))
          return false;
        uint32_t raw[32];
        tmem_load32(lanes + col, raw);
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = (mask[l] >> j & 1u) ? __uint_as_float(raw[j]) : 0.f;
        store_row32(sm + S::kD, row, col, v);
        red[(l * 4 + (warp & 3)) * H + col + lane] = column_sums(v, lane);
      }
      if (!run_mmas([&] {
            mma_chain(tmem + kDW1, dd, kS, kL, kStepT, sx, kS, kL, kStepT, id16 | kTA | kTB, 8,
                      !first);
          }))
        return false;
      if (tid < H) {
#pragma unroll
        for (int l = 0; l < 3; ++l)
#pragma unroll
          for (int q = 0; q < 4; ++q) db[l] += red[(l * 4 + q) * H + tid];
      }
      first = false;
    }
    return true;
  };
  bool done = true;
  for (int t = blockIdx.x; t < tiles && done; t += gridDim.x) done = one_tile(t);
  done = __syncthreads_and((done && ok) ? 1 : 0) != 0;
  if constexpr (HELD) {  // every CTA arrives, whatever its waits gave
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (done)
      for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        for (int i = tid; i < 128 * RH_MLP_OUT; i += kRowThreads)
          if (t * 128 + i / RH_MLP_OUT < a.n)
            a.y[(size_t)t * 128 * RH_MLP_OUT + i] = held[(t / gridDim.x) * 128 * RH_MLP_OUT + i];
  }
  if (!done) {
    if (tid == 0 && a.err) *a.err = 1;  // host memory, read after a synchronisation
    if (TRAIN && tid == 0) *a.failed = 1;
    // nothing may still write this CTA's shared or tensor memory when it ends:
    // the weights' copy, the last MMAs committed (if none were, the phase
    // before the first counts as complete)
    if (a.img) tc::mbar_wait(w_bar, 0);
    tc::mbar_wait(mma_bar, phase ^ 1u);
    if (!TRAIN && !a.err)
      for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        for (int i = tid; i < 128 * RH_MLP_OUT; i += kRowThreads)
          if (t * 128 + i / RH_MLP_OUT < a.n)
            a.y[(size_t)t * 128 * RH_MLP_OUT + i] = __int_as_float(0x7fc00000);
  } else if constexpr (TRAIN) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float* g = a.part + (size_t)blockIdx.x * kNPar;
    // the lower two quarters write dW2 and dW1, the upper two dW3 and dW4
    // (64 columns of a thread's accumulator row each)
    const bool lower = quarter < 2;
    const int c0 = (quarter & 1) * 64;
    float* gw = g + (lower ? kW2 : kW3) + row * H + c0;
#pragma unroll 1
    for (int c = 0; c < 64; c += 32) {
      uint32_t raw[32];
      tmem_load32(lanes + (lower ? kDW2 : kDW3) + c0 + c, raw);
#pragma unroll
      for (int j = 0; j < 32; j += 4)  // parameter offsets are multiples of 4
        *reinterpret_cast<uint4*>(gw + c + j) =
            make_uint4(raw[j], raw[j + 1], raw[j + 2], raw[j + 3]);
    }
    {
      uint32_t raw[8];
      if (lower) {  // 8 of the 16 input columns
        const int q = quarter * 8;
        tmem_load8(lanes + kDW1 + q, raw);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[kW1 + row * KIN + q + j] = __uint_as_float(raw[j]);
      } else if (quarter == 2) {
        tmem_load8(lanes + kDW4, raw);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[kW4 + j * H + row] = __uint_as_float(raw[j]);
      }
    }
    if (tid < H) {
      g[kB1 + tid] = db[0];
      g[kB2 + tid] = db[1];
      g[kB3 + tid] = db[2];
    }
    float* red = reinterpret_cast<float*>(sm + S::kRed);
    __syncthreads();  // the sums of the last tile have been read
    if (quarter == 0 && lane < NOUT) red[(warp & 3) * NOUT + lane] = db[3];
    __syncthreads();
    if (tid < NOUT)
      g[kB4 + tid] = red[tid] + red[NOUT + tid] + red[2 * NOUT + tid] + red[3 * NOUT + tid];
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols)
                 : "memory");
}

// What follows a training pass: the CTAs' gradients added in order, then
// either written out or taken as one Adam step on the FP32 master weights,
// refreshing the BF16 image.  Padding weights stay zero.  After a pass whose
// wait gave up (`failed`), whose CTA has left no gradients, no step is taken.
struct AdamStep {
  float lr, b1, b2, eps, bc1, bc2;
};
__global__ void mlp_finish(const float* part, int nparts, float* grads, float* w, float* m, float* v,
                           unsigned char* img, const int* failed, AdamStep s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kNPar) return;
  float gi = 0.f;
  for (int c = 0; c < nparts; ++c) gi += part[(size_t)c * kNPar + i];
  if (grads) {
    grads[i] = gi;
    return;
  }
  const ParamPlace p = place_of(i);
  if (p.padded) return;
  const bool none = *failed != 0;  // read beside the moments, whose latency hides it
  const float mi = s.b1 * m[i] + (1.f - s.b1) * gi;
  const float vi = s.b2 * v[i] + (1.f - s.b2) * gi * gi;
  const float wi = w[i] - s.lr * (mi / s.bc1) / (sqrtf(vi / s.bc2) + s.eps);
  if (none) return;
  m[i] = mi;
  v[i] = vi;
  w[i] = wi;
  if (p.img >= 0) *reinterpret_cast<__nv_bfloat16*>(img + p.img) = __float2bfloat16(wi);
}

// New parameters in w: padding weights to zero, the BF16 image refreshed.
__global__ void mlp_load(float* w, unsigned char* img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kNPar) return;
  const ParamPlace p = place_of(i);
  if (p.padded) w[i] = 0.f;
  if (p.img >= 0) *reinterpret_cast<__nv_bfloat16*>(img + p.img) = __float2bfloat16(w[i]);
}

unsigned blocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ---------------------------------------------------------------- host side

constexpr int kChunk = 16384;    // samples of one forward launch
constexpr int kMaxParts = 152;   // CTAs of a training pass
// Largest batch of a handle: more pinned memory (24 bytes a sample) than that is
// no screening network's, and sample indices stay far from overflow.
constexpr int kMaxBatch = 1 << 26;

struct rh_mlp {
  int bmax = 0;
  int device = 0;
  cudaStream_t st = nullptr;
  float* P = nullptr;            // w, m, v, then the CTAs' gradients
  float *w = nullptr, *m = nullptr, *v = nullptr, *part = nullptr;
  unsigned char* img = nullptr;  // BF16 weights (kImgBytes), then `failed`
  // Host memory the kernels read and write directly (pinned, mapped): outputs
  // of two chunks or loss terms, gradients, the error flag; and, made when first
  // needed, copies of the caller's arrays (reachable(), below).
  unsigned char* host = nullptr;
  float *h_out = nullptr, *h_g = nullptr, *copies = nullptr;
  int* h_err = nullptr;          // set by a pass whose wait gave up
  int* failed = nullptr;         // and its copy for mlp_finish, on the device
  cudaEvent_t ev[2] = {nullptr, nullptr};
  bool direct = false;  // kernels can read pageable host memory (hardware page tables)
  int chunk = 0;        // samples of one forward launch
  int64_t step = 0;
  std::string err;
};

namespace {

int ck(rh_mlp* m, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return RH_OK;
  if (m) m->err = std::string(what) + ": " + cudaGetErrorString(e);
  return RH_ERR_CUDA;
}
#define MCK(x)                                 \
  do {                                         \
    int r_ = ck(m, (x), #x);                   \
    if (r_) return r_;                         \
  } while (0)

// After a stream synchronisation: RH_ERR_TIMEOUT when a pass's wait gave up.
int check_wait(rh_mlp* m) {
  if (*m->h_err) {
    *m->h_err = 0;
    MCK(cudaMemsetAsync(m->failed, 0, sizeof(int), m->st));
    m->err = "a wait for the tensor cores ran out";
    return RH_ERR_TIMEOUT;
  }
  return RH_OK;
}

// Where the kernels read `count` floats of the caller's `p`: in place, or
// from a pinned copy (kCopyX0, kCopyX1: inputs of a chunk; kCopyT: targets of
// a batch) on a device that cannot read pageable memory, and of an array that
// is not on a 4-byte boundary (numpy makes such arrays from the middle of a
// buffer), which would fault a kernel's loads.  In place is as fast or faster
// (a 65,536-point sweep 95 against 130 us, gradients of 4,096 samples 58
// against 64, a 256-sample step 70 either way).
enum CopySlot { kCopyX0, kCopyX1, kCopyT };
int reachable(rh_mlp* m, const float* p, size_t count, CopySlot slot, const float** out) {
  *out = p;
  if (m->direct && reinterpret_cast<uintptr_t>(p) % alignof(float) == 0) return RH_OK;
  const size_t nx = (size_t)m->chunk * RH_MLP_IN;
  if (!m->copies)
    MCK(cudaHostAlloc(reinterpret_cast<void**>(&m->copies),
                      (2 * nx + (size_t)m->bmax * RH_MLP_OUT) * sizeof(float),
                      cudaHostAllocMapped));
  float* to = m->copies + (size_t)slot * nx;
  memcpy(to, static_cast<const void*>(p), count * sizeof(float));
  *out = to;
  return RH_OK;
}

// One training pass: loss terms to h_out, each CTA's gradients to part.  A
// batch is spread a tile to a CTA; the short accumulations and the ordered FP32
// sum of the CTAs' gradients are more exact than one accumulator over the batch
// (4,096 samples: median error 8e-8 relative against 2e-6).  Up to two tiles
// are one CTA's work: one accumulator, so that a step of the default batch of
// 256 samples adds in the order in which it always has.  Two CTAs would save it
// about 13 of 41 us and change that order.
int train_pass(rh_mlp* m, const float* x, const float* target, int n, int* nparts) {
  const int tiles = (n + 127) / 128;
  *nparts = tiles <= 2 ? 1 : std::min(tiles, kMaxParts);
  RowsArgs a{};
  a.img = m->img;
  a.params = m->w;
  int r = reachable(m, x, (size_t)n * RH_MLP_IN, kCopyX0, &a.x);
  if (r == RH_OK) r = reachable(m, target, (size_t)n * RH_MLP_OUT, kCopyT, &a.target);
  if (r != RH_OK) return r;
  a.loss = m->h_out;
  a.part = m->part;
  a.n = n;
  a.err = m->h_err;
  a.failed = m->failed;
  mlp_rows<true><<<*nparts, kRowThreads, RowsSmem::bytes(true), m->st>>>(a);
  return ck(m, cudaGetLastError(), "training pass");
}

float mean_loss(const rh_mlp* m, int n) {
  double s = 0;
  for (int i = 0; i < n; ++i) s += m->h_out[i];
  return (float)(s / n);
}

}  // namespace

extern "C" {

int rh_mlp_gemm_check(const void* A, int32_t sam, int32_t sak, const void* B, int32_t sbk,
                      int32_t sbn, float* C, int32_t ldc, int32_t M, int32_t N, int32_t K,
                      int32_t tensor_cores) {
  if (!A || !B || !C || M <= 0 || N <= 0 || N > tc::kNmax || K <= 0) return RH_ERR_ARG;
  const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(A);
  const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(B);
  if (!tensor_cores) {
    const int tiles = ((M + 15) / 16) * ((N + 7) / 8);
    gemm_bf16<<<blocks((int64_t)tiles * 32, 128), 128>>>(a, sam, sak, b, sbk, sbn, C, ldc, M, N,
                                                         K, 0);
  } else {
    int* err = nullptr;
    if (cudaMalloc(&err, sizeof(int)) != cudaSuccess) return RH_ERR_NOMEM;
    cudaMemset(err, 0, sizeof(int));
    const int smem = tc::kSmemA + tc::kSmemB;
    cudaFuncSetAttribute(gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    gemm_tc<<<(M + tc::kM - 1) / tc::kM, 128, smem>>>(a, sam, sak, b, sbk, sbn, C, ldc, M, N, K,
                                                      0, err);
    int h = 0;
    cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(err);
    if (h) return RH_ERR_TIMEOUT;
  }
  if (cudaDeviceSynchronize() != cudaSuccess || cudaGetLastError() != cudaSuccess) return RH_ERR_CUDA;
  return RH_OK;
}

int rh_mlp_create(int32_t batch_max, int32_t device, rh_mlp** out) {
  if (!out || batch_max <= 0) return RH_ERR_ARG;
  *out = nullptr;
  if (batch_max > kMaxBatch) return RH_ERR_NOMEM;
  rh_mlp* m = new rh_mlp();
  m->bmax = batch_max;
  m->device = device;
  m->chunk = std::max(batch_max, kChunk);
  const size_t B = (size_t)batch_max, chunk = (size_t)m->chunk;
  const size_t parts = std::min<size_t>((B + 127) / 128, kMaxParts);
  auto round256 = [](size_t b) { return (b + 255) / 256 * 256; };
  int direct = 0;
  if (cudaDeviceGetAttribute(&direct, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device) !=
      cudaSuccess)
    cudaGetLastError();
  m->direct = direct != 0;
  const size_t no = round256(2 * chunk * RH_MLP_OUT * 4), ng = round256(kNPar * 4);
  if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreate(&m->st) != cudaSuccess ||
      cudaMalloc(&m->P, (3 + parts) * (size_t)kNPar * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->img, kImgBytes + 256) != cudaSuccess ||
      cudaHostAlloc(&m->host, no + ng + 256, cudaHostAllocMapped) != cudaSuccess ||
      cudaEventCreateWithFlags(&m->ev[0], cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&m->ev[1], cudaEventDisableTiming) != cudaSuccess ||
      cudaFuncSetAttribute(mlp_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           RowsSmem::bytes(true)) != cudaSuccess ||
      cudaFuncSetAttribute(mlp_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           RowsSmem::bytes(false)) != cudaSuccess ||
      cudaMemset(m->P, 0, 3 * (size_t)kNPar * sizeof(float)) != cudaSuccess ||
      cudaMemset(m->img, 0, kImgBytes + 256) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
    m->err = "allocation failed";
    cudaGetLastError();
    rh_mlp_destroy(m);
    return RH_ERR_NOMEM;
  }
  m->w = m->P;
  m->m = m->w + kNPar;
  m->v = m->m + kNPar;
  m->part = m->v + kNPar;
  m->failed = reinterpret_cast<int*>(m->img + kImgBytes);
  m->h_out = reinterpret_cast<float*>(m->host);
  m->h_g = reinterpret_cast<float*>(m->host + no);
  m->h_err = reinterpret_cast<int*>(m->host + no + ng);
  *m->h_err = 0;
  *out = m;
  return RH_OK;
}

int rh_mlp_destroy(rh_mlp* m) {
  if (!m) return RH_ERR_ARG;
  if (m->st) cudaStreamSynchronize(m->st);
  cudaFree(m->P);
  cudaFree(m->img);
  if (m->host) cudaFreeHost(m->host);
  if (m->copies) cudaFreeHost(m->copies);
  for (cudaEvent_t e : m->ev)
    if (e) cudaEventDestroy(e);
  if (m->st) cudaStreamDestroy(m->st);
  delete m;
  return RH_OK;
}

int rh_mlp_param_count(const rh_mlp* m, int32_t* n) {
  if (!m || !n) return RH_ERR_ARG;
  *n = kNPar;
  return RH_OK;
}

// Parameter order: for each layer, W (n x k row-major, padded) then b (n).
int rh_mlp_set_params(rh_mlp* m, const float* params) {
  if (!m || !params) return RH_ERR_ARG;
  MCK(cudaMemcpyAsync(m->w, params, kNPar * sizeof(float), cudaMemcpyHostToDevice, m->st));
  mlp_load<<<blocks(kNPar, 256), 256, 0, m->st>>>(m->w, m->img);
  MCK(cudaGetLastError());
  MCK(cudaMemsetAsync(m->m, 0, 2 * (size_t)kNPar * sizeof(float), m->st));  // Adam's moments
  m->step = 0;
  MCK(cudaStreamSynchronize(m->st));
  return RH_OK;
}

int rh_mlp_get_params(rh_mlp* m, float* params) {
  if (!m || !params) return RH_ERR_ARG;
  MCK(cudaMemcpyAsync(params, m->w, kNPar * sizeof(float), cudaMemcpyDeviceToHost, m->st));
  MCK(cudaStreamSynchronize(m->st));
  return RH_OK;
}

// The sweep runs in launches of `chunk` samples that write their outputs to
// two mapped host buffers in turn, so that the host copies one chunk's
// outputs out while the next one runs.
int rh_mlp_forward(rh_mlp* m, const float* x, int32_t n, float* y) {
  if (!m || !x || !y || n <= 0) return RH_ERR_ARG;
  const int64_t C = m->chunk;
  const int nch = (int)((n + C - 1) / C);
  auto rows = [&](int c) { return (int)std::min<int64_t>(C, n - c * C); };
  auto buffer = [&](int c) { return m->h_out + (size_t)(c & 1) * C * RH_MLP_OUT; };
  auto launch = [&](int c) -> int {
    RowsArgs a{};
    a.img = m->img;
    a.params = m->w;
    const int rx = reachable(m, x + (size_t)c * C * RH_MLP_IN, (size_t)rows(c) * RH_MLP_IN,
                             c & 1 ? kCopyX1 : kCopyX0, &a.x);
    if (rx != RH_OK) return rx;
    a.y = buffer(c);
    a.n = rows(c);
    a.err = m->h_err;
    const int tiles = (a.n + 127) / 128;
    mlp_rows<false><<<std::min(tiles, kMaxParts), kRowThreads, RowsSmem::bytes(false), m->st>>>(a);
    MCK(cudaGetLastError());
    MCK(cudaEventRecord(m->ev[c & 1], m->st));
    return RH_OK;
  };
  int r = launch(0);
  for (int c = 0; c < nch && r == RH_OK; ++c) {
    // the next chunk's buffers: last used by chunk c - 1, already copied out
    if (c + 1 < nch) r = launch(c + 1);
    if (r == RH_OK) r = ck(m, cudaEventSynchronize(m->ev[c & 1]), "forward");
    if (r == RH_OK)
      memcpy(y + (size_t)c * C * RH_MLP_OUT, buffer(c), sizeof(float) * RH_MLP_OUT * rows(c));
  }
  if (r != RH_OK) {
    cudaStreamSynchronize(m->st);  // no launch still reads or writes host memory
    return r;
  }
  return check_wait(m);
}

int rh_mlp_gradients(rh_mlp* m, const float* x, const float* target, int32_t n, float* grads,
                     float* loss) {
  if (!m || !x || !target || n <= 0 || n > m->bmax) return RH_ERR_ARG;
  int parts = 0;
  int r = train_pass(m, x, target, n, &parts);
  if (r) return r;
  if (grads) {
    mlp_finish<<<blocks(kNPar, 256), 256, 0, m->st>>>(m->part, parts, m->h_g, nullptr, nullptr,
                                                      nullptr, nullptr, m->failed, AdamStep{});
    r = ck(m, cudaGetLastError(), "gradients");
  }
  const int rs = ck(m, cudaStreamSynchronize(m->st), "gradients");
  if (r) return r;
  if (rs) return rs;
  if ((r = check_wait(m))) return r;
  if (grads) memcpy(grads, m->h_g, kNPar * sizeof(float));
  if (loss) *loss = mean_loss(m, n);
  return RH_OK;
}

int rh_mlp_train_step(rh_mlp* m, const float* x, const float* target, int32_t n, float lr,
                      float* loss) {
  if (!m || !x || !target || n <= 0 || n > m->bmax) return RH_ERR_ARG;
  int parts = 0;
  int r = train_pass(m, x, target, n, &parts);
  if (r) return r;
  const float step = (float)(m->step + 1);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const AdamStep s{lr, b1, b2, eps, 1.f - powf(b1, step), 1.f - powf(b2, step)};
  mlp_finish<<<blocks(kNPar, 256), 256, 0, m->st>>>(m->part, parts, nullptr, m->w, m->m, m->v,
                                                    m->img, m->failed, s);
  r = ck(m, cudaGetLastError(), "training step");
  const int rs = ck(m, cudaStreamSynchronize(m->st), "training step");
  if (r) return r;
  if (rs) return rs;
  if ((r = check_wait(m))) return r;
  m->step += 1;
  if (loss) *loss = mean_loss(m, n);
  return RH_OK;
}

int rh_mlp_last_error(const rh_mlp* m, char* buf, size_t n) {
  if (!buf || n == 0) return RH_ERR_ARG;
  snprintf(buf, n, "%s", m ? m->err.c_str() : "");
  return RH_OK;
}

}  // extern "C"

// ------------------------------------------------ forward pass without allocation
//
// rh_mlp_forward above works on a handle whose buffers rh_mlp_create obtained
// with cudaMalloc.  Some callers cannot make that call: a host program whose
// device memory is all handed out by its own allocator or pool, a co-simulation
// loop that budgets device memory up front, or a caller that must not pay the
// device-wide synchronisation an allocation can imply.  rh_mlp_forward_noalloc
// serves them: the caller brings the parameters, inputs and outputs in device
// memory, and one launch of mlp_rows converts the weights into shared memory
// and keeps every intermediate value there.

namespace {

constexpr int kMaxDevices = 64;

void na_msg(char* err, size_t len, const char* fmt, ...) __attribute__((format(printf, 3, 4)));
void na_msg(char* err, size_t len, const char* fmt, ...) {
  if (!err || len == 0) return;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(err, len, fmt, ap);
  va_end(ap);
}

bool overlap(const float* a, size_t na, const float* b, size_t nb) {
  const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pb = reinterpret_cast<uintptr_t>(b);
  return pa < pb + nb * sizeof(float) && pb < pa + na * sizeof(float);
}

bool on_device(const void* p, int dev) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (a.type == cudaMemoryTypeDevice && a.device == dev) || a.type == cudaMemoryTypeManaged;
}

}  // namespace

extern "C" int rh_mlp_forward_noalloc(const float* d_params, const float* d_x, int32_t n,
                                      float* d_y, void* stream, char* err, size_t err_len) {
  if (err && err_len) err[0] = '\0';
  if (!d_params || !d_x || !d_y) {
    na_msg(err, err_len, "rh_mlp_forward_noalloc: params, x and y must be device pointers");
    return RH_ERR_ARG;
  }
  if (n <= 0 || n > RH_MLP_NOALLOC_MAX_BATCH) {
    na_msg(err, err_len,
           "rh_mlp_forward_noalloc: n = %d is outside 1..%d; split the batch", (int)n,
           RH_MLP_NOALLOC_MAX_BATCH);
    return RH_ERR_ARG;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    na_msg(err, err_len, "rh_mlp_forward_noalloc: no usable current device (%s)",
           cudaGetErrorString(e));
    return RH_ERR_CUDA;
  }
  if (!on_device(d_params, dev) || !on_device(d_x, dev) || !on_device(d_y, dev)) {
    na_msg(err, err_len,
           "rh_mlp_forward_noalloc: params, x and y must be device memory of the current "
           "device %d",
           dev);
    return RH_ERR_ARG;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int tiles = (n + 127) / 128;
  const size_t ny = (size_t)n * RH_MLP_OUT;
  // (a single CTA reads everything before it writes)
  const bool held = tiles > 1 && (overlap(d_y, ny, d_x, (size_t)n * RH_MLP_IN) ||
                                  overlap(d_y, ny, d_params, kNPar));
  e = held ? cudaFuncSetAttribute(mlp_rows<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  RowsSmem::bytes_held())
           : cudaFuncSetAttribute(mlp_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  RowsSmem::bytes(false));
  if (e != cudaSuccess) {
    na_msg(err, err_len, "rh_mlp_forward_noalloc: set-up failed on device %d: %s", dev,
           cudaGetErrorString(e));
    return RH_ERR_CUDA;
  }
  RowsArgs a{};
  a.params = d_params;
  a.x = d_x;
  a.y = d_y;
  a.n = n;
  if (held) {
    unsigned ctas = 2;
    while ((int)ctas < std::min(tiles, kHeldCtas)) ctas *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kRowThreads);
    cfg.dynamicSmemBytes = RowsSmem::bytes_held();
    cfg.stream = st;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim = {ctas, 1, 1};
    cfg.attrs = &cluster;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, mlp_rows<false, true>, a);
    if (e != cudaSuccess) cudaGetLastError();
  } else {
    mlp_rows<false><<<tiles, kRowThreads, RowsSmem::bytes(false), st>>>(a);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    na_msg(err, err_len, "rh_mlp_forward_noalloc: launch failed: %s", cudaGetErrorString(e));
    return RH_ERR_CUDA;
  }
  return RH_OK;
}
