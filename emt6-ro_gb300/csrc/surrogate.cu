// surrogate.cu -- the protocol-outcome surrogate: a 100 -> 512 -> 512 -> 512 -> 1
// GELU MLP trained and evaluated on the GPU with hand-written kernels.
//
// All matrix products run on the 5th-generation tensor cores (tcgen05.mma, M =
// 128, N = 128, K = 16, BF16 in, FP32 accumulators in tensor memory); operands
// are 64-column blocks in shared memory with the 128-byte swizzle, K-major for
// the layers, rows of the batch (MN-major) for the weight gradients.  A training
// step is two launches, a prediction one:
//   mlp_rows_kernel   everything that stays within a row: a cluster of 4 CTAs
//     owns 128 rows, each CTA 128 of the 512 columns of every layer.  It packs
//     the inputs, runs the hidden layers, the head, and (training) the error
//     back through the layers.  A layer's activations go from a CTA's
//     accumulator into its shared memory and from there, by bulk copies, into
//     its three peers', where the next product reads them; weights stream in by
//     TMA.
//   mlp_grads_kernel  the weight gradients (products over the batch), split
//     over a cluster's CTAs and summed in a fixed order through their shared
//     memory, with Adam on the spot; the vectors' gradients beside them.
//
// Every wait on an mbarrier is bounded (kWaitLimitNs); a wait that runs out
// sets an error flag, the CTA stops issuing products and loads, goes through its
// cluster's exchanges and barriers with the others, waits (bounded) for its own
// tensor-core work, frees its TMEM and returns; weights that would be spoiled are not
// updated, and the host reports the flag.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <random>
#include <string>
#include <utility>
#include <vector>

#include "emt6ro_gb300.h"
#include "emt6ro_surrogate.h"

namespace emt6 {
int set_error(int code, const std::string &msg);
}

namespace {

// 16 warps: warp w reads TMEM lane quarter w % 4 (tile rows 32(w % 4)..+31)
// and runs the epilogue of column group w / 4 (32 columns), so the
// epilogue's transcendental work and stores spread over 4x more warps
constexpr int BM = 128, BN = 128, BK = 64, STAGES = 4, GEMM_THREADS = 512;
constexpr int TILE_BYTES = BM * BK * 2;  // 16 KB per operand per stage
constexpr int GEMM_SMEM = 1024 + STAGES * 2 * TILE_BYTES + 256;
constexpr uint64_t kWaitLimitNs = 1000000000ull;  // 1 s
constexpr int IN = EMT6_MLP_IN, INP = EMT6_MLP_IN_PAD, HID = EMT6_MLP_HIDDEN;
constexpr int CLUSTER = HID / BN;  // CTAs that share a tile of 128 rows

// ---- PTX wrappers ----------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase of `parity` to complete.  Gives up after
// limit_ns (default kWaitLimitNs), or early when another thread of the CTA
// raised `abort`.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int *abort,
                          uint64_t limit_ns = kWaitLimitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (abort && *abort) return false;
    if (global_ns() - t0 > limit_ns) return false;
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// a box from shared memory to global; wait for the reads of it, or for its writes
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(x), "r"(y), "r"(src)
               : "memory");
}

__device__ __forceinline__ void store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void store_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Clusters.  Every CTA of a cluster reaches every barrier, also after a wait
// that gave up.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// the address of shared-memory address `addr` in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// The same without ordering any data: the CTAs have all come this far.
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait;" ::: "memory");
}

// `bytes` of this CTA's shared memory at `src` to shared-memory address `dst` of a
// peer, counted on the peer's mbarrier `bar` (both from peer_addr)
__device__ __forceinline__ void peer_copy(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "r"(src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void peer_store4(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

__device__ __forceinline__ int peer_load4(uint32_t addr) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float4 peer_load16(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// orders this thread's shared-memory writes before later reads of the tensor cores
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Programmatic dependent launch: the kernels of a training step are launched
// with programmatic stream serialisation, so each one's launch and prologue
// overlap the tail of the one before.  pdl_wait() blocks until the previous
// kernel in the stream has completed and its writes are visible (a no-op
// without the launch attribute); pdl_trigger(), issued after a CTA's last
// global write, lets the next kernel be scheduled.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, BF16 inputs, FP32 accumulator.
__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane; the wait is in the
// same statement so no use of the registers can be scheduled before it.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 8 consecutive FP32 columns (see tmem_ld32)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor: K-major tile written by TMA with the
// 128-byte swizzle (rows of 64 BF16 = 128 B, 8-row atoms of 1024 B).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) |
         (static_cast<uint64_t>(1) << 16) |            // leading offset (unused when swizzled)
         (static_cast<uint64_t>(1024 >> 4) << 32) |    // stride offset: next 8-row atom
         (static_cast<uint64_t>(1) << 46) |            // descriptor version
         (static_cast<uint64_t>(2) << 61);             // 128-byte swizzle
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 128, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) |
                            (static_cast<uint32_t>(BN >> 3) << 17) |
                            (static_cast<uint32_t>(BM >> 4) << 24);

// The same for operands stored with their reduction dimension outermost (weight
// gradients: rows of the batch): boxes of 64 columns x 64 rows with the 128-byte
// swizzle, two of them for 128 columns (leading offset), 8-row atoms (stride).
constexpr int BOX_BYTES = BK * 64 * 2;
__device__ __forceinline__ uint64_t mn_desc(uint32_t saddr) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) |
         (static_cast<uint64_t>(BOX_BYTES >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
constexpr uint32_t kIdescMN = kIdesc | (1u << 15) | (1u << 16);

// The handle's error flag: on the device, and (host_err) where the host reads it
// without a copy.
__device__ __forceinline__ void raise_error(int *err, int *host_err) {
  atomicOr(err, 1);
  *reinterpret_cast<volatile int *>(host_err) = 1;
  __threadfence_system();
}

// GELU and its derivative, by erff and expf: they round as the library's do, which
// a cheaper normal tail did not, and an activation that rounds to the other of two
// BF16 values travels through every layer above.
__device__ __forceinline__ float gelu(float z) {
  return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}

__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) +
         z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// C tile (blockIdx.y, blockIdx.x) of C[M,N] = A[M,K] B[N,K]^T in FP32: the
// building block of the two kernels below on its own, for tests.  stall_ns
// (emt6_test_mlp_gemm_timeout): when nonzero, the MMA issuer first waits this
// many ns on a barrier nothing arrives on, so it gives up exactly as a
// timed-out pipeline wait would.
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    mlp_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    int nk, int N, float *c_out, int *err, uint32_t stall_ns) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~static_cast<uintptr_t>(1023));
  uint8_t *sA = smem;
  uint8_t *sB = smem + STAGES * TILE_BYTES;
  // barriers: full[STAGES], empty[STAGES], done, never (nothing arrives on
  // it: the target of the test hook's stalled wait)
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + 2 * STAGES * TILE_BYTES);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 2);
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES),
                 done = smem_u32(bars + 2 * STAGES), never = smem_u32(bars + 2 * STAGES + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done, 1);
    mbar_init(never, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  bool failed = false;
  int issued = 0;  // k-blocks whose loads thread 0 issued
  if (threadIdx.x == 0) {
    // TMA producer
    for (int kb = 0; kb < nk; ++kb) {
      const int s = kb % STAGES;
      if (kb >= STAGES && !mbar_wait(empty0 + 8 * s, ((kb / STAGES) - 1) & 1, abort)) {
        failed = true;
        *abort = 1;
        break;
      }
      mbar_expect_tx(full0 + 8 * s, 2 * TILE_BYTES);
      tma_load_2d(smem_u32(sA + s * TILE_BYTES), &tmA, full0 + 8 * s, kb * BK, m0);
      tma_load_2d(smem_u32(sB + s * TILE_BYTES), &tmB, full0 + 8 * s, kb * BK, n0);
      ++issued;
    }
  } else if (threadIdx.x == 32) {
    // MMA issuer
    if (stall_ns && !mbar_wait(never, 0, abort, stall_ns)) {
      failed = true;
      *abort = 1;
      __threadfence_block();
    }
    for (int kb = 0; kb < nk && !failed; ++kb) {
      const int s = kb % STAGES;
      if (!mbar_wait(full0 + 8 * s, (kb / STAGES) & 1, abort)) {
        failed = true;
        *abort = 1;
        __threadfence_block();
        break;
      }
      tc_fence_after();
      const uint32_t a = smem_u32(sA + s * TILE_BYTES), b = smem_u32(sB + s * TILE_BYTES);
#pragma unroll
      for (int k = 0; k < BK / 16; ++k)
        umma_bf16(tmem, sw128_desc(a + 32 * k), sw128_desc(b + 32 * k), kIdesc,
                  (kb | k) != 0 ? 1u : 0u);
      umma_commit(empty0 + 8 * s);
    }
    // arrives once every MMA issued above has completed, failed or not
    umma_commit(done);
  }
  __syncwarp();
  bool have = mbar_wait(done, 0, nullptr);
  if (threadIdx.x == 0 && *abort) {
    // a pipeline wait gave up: let the loads still in flight (at most the
    // last STAGES issued; older stages were consumed before being reused)
    // land before the CTA frees its shared memory
    for (int kb = issued - STAGES < 0 ? 0 : issued - STAGES; kb < issued; ++kb)
      mbar_wait(full0 + 8 * (kb % STAGES), (kb / STAGES) & 1, nullptr);
  }
  have = __all_sync(0xffffffffu, have && !*abort && !failed);
  tc_fence_after();
  if (have) {
    const int quarter = warp & 3, group = warp >> 2;
    float v[32];
    tmem_ld32(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + group * 32, v);
    float4 *dst = reinterpret_cast<float4 *>(
        c_out + static_cast<size_t>(m0 + quarter * 32 + lane) * N + n0 + group * 32);
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else if (lane == 0) {
    atomicOr(err, 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, BN);
  }
}

// ---- rows: forward, head, error ---------------------------------------------------
struct RowsArgs {
  const float *x;            // [n][100]
  int n;                     // rows; training: a multiple of 128
  int norm;                  // inputs are (x - mean) / std
  float mean[IN], std[IN];
  const float *b[3], *w4, *b4;
  float *y;                  // prediction: [n]
  // training
  const float *target;
  float *dy, *loss;
  uint4 *z[3];         // pre-activations, 8 columns of a row each (z_at)
  __nv_bfloat16 *x16;  // [n][128]
  int *err, *host_err;
  // test hook (emt6_test_mlp_stall): the phase whose products the first CTA's
  // issuer gives up on after waiting stall_ns (0: none) for them to complete
  int stall_phase;
  uint32_t stall_ns;
};

// where training's operands of the weight gradients go, [n][512]
struct RowsMaps {
  CUtensorMap a[3], dz[3];
};

// shared memory of mlp_rows_kernel: the 8 blocks of the current operand, the
// ring of weight tiles, barriers and the head's errors
constexpr int ACT_BYTES = (HID / BK) * TILE_BYTES, RING = 6;
constexpr int ROWS_SMEM = 1024 + ACT_BYTES + RING * TILE_BYTES + 2048;  // 227 KB: all there is

// byte offset of the 16-byte chunk holding columns 8 * chunk .. of `row` in a
// K-major operand of 128 rows (64-column blocks, 128-byte swizzle)
__device__ __forceinline__ uint32_t act_chunk(int row, int chunk) {
  return static_cast<uint32_t>((chunk >> 3) * TILE_BYTES + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}

// What bounds it: a latency chain of product, epilogue and exchange per layer, as
// long at 640 rows as at 4,096.  What an epilogue reads from memory is loaded ahead
// of the product (scoring 200,000 rows 2.24 -> 2.08 ms), and a CTA's first block of
// the next operand leaves while the second is computed (1.93 ms).  Predicting, a
// resident cluster goes over tiles of rows, the next one's inputs and first weights
// on their way during the last layer (1.88 ms).  Training's operands of the weight
// gradients leave by bulk copies of the operand blocks that the exchange needs
// anyway, as rows; transposed from registers they took 4,600 cycles a layer.  The
// phases and the columns of an epilogue are loops, not unrolled: code that each
// warp runs once is fetched as it goes.  With one launch per layer, and input,
// head and error launches between, a step's rows took 75 us of GPU time.
template <bool TRAIN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    mlp_rows_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                    const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmT1,
                    const __grid_constant__ CUtensorMap tmT2, const __grid_constant__ RowsMaps out,
                    const __grid_constant__ RowsArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~static_cast<uintptr_t>(1023));
  const uint32_t act = smem_u32(smem), ring = act + ACT_BYTES;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + ACT_BYTES + RING * TILE_BYTES);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * RING + 2);
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *s_dy = reinterpret_cast<float *>(bars + 16);  // [128]
  float *s_loss = s_dy + BM;                           // [16]
  float *s_norm = s_loss + 16;                         // [2][100]
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + RING), done = smem_u32(bars + 2 * RING),
                 in = smem_u32(bars + 2 * RING + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int n0 = static_cast<int>(rank) * BN;
  int m0 = static_cast<int>(blockIdx.x / CLUSTER) * BM;  // the cluster's rows, in turn
  const int stride = static_cast<int>(gridDim.x / CLUSTER) * BM;
  constexpr int PHASES = TRAIN ? 5 : 3;

  if (tid == 0) {
    for (int s = 0; s < RING; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done, 1);
    mbar_init(in, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // weights come from the previous kernel

  // weight tiles of all phases in one sequence: layer 1 has 2 k-blocks, the
  // others 8; the producer runs ahead of the products by the ring's 6 stages
  int issued = 0;
  bool failed = false;
  auto load_tiles = [&](int phase, int from, int to) {  // thread 0
    const CUtensorMap *map = phase == 0 ? &tmW0 : phase == 1 ? &tmW1 : phase == 2 ? &tmW2
                             : phase == 3 ? &tmT2 : &tmT1;
    for (int kb = from; kb < to && !*abort; ++kb) {
      const int s = issued % RING;
      if (issued >= RING && !mbar_wait(empty0 + 8 * s, ((issued / RING) - 1) & 1, abort)) {
        *abort = 1;
        break;
      }
      mbar_expect_tx(full0 + 8 * s, TILE_BYTES);
      tma_load_2d(ring + s * TILE_BYTES, map, full0 + 8 * s, kb * BK, n0);
      ++issued;
    }
  };
  if (tid == 0) load_tiles(0, 0, 2);
  if (!TRAIN && a.norm) {
    if (tid < IN) {
      s_norm[tid] = a.mean[tid];
      s_norm[IN + tid] = a.std[tid];
    }
    __syncthreads();
  }

  // Exchange of operand blocks within the cluster: each CTA writes its own part
  // of the next operand locally, then bulk copies take it to the three peers
  // (scattered remote stores of the same values took 5 us a layer).  `in` counts
  // what arrives from them.
  int exchanges = 0;
  const auto exchange = [&](uint32_t at, uint32_t bytes, int pieces, uint32_t pitch) {
    fence_async();
    __syncthreads();
    if (tid == 0) {
      mbar_expect_tx(in, (CLUSTER - 1) * bytes * pieces);
      for (uint32_t p = 1; p < CLUSTER; ++p) {
        const uint32_t to = (rank + p) % CLUSTER;
        for (int i = 0; i < pieces; ++i)
          peer_copy(peer_addr(act + at + i * pitch, to), act + at + i * pitch, bytes, peer_addr(in, to));
      }
    }
    ++exchanges;
  };
  const auto arrived = [&]() -> bool { return mbar_wait(in, (exchanges - 1) & 1, nullptr); };
  cluster_meet();  // every CTA runs, its barriers initialised

  // inputs: each CTA takes a quarter of the rows, a thread one 16-byte chunk of
  // BF16 (zero columns 100..127, zero rows beyond n)
  static_assert(BM / CLUSTER * (INP / 8) == GEMM_THREADS, "one chunk per thread");
  const int xr = static_cast<int>(rank) * (BM / CLUSTER) + tid / (INP / 8), xc = tid % (INP / 8);
  float f[8];
  const auto load_x = [&](int from) {
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = 0.0f;
    if (from + xr < a.n) {
      const float *src = a.x + static_cast<size_t>(from + xr) * IN + xc * 8;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (xc * 8 + q < IN) f[q] = src[q];
    }
  };
  load_x(m0);

  const int quarter = warp & 3, group = warp >> 2;
  // this thread's row, and its 4 x 8 columns: two of each of the CTA's blocks, the
  // first block's first, so that it leaves while the second is computed
  const int row = quarter * 32 + lane;
  const auto col = [&](int j) { return (j >> 1) * BK + group * 16 + (j & 1) * 8; };
  const int lane_col = n0 + col(lane >> 3) + (lane & 7);  // of the warp's 32, the lane's
  const uint32_t acc0 = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
  // 8 BF16 values of this thread (columns n0 + col(j) ..) into the next operand
  const auto publish = [&](int j, const uint4 &v) {
    *reinterpret_cast<uint4 *>(smem + act_chunk(row, (n0 + col(j)) / 8)) = v;
  };
  const uint32_t own = rank * (BN / BK) * TILE_BYTES;  // this CTA's two blocks of it
  const auto push = [&](int half) {  // one of them to the peers
    fence_async();
    __syncthreads();
    if (tid == 0) {
      if (half == 0) mbar_expect_tx(in, (CLUSTER - 1) * BN / BK * TILE_BYTES);
      const uint32_t at = act + own + half * TILE_BYTES;
      for (uint32_t p = 1; p < CLUSTER; ++p) {
        const uint32_t to = (rank + p) % CLUSTER;
        peer_copy(peer_addr(at, to), at, TILE_BYTES, peer_addr(in, to));
      }
    }
    exchanges += half;
  };
  // these two blocks at shared address `from` to rows of global memory
  const auto store_rows = [&](const CUtensorMap *map, uint32_t from) {  // thread 0
#pragma unroll
    for (int i = 0; i < 4; ++i)
      tma_store_2d(map, from + i * BOX_BYTES, n0 + (i >> 1) * BK, m0 + (i & 1) * 64);
    store_commit();
  };
  // each thread reads back what it wrote: laid out so that a warp's are adjacent
  const auto z_at = [&](int l, int j) -> uint4 & {
    return a.z[l][(static_cast<size_t>(blockIdx.x) * 16 + group * 4 + j) * BM + row];
  };

  int used = 0, products = 0;  // weight tiles consumed, products run
  for (;;) {
    // ---- inputs into the operand
    if (!TRAIN && a.norm && m0 + xr < a.n)
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (xc * 8 + q < IN) f[q] = (f[q] - s_norm[xc * 8 + q]) / s_norm[IN + xc * 8 + q];
    {
      alignas(16) __nv_bfloat16 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = __float2bfloat16_rn(f[q]);
      *reinterpret_cast<uint4 *>(smem + act_chunk(xr, xc)) = *reinterpret_cast<const uint4 *>(v);
      if (TRAIN)
        *reinterpret_cast<uint4 *>(a.x16 + static_cast<size_t>(m0 + xr) * INP + 8 * xc) =
            *reinterpret_cast<const uint4 *>(v);
    }
    // 32 rows of the 2 blocks
    exchange(rank * (BM / CLUSTER) * 128, BM / CLUSTER * 128, INP / BK, TILE_BYTES);
    const bool more = !TRAIN && m0 + stride < a.n;
#pragma unroll 1
    for (int phase = 0; phase < PHASES; ++phase) {
      const int nk = phase == 0 ? INP / BK : HID / BK;
      // what the epilogue reads from memory, ahead of the product: a lane's share of
      // the warp's 32 biases, or the thread's pre-activations
      const float bias = phase < 3 ? __ldg(a.b[phase < 3 ? phase : 0] + lane_col) : 0.0f;
      uint4 zq[4];
      if (TRAIN && phase >= 3)
#pragma unroll
        for (int j = 0; j < 4; ++j) zq[j] = z_at(phase == 3 ? 1 : 0, j);
      if (phase == 2 && more) load_x(m0 + stride);
      // ---- product: accumulator = operand x this CTA's 128 weight rows
      if (tid == 0) {
        load_tiles(phase, phase == 0 ? 2 : RING, nk);
      } else if (tid == 32) {
        // waited for after an abort too: the peers' copies still come, each
        // exchange's are counted on `in` before the next one's, and none may
        // reach a CTA that has left
        if (!arrived() || *abort) *abort = 1;
        if (a.stall_ns && blockIdx.x == 0 && phase == a.stall_phase && !*abort &&
            !mbar_wait(done, products & 1, nullptr, a.stall_ns))
          *abort = 1;
        tc_fence_after();
        for (int kb = 0; kb < nk && !*abort; ++kb) {
          const int s = (used + kb) % RING;
          if (!mbar_wait(full0 + 8 * s, ((used + kb) / RING) & 1, abort)) {
            *abort = 1;
            break;
          }
          tc_fence_after();
          const uint32_t pa = act + kb * TILE_BYTES, pb = ring + s * TILE_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16(tmem, sw128_desc(pa + 32 * k), sw128_desc(pb + 32 * k), kIdesc,
                      (kb | k) != 0 ? 1u : 0u);
          umma_commit(empty0 + 8 * s);
        }
        umma_commit(done);  // arrives once every product above has completed
      }
      __syncwarp();
      // (after a wait ran out: no further ones)
      if (!failed && !mbar_wait(done, products & 1, nullptr)) failed = true;
      ++products;
      tc_fence_after();
      used += nk;
      // the ring is free: the next phase's first tiles load during the epilogue
      if (tid == 0) {
        if (phase + 1 < PHASES) load_tiles(phase + 1, 0, RING);
        else if (more) load_tiles(0, 0, INP / BK);
      }
      __syncwarp();
      const bool last = TRAIN && phase == PHASES - 1;  // the lowest layer's error goes no further
      if (TRAIN && tid == 0) store_read();  // the operand's own blocks are overwritten next
      if (!last) cluster_meet();  // every CTA's products have read the operand and its copies
      // ---- epilogue
      if (phase < 3) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          float v[8];
          tmem_ld8(acc0 + col(j), v);
          alignas(16) __nv_bfloat16 zb[8], h[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float z = v[i] + __shfl_sync(0xffffffffu, bias, 8 * j + i);
            zb[i] = __float2bfloat16_rn(z);
            h[i] = __float2bfloat16_rn(gelu(z));
          }
          const uint4 &hv = *reinterpret_cast<const uint4 *>(h);
          publish(j, hv);
          if (TRAIN) z_at(phase, j) = *reinterpret_cast<const uint4 *>(zb);
          if (j == 1) push(0);
        }
      } else {
        const int l = phase == 3 ? 1 : 0;  // layer whose pre-activations the error passes
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          const uint4 zj = j == 0 ? zq[0] : j == 1 ? zq[1] : j == 2 ? zq[2] : zq[3];
          const __nv_bfloat16 *zb = reinterpret_cast<const __nv_bfloat16 *>(&zj);
          float v[8];
          tmem_ld8(acc0 + col(j), v);
          alignas(16) __nv_bfloat16 h[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16_rn(v[i] * gelu_grad(__bfloat162float(zb[i])));
          const uint4 &hv = *reinterpret_cast<const uint4 *>(h);
          if (!last)
            publish(j, hv);
          else  // the ring is free; a peer's copy of this CTA's operand blocks may not be done
            *reinterpret_cast<uint4 *>(smem + ACT_BYTES + act_chunk(row, col(j) / 8)) = hv;
          if (!last && j == 1) push(0);
        }
      }
      if (last) {
        fence_async();
        __syncthreads();
        if (tid == 0) store_rows(&out.dz[0], ring);
        break;
      }
      tc_fence_before();
      push(1);
      if (TRAIN && tid == 0) {
        store_rows(phase < 3 ? &out.a[phase] : &out.dz[1], act + own);
        if (phase == 2) store_read();  // dZ3 replaces A3 below
      }
      if (phase == 2) {
        const float w4l = TRAIN ? __ldg(a.w4 + lane_col) : 0.0f;
        float wh[HID / 256][8];  // the head's weights
#pragma unroll
        for (int j = 0; j < HID / 256; ++j)
#pragma unroll
          for (int q = 0; q < 8; ++q) wh[j][q] = __ldg(a.w4 + 8 * (lane + 32 * j) + q);
        if (TRAIN)
#pragma unroll
          for (int j = 0; j < 4; ++j) zq[j] = z_at(2, j);
        if (!failed && !arrived()) failed = true;
        // ---- head: y = A3 w4 + b4, one warp per row
#pragma unroll 1
        for (int k = 0; k < BM / CLUSTER / 16; ++k) {
          const int r = static_cast<int>(rank) * (BM / CLUSTER) + warp * (BM / CLUSTER / 16) + k;
          float acc = 0.0f;
#pragma unroll
          for (int j = 0; j < HID / 256; ++j) {
            const uint4 u = *reinterpret_cast<const uint4 *>(smem + act_chunk(r, lane + 32 * j));
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&u);
#pragma unroll
            for (int q = 0; q < 8; ++q) acc += __bfloat162float(e[q]) * wh[j][q];
          }
#pragma unroll
          for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          const float yr = acc + a.b4[0];
          if (!TRAIN) {
            if (lane == 0 && m0 + r < a.n) a.y[m0 + r] = yr;
          } else {
            const float e = yr - a.target[m0 + r], d = 2.0f * e / static_cast<float>(a.n);
            if (lane == 0) {
              a.dy[m0 + r] = d;
              s_loss[warp] = (k ? s_loss[warp] : 0.0f) + e * e;
            }
            if (lane < CLUSTER) peer_store4(peer_addr(smem_u32(s_dy + r), lane), d);
          }
        }
        if (TRAIN) {
          cluster_sync();  // dy is everywhere, and the operand may be overwritten
          if (tid == 0) {
            float t = 0.0f;
#pragma unroll
            for (int k = 0; k < 16; ++k) t += s_loss[k];
            atomicAdd(a.loss, t);
          }
          const float d = s_dy[row];
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {
            const uint4 zj = j == 0 ? zq[0] : j == 1 ? zq[1] : j == 2 ? zq[2] : zq[3];
            const __nv_bfloat16 *zb = reinterpret_cast<const __nv_bfloat16 *>(&zj);
            alignas(16) __nv_bfloat16 h[8];
            float wj[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) wj[i] = __shfl_sync(0xffffffffu, w4l, 8 * j + i);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              h[i] = __float2bfloat16_rn(d * wj[i] * gelu_grad(__bfloat162float(zb[i])));
            const uint4 &hv = *reinterpret_cast<const uint4 *>(h);
            publish(j, hv);
            if (j == 1) push(0);
          }
          push(1);
          if (tid == 0) store_rows(&out.dz[2], act + own);
        }
      }
    }
    if (!more) break;
    m0 += stride;
    cluster_sync();  // the heads have read the operand
  }
  // no CTA leaves while a peer may still read from or write to it
  if (TRAIN && tid == 0) store_wait();
  cluster_meet();
  pdl_trigger();
  if (*abort || failed) {
    if (lane == 0) raise_error(a.err, a.host_err);
    // loads still in flight (at most the last RING issued) land before the
    // CTA frees its shared memory
    if (tid == 0)
      for (int k = issued - RING < 0 ? 0 : issued - RING; k < issued; ++k)
        mbar_wait(full0 + 8 * (k % RING), (k / RING) & 1, nullptr);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, BN);
  }
}

// ---- weight gradients and Adam -------------------------------------------------------
struct VecAdam {
  float *w, *m, *v;
  const __nv_bfloat16 *rows;  // [n][512]: dZ, or A3 for w4
  float *grad_out;
};

struct GradsArgs {
  float *w[3], *m[3], *v[3];
  __nv_bfloat16 *wb[3], *wbt[3];  // BF16 W and (null for the first layer) W^T
  float *grad[3];                 // export instead of the update, or null
  VecAdam vec[5];
  const float *dy;
  float *clear;  // the next step's loss sum
  int B, splits;
  float lr, beta1, beta2, eps, bc1, bc2;
  int *err, *host_err;
  uint32_t stall_ns;  // test hook, as in RowsArgs: of the first CTA's products
};

// The step's rows failed, or another CTA's products have: nothing is updated.  Read
// where it is needed: held from the start it slowed the vectors' sums (a step of
// 65,536 rows 1.11 vs 1.06 ms).
__device__ __forceinline__ bool step_failed(const GradsArgs &a) {
  return *static_cast<const volatile int *>(a.err) != 0;
}

__device__ __forceinline__ void vec_update(const GradsArgs &a, const VecAdam &p, int idx, float g) {
  if (p.grad_out) {
    p.grad_out[idx] = g;
    return;
  }
  const float w = p.w[idx];
  const float m = a.beta1 * p.m[idx] + (1.0f - a.beta1) * g;
  const float s = a.beta2 * p.v[idx] + (1.0f - a.beta2) * g * g;
  if (step_failed(a)) return;
  p.m[idx] = m;
  p.v[idx] = s;
  p.w[idx] = w - a.lr * (m / a.bc1) / (sqrtf(s / a.bc2) + a.eps);
}

// Gradients and Adam updates of 16 elements of b1, b2, b3 (sums of dZ over the
// batch) or w4 (A3^T dy), by 8 warps.  Rows 8 q .. 8 q + 7, and those 256 further
// and so on, are summed in order by slot q = 8 (lane / 8) + w, a thread two
// columns of it; then slots 16, 8, 4, 2 and 1 apart.  Latency bound, beside the
// products: 32 bytes of 8 rows per load round.
constexpr int VEC_COLS = 16, VEC_TASKS = 4 * HID / VEC_COLS, VEC_WARPS = 8;
__device__ __forceinline__ void vec_adam(const GradsArgs &a, int task, float *part, int w, int lane) {
  const int k = task / (HID / VEC_COLS), c0 = task % (HID / VEC_COLS) * VEC_COLS;
  const uint32_t *src =
      reinterpret_cast<const uint32_t *>(a.vec[k].rows + c0) + (lane & 7);
  float g[2] = {0.0f, 0.0f};
#pragma unroll 2
  for (int r = 8 * (8 * (lane >> 3) + w); r < a.B; r += 256) {
    uint32_t u[8];
    float h[2][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = src[static_cast<size_t>(r + i) * (HID / 2)];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      h[0][i] = __uint_as_float(u[i] << 16);
      h[1][i] = __uint_as_float(u[i] & 0xffff0000u);
    }
    if (k == 3) {
      const float4 d0 = *reinterpret_cast<const float4 *>(a.dy + r);
      const float4 d1 = *reinterpret_cast<const float4 *>(a.dy + r + 4);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        g[q] += h[q][0] * d0.x + h[q][1] * d0.y + h[q][2] * d0.z + h[q][3] * d0.w +
                h[q][4] * d1.x + h[q][5] * d1.y + h[q][6] * d1.z + h[q][7] * d1.w;
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) g[q] += h[q][i];
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    g[q] += __shfl_xor_sync(0xffffffffu, g[q], 16);
    g[q] += __shfl_xor_sync(0xffffffffu, g[q], 8);
  }
  if (lane < 8) *reinterpret_cast<float2 *>(part + w * VEC_COLS + 2 * lane) = make_float2(g[0], g[1]);
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(32 * VEC_WARPS) : "memory");
  if (w == 0 && lane < VEC_COLS) {
    float t[VEC_WARPS];
#pragma unroll
    for (int q = 0; q < VEC_WARPS; ++q) t[q] = part[q * VEC_COLS + lane];
#pragma unroll
    for (int o = 4; o; o >>= 1)
#pragma unroll
      for (int q = 0; q < o; ++q) t[q] += t[q + o];
    vec_update(a, a.vec[k], c0 + lane, t[0]);
  }
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(32 * VEC_WARPS) : "memory");  // part is free again
}

// tiles of 128 x 128 weights: 16 of layer 3, 16 of layer 2, 4 of layer 1
constexpr int GRAD_TILES = 36;
constexpr int RED_BYTES = 2 * BM * BN * 4;  // two partial tiles, over the ring
constexpr int TILE_T_BYTES = BN * (BM + 8) * 2;  // W^T on its way out, rows padded
constexpr int GRADS_SMEM = 1024 + RED_BYTES + TILE_T_BYTES + 256 + VEC_WARPS * VEC_COLS * 4;
static_assert(RED_BYTES >= STAGES * 2 * TILE_BYTES, "the partial tiles replace the ring");

// One cluster per tile of dW = dZ^T A (a product over the batch): its CTAs take
// consecutive parts of the batch (`splits` parts in all, one or two per CTA,
// each with an accumulator of its own), lay the partial tiles down in shared
// memory, and each sums a share of the rows over all parts in order, applies
// Adam and writes W and W^T.  Warps that do not feed the tensor cores compute
// the vectors' gradients meanwhile.  Bound by L2 reads at 4,096 rows (75 MB of
// operands in 9.5 us); the seven launches it replaces took 40.
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    mlp_grads_kernel(const __grid_constant__ CUtensorMap tmZ0, const __grid_constant__ CUtensorMap tmZ1,
                     const __grid_constant__ CUtensorMap tmZ2, const __grid_constant__ CUtensorMap tmX,
                     const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                     const __grid_constant__ GradsArgs a, int cluster) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~static_cast<uintptr_t>(1023));
  const uint32_t ringA = smem_u32(smem), ringB = ringA + STAGES * TILE_BYTES;
  float *red = reinterpret_cast<float *>(smem);  // [part][128][128], columns swizzled
  __nv_bfloat16 *tile_t = reinterpret_cast<__nv_bfloat16 *>(smem + RED_BYTES);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + RED_BYTES + TILE_T_BYTES);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 1);
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *vec_part = reinterpret_cast<float *>(smem + RED_BYTES + TILE_T_BYTES + 256);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES), done = smem_u32(bars + 2 * STAGES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int t = static_cast<int>(blockIdx.x) / cluster;
  const int l = t < 16 ? 2 : t < 32 ? 1 : 0, N = l ? HID : INP;
  const int k = t < 16 ? t : t < 32 ? t - 16 : t - 32;
  const int m0 = (l ? k / 4 : k) * BM, n0 = (l ? k % 4 : 0) * BN;
  const int parts = a.splits / cluster, nkp = a.B / BK / a.splits, nk = parts * nkp;
  const int kb0 = rank * nk;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 2 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // operands come from the previous kernel

  int issued = 0;
  if (tid == 0) {
    const CUtensorMap *ma = l == 2 ? &tmZ2 : l == 1 ? &tmZ1 : &tmZ0;
    const CUtensorMap *mb = l == 2 ? &tmA1 : l == 1 ? &tmA0 : &tmX;
    for (int kb = 0; kb < nk; ++kb) {
      const int s = kb % STAGES;
      if (kb >= STAGES && !mbar_wait(empty0 + 8 * s, ((kb / STAGES) - 1) & 1, abort)) {
        *abort = 1;
        break;
      }
      mbar_expect_tx(full0 + 8 * s, 2 * TILE_BYTES);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t at = s * TILE_BYTES + i * BOX_BYTES;
        tma_load_2d(ringA + at, ma, full0 + 8 * s, m0 + 64 * i, (kb0 + kb) * BK);
        tma_load_2d(ringB + at, mb, full0 + 8 * s, n0 + 64 * i, (kb0 + kb) * BK);
      }
      ++issued;
    }
  } else if (tid == 32) {
    const bool stall = a.stall_ns && blockIdx.x == 0 && !mbar_wait(done, 0, abort, a.stall_ns);
    if (stall) *abort = 1;
    for (int kb = 0; kb < nk && !stall; ++kb) {  // (an abort ends it at a wait)
      const int s = kb % STAGES;
      if (!mbar_wait(full0 + 8 * s, (kb / STAGES) & 1, abort)) {
        *abort = 1;
        break;
      }
      tc_fence_after();
      const uint32_t pa = ringA + s * TILE_BYTES, pb = ringB + s * TILE_BYTES;
#pragma unroll
      for (int q = 0; q < BK / 16; ++q)
        umma_bf16(tmem + static_cast<uint32_t>(kb / nkp) * BN, mn_desc(pa + 2048 * q),
                  mn_desc(pb + 2048 * q), kIdescMN, (kb % nkp | q) != 0 ? 1u : 0u);
      umma_commit(empty0 + 8 * s);
    }
    umma_commit(done);  // arrives once every product above has completed
  } else if (warp >= 2) {
    if (blockIdx.x == 0 && tid == 64) *a.clear = 0.0f;
    if (warp < 2 + VEC_WARPS) {
      for (int task = blockIdx.x; task < VEC_TASKS; task += gridDim.x)
        vec_adam(a, task, vec_part, warp - 2, lane);
    } else if (blockIdx.x == gridDim.x - 1 && warp == 2 + VEC_WARPS) {  // b4: sum dy
      float g = 0.0f;
      for (int j = lane; j < a.B; j += 32) g += a.dy[j];
#pragma unroll
      for (int o = 16; o; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
      if (lane == 0) vec_update(a, a.vec[4], 0, g);
    } else if (step_failed(a)) {
      *abort = 1;
    }
  }
  __syncwarp();
  bool failed = !mbar_wait(done, 0, nullptr);
  if (tid == 0 && *abort)
    for (int q = issued - STAGES < 0 ? 0 : issued - STAGES; q < issued; ++q)
      mbar_wait(full0 + 8 * (q % STAGES), (q / STAGES) & 1, nullptr);
  failed = failed || *abort;
  if (failed) *abort = 1;
  tc_fence_after();
  __syncthreads();  // (after an abort: nothing lands in the ring any more)
  const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane;
  for (int p = 0; p < parts; ++p) {
    float v[32];
    tmem_ld32(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + p * BN + group * 32, v);
    // 16-byte columns of a row swizzled by the row: conflict-free both ways
    float4 *dst = reinterpret_cast<float4 *>(red + p * BM * BN + row * BN);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      dst[(group * 8 + i) ^ (row & 31)] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  }
  if (failed && lane == 0) raise_error(a.err, a.host_err);
  tc_fence_before();
  cluster_sync();
  // a part that failed would spoil the tile: no CTA of its cluster updates it
  int part_failed = 0;
  if (lane < cluster) part_failed = peer_load4(peer_addr(smem_u32(const_cast<int *>(abort)), lane));
  bool skip = false;
  const int share = BM / cluster, r0 = rank * share;  // rows this CTA finishes
  const uint32_t base = smem_u32(red);
  for (int i = tid; i < share * 32; i += GEMM_THREADS) {
    const int r = r0 + (i >> 5), c4 = i & 31;
    const uint32_t at = base + static_cast<uint32_t>((r * 32 + (c4 ^ (r & 31))) * 16);
    const size_t at_w = static_cast<size_t>(m0 + r) * N + n0 + 4 * c4;
    float4 m4 = make_float4(0.f, 0.f, 0.f, 0.f), v4 = m4, w4 = m4;
    if (!a.grad[l]) {
      m4 = *reinterpret_cast<const float4 *>(a.m[l] + at_w);
      v4 = *reinterpret_cast<const float4 *>(a.v[l] + at_w);
      w4 = *reinterpret_cast<const float4 *>(a.w[l] + at_w);
    }
    float4 q[8];  // all parts' loads in flight, then summed in order
#pragma unroll
    for (int p = 0; p < 8; ++p)
      if (p < a.splits)
        q[p] = peer_load16(peer_addr(at + (parts == 2 ? p & 1 : 0) * (BM * BN * 4), parts == 2 ? p >> 1 : p));
    float4 g = q[0];
#pragma unroll
    for (int p = 1; p < 8; ++p)
      if (p < a.splits) {
        g.x += q[p].x; g.y += q[p].y; g.z += q[p].z; g.w += q[p].w;
      }
    if (a.grad[l]) {
      *reinterpret_cast<float4 *>(a.grad[l] + at_w) = g;
      continue;
    }
    skip = __any_sync(0xffffffffu, part_failed);  // (every thread runs as many rounds)
    if (skip) continue;
    const float gg[4] = {g.x, g.y, g.z, g.w}, mo[4] = {m4.x, m4.y, m4.z, m4.w},
                vo[4] = {v4.x, v4.y, v4.z, v4.w}, wo[4] = {w4.x, w4.y, w4.z, w4.w};
    float mn[4], vn[4], wn[4];
    alignas(8) __nv_bfloat16 wb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      mn[q] = a.beta1 * mo[q] + (1.0f - a.beta1) * gg[q];
      vn[q] = a.beta2 * vo[q] + (1.0f - a.beta2) * gg[q] * gg[q];
      wn[q] = wo[q] - a.lr * (mn[q] / a.bc1) / (sqrtf(vn[q] / a.bc2) + a.eps);
      wb[q] = __float2bfloat16_rn(wn[q]);
      tile_t[(4 * c4 + q) * (share + 8) + ((((r - r0) >> 3) ^ ((c4 >> 1) & 3)) << 3) + (r & 7)] = wb[q];
    }
    *reinterpret_cast<float4 *>(a.m[l] + at_w) = make_float4(mn[0], mn[1], mn[2], mn[3]);
    *reinterpret_cast<float4 *>(a.v[l] + at_w) = make_float4(vn[0], vn[1], vn[2], vn[3]);
    *reinterpret_cast<float4 *>(a.w[l] + at_w) = make_float4(wn[0], wn[1], wn[2], wn[3]);
    *reinterpret_cast<uint2 *>(a.wb[l] + at_w) = *reinterpret_cast<const uint2 *>(wb);
  }
  __syncthreads();
  if (!a.grad[l] && a.wbt[l] && !skip)
    for (int i = tid; i < BN * share / 8; i += GEMM_THREADS) {
      const int c = i / (share / 8), q = i % (share / 8);
      *reinterpret_cast<uint4 *>(a.wbt[l] + static_cast<size_t>(n0 + c) * HID + m0 + r0 + 8 * q) =
          *reinterpret_cast<const uint4 *>(tile_t + c * (share + 8) + ((q ^ ((c >> 3) & 3)) << 3));
    }
  pdl_trigger();
  cluster_sync();  // no CTA leaves while another reads its partial tiles
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, 2 * BN);
  }
}

__global__ void to_bf16_kernel(const float *src, __nv_bfloat16 *dst, __nv_bfloat16 *dst_t, int rows,
                               int cols) {
  const int total = rows * cols;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int r = i / cols, c = i % cols;
    const __nv_bfloat16 b = __float2bfloat16_rn(src[i]);
    dst[i] = b;
    if (dst_t) dst_t[static_cast<size_t>(c) * rows + r] = b;
  }
}

// ---- host side -------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// BF16 matrix [rows][cols], boxes of 64 columns x `high` rows.
bool make_map(CUtensorMap *map, const void *base, int rows, int cols, int high = BM) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  cuuint32_t box[2] = {BK, static_cast<cuuint32_t>(high)};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launch in clusters, with programmatic stream serialisation (see pdl_wait /
// pdl_trigger).
template <typename... KArgs, typename... Args>
cudaError_t launch_clusters(void (*kernel)(KArgs...), int grid, int cluster, size_t smem,
                            cudaStream_t st, const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Dynamic shared memory of a kernel, raised once per device.
template <typename K>
cudaError_t raise_smem(K kernel, int bytes, bool (&done)[64]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (done[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

// Clusters of mlp_rows_kernel<false> that are resident at once, asked once per device.
cudaError_t resident_clusters(int *out) {
  static std::atomic<int> known[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  *out = known[dev].load();
  if (*out) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CLUSTER);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = ROWS_SMEM;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = CLUSTER;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  e = cudaOccupancyMaxActiveClusters(out, mlp_rows_kernel<false>, &cfg);
  if (e == cudaSuccess) known[dev].store(*out = std::max(*out, 1));
  return e;
}

template <typename T>
struct DevArr {
  T *p = nullptr;
  size_t n = 0;
  bool alloc(size_t count) {
    n = count;
    return cudaMalloc(&p, count * sizeof(T)) == cudaSuccess;
  }
  ~DevArr() {
    if (p) cudaFree(p);
  }
};

}  // namespace

struct emt6_mlp {
  int device = 0, max_batch = 0;
  cudaStream_t stream = nullptr;
  int64_t step = 0;
  int slot = 0;  // of the running step's loss sum; the step clears the other
  float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
  // parameters: FP32 masters, Adam moments, BF16 copies (W; W^T of layers 2, 3)
  DevArr<float> w[3], m[3], v[3], b[3], bm[3], bv[3], w4, m4, v4, b4, mb4, vb4;
  DevArr<__nv_bfloat16> wb[3], wbt[3];
  DevArr<__nv_bfloat16> X16, A[3], dZ[3];  // operands of the weight gradients, [max_batch][columns]
  DevArr<uint4> Z[3];                      // pre-activations, 8 to an element
  DevArr<float> dy, loss, gradw[3], gradv[5];
  int split_override = 0;  // 0: choose per batch size
  int stall_phase = 0;     // emt6_test_mlp_stall: PHASES - 1 and below, or kStallGrads
  uint32_t stall_ns = 0;   // of the next launch concerned, 0: none
  DevArr<int> err;
  int *host_err = nullptr, *host_err_dev = nullptr;  // pinned, written by the kernels
  ~emt6_mlp() {
    if (host_err) cudaFreeHost(host_err);
  }
  CUtensorMap mX, mW[3], mWT[3];
  RowsMaps mRows;
};

namespace {

constexpr int kStallGrads = 5;

// the stall asked of the launch about to be made, once
uint32_t take_stall(emt6_mlp *net, bool grads) {
  if (!net->stall_ns || grads != (net->stall_phase == kStallGrads)) return 0;
  return std::exchange(net->stall_ns, 0u);
}

int rows_of(int) { return EMT6_MLP_HIDDEN; }
int cols_of(int l) { return l == 0 ? EMT6_MLP_IN_PAD : EMT6_MLP_HIDDEN; }

int fail(const std::string &m, int code = EMT6_ERR_DEVICE) { return emt6::set_error(code, m); }

int cuda_fail(cudaError_t e, const char *what) {
  return fail(std::string(what) + ": " + cudaGetErrorString(e), EMT6_ERR_CUDA);
}

int check_batch(emt6_mlp *net, int B) {
  if (B <= 0 || B > net->max_batch || B % 128 != 0)
    return fail("surrogate batch must be a positive multiple of 128 up to max_batch",
                EMT6_ERR_INVALID);
  return EMT6_OK;
}

int status(const emt6_mlp *net) {
  if (*static_cast<const volatile int *>(net->host_err))
    return fail("surrogate GEMM: a tensor-core pipeline wait timed out");
  return EMT6_OK;
}

int read_err(emt6_mlp *net) {
  const cudaError_t e = cudaStreamSynchronize(net->stream);
  return e == cudaSuccess ? status(net) : cuda_fail(e, "surrogate");
}

// every map covers a whole allocation: batches use its first rows or columns
bool build_maps(emt6_mlp *net) {
  bool ok = make_map(&net->mX, net->X16.p, net->max_batch, INP, 64);
  for (int l = 0; l < 3 && ok; ++l) {
    ok = make_map(&net->mW[l], net->wb[l].p, rows_of(l), cols_of(l)) &&
         make_map(&net->mRows.dz[l], net->dZ[l].p, net->max_batch, HID, 64);
    ok = ok && make_map(&net->mRows.a[l], net->A[l].p, net->max_batch, HID, 64);
    if (l > 0) ok = ok && make_map(&net->mWT[l], net->wbt[l].p, cols_of(l), rows_of(l));
  }
  return ok;
}

// Split of the weight-gradient GEMMs' K (= B) dimension: the most of 8, 4, 2
// that leaves every CTA at least 4 k-blocks of 64 rows.
int weight_splits(const emt6_mlp *net, int B) {
  const int nkb = B / BK;
  if (net->split_override > 0) return nkb % net->split_override == 0 ? net->split_override : 1;
  for (int sp : {8, 4, 2})
    if (nkb % sp == 0 && nkb / sp >= 4) return sp;
  return 1;
}

// rows through the network: predictions, or (with targets) all that the weight
// gradients need
int run_rows(emt6_mlp *net, const float *d_x, int64_t n, const float *mean, const float *std,
             const float *d_target, float *d_y) {
  static bool raised[2][64];
  cudaError_t e = d_target ? raise_smem(mlp_rows_kernel<true>, ROWS_SMEM, raised[1])
                           : raise_smem(mlp_rows_kernel<false>, ROWS_SMEM, raised[0]);
  if (e != cudaSuccess) return cuda_fail(e, "surrogate rows");
  // rows per launch: the kernel counts them in 32 bits
  const int64_t most = int64_t(1) << 30;
  for (int64_t at = 0; at < n; at += most) {
    RowsArgs a;
    std::memset(&a, 0, sizeof(a));
    a.n = static_cast<int>(n - at < most ? n - at : most);
    a.x = d_x + at * IN;
    a.norm = mean != nullptr;
    if (mean)
      for (int c = 0; c < IN; ++c) {
        a.mean[c] = mean[c];
        a.std[c] = std[c];
      }
    for (int l = 0; l < 3; ++l) a.b[l] = net->b[l].p;
    a.w4 = net->w4.p;
    a.b4 = net->b4.p;
    a.err = net->err.p;
    a.host_err = net->host_err_dev;
    a.stall_phase = net->stall_phase;
    a.stall_ns = take_stall(net, false);
    int grid = (a.n + BM - 1) / BM * CLUSTER;
    if (d_target) {
      a.target = d_target;
      a.dy = net->dy.p;
      a.loss = net->loss.p + net->slot;
      a.x16 = net->X16.p;
      for (int l = 0; l < 3; ++l) a.z[l] = net->Z[l].p;
      e = launch_clusters(mlp_rows_kernel<true>, grid, CLUSTER, ROWS_SMEM, net->stream, net->mW[0],
                          net->mW[1], net->mW[2], net->mWT[1], net->mWT[2], net->mRows, a);
    } else {
      a.y = d_y + at;
      int resident = 0;
      e = resident_clusters(&resident);
      if (e != cudaSuccess) return cuda_fail(e, "surrogate rows");
      grid = std::min(grid, resident * CLUSTER);
      e = launch_clusters(mlp_rows_kernel<false>, grid, CLUSTER, ROWS_SMEM, net->stream, net->mW[0],
                          net->mW[1], net->mW[2], net->mWT[1], net->mWT[2], net->mRows, a);
    }
    if (e != cudaSuccess) return cuda_fail(e, "surrogate rows");
  }
  return EMT6_OK;
}

// weight gradients of the rows just run, with Adam or (apply false) exported
int run_grads(emt6_mlp *net, int B, bool apply, float lr) {
  static bool raised[64];
  cudaError_t e = raise_smem(mlp_grads_kernel, GRADS_SMEM, raised);
  if (e != cudaSuccess) return cuda_fail(e, "surrogate gradients");
  GradsArgs a;
  std::memset(&a, 0, sizeof(a));
  const float step = static_cast<float>(net->step + 1);
  for (int l = 0; l < 3; ++l) {
    a.w[l] = net->w[l].p;
    a.m[l] = net->m[l].p;
    a.v[l] = net->v[l].p;
    a.wb[l] = net->wb[l].p;
    a.wbt[l] = net->wbt[l].p;
    a.grad[l] = apply ? nullptr : net->gradw[l].p;
    a.vec[l] = {net->b[l].p, net->bm[l].p, net->bv[l].p, net->dZ[l].p, apply ? nullptr : net->gradv[l].p};
  }
  a.vec[3] = {net->w4.p, net->m4.p, net->v4.p, net->A[2].p, apply ? nullptr : net->gradv[3].p};
  a.vec[4] = {net->b4.p, net->mb4.p, net->vb4.p, nullptr, apply ? nullptr : net->gradv[4].p};
  a.dy = net->dy.p;
  a.clear = net->loss.p + (net->slot ^ 1);
  a.B = B;
  a.splits = weight_splits(net, B);
  a.lr = lr;
  a.beta1 = net->beta1;
  a.beta2 = net->beta2;
  a.eps = net->eps;
  a.bc1 = 1.0f - std::pow(net->beta1, step);
  a.bc2 = 1.0f - std::pow(net->beta2, step);
  a.err = net->err.p;
  a.host_err = net->host_err_dev;
  a.stall_ns = take_stall(net, true);
  // at most two parts per CTA (two accumulators, two tiles of shared memory),
  // and clusters of 4, 36 of which are resident at once
  const int cluster = a.splits < 4 ? a.splits : 4;
  e = launch_clusters(mlp_grads_kernel, GRAD_TILES * cluster, cluster, GRADS_SMEM, net->stream,
                      net->mRows.dz[0], net->mRows.dz[1], net->mRows.dz[2], net->mX, net->mRows.a[0],
                      net->mRows.a[1], a,
                      cluster);
  if (e != cudaSuccess) return cuda_fail(e, "surrogate gradients");
  if (apply) ++net->step;
  return EMT6_OK;
}

// The batch's mean squared error; the next batch sums into the other slot.
int read_loss(emt6_mlp *net, int B, int slot, float *h_loss) {
  float s = 0.0f;
  cudaError_t e = cudaMemcpyAsync(&s, net->loss.p + slot, 4, cudaMemcpyDeviceToHost, net->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(net->stream);
  if (e != cudaSuccess) return cuda_fail(e, "surrogate loss");
  *h_loss = s / static_cast<float>(B);
  return EMT6_OK;
}

int refresh_bf16(emt6_mlp *net) {
  for (int l = 0; l < 3; ++l) {
    to_bf16_kernel<<<304, 256, 0, net->stream>>>(net->w[l].p, net->wb[l].p, net->wbt[l].p,
                                                  rows_of(l), cols_of(l));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "surrogate weights");
  }
  return EMT6_OK;
}

// The 8 FP32 parameter arrays in the C ABI's order and their element counts.
void param_arrays(emt6_mlp *net, float *dev[8], size_t cnt[8]) {
  for (int l = 0; l < 3; ++l) {
    dev[2 * l] = net->w[l].p;
    cnt[2 * l] = static_cast<size_t>(rows_of(l)) * cols_of(l);
    dev[2 * l + 1] = net->b[l].p;
    cnt[2 * l + 1] = HID;
  }
  dev[6] = net->w4.p;
  cnt[6] = HID;
  dev[7] = net->b4.p;
  cnt[7] = 1;
}

cudaError_t launch_test_gemm(const CUtensorMap &ma, const CUtensorMap &mb, float *c, int M, int N,
                             int K, int *err, uint32_t stall_ns, cudaStream_t st) {
  static bool raised[64];
  cudaError_t e = raise_smem(mlp_gemm_kernel, GEMM_SMEM, raised);
  if (e != cudaSuccess) return e;
  mlp_gemm_kernel<<<dim3(N / BN, M / BM), GEMM_THREADS, GEMM_SMEM, st>>>(ma, mb, K / BK, N, c, err,
                                                                        stall_ns);
  return cudaGetLastError();
}

}  // namespace

extern "C" {

int emt6_mlp_create(int max_batch, uint64_t seed, int device, emt6_mlp **out) {
  if (!out) return fail("emt6_mlp_create: null output", EMT6_ERR_INVALID);
  *out = nullptr;
  if (max_batch <= 0 || max_batch % 128 != 0)
    return fail("emt6_mlp_create: max_batch must be a positive multiple of 128", EMT6_ERR_INVALID);
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_mlp_create");
  if (!encode_fn()) return fail("emt6_mlp_create: cuTensorMapEncodeTiled unavailable");
  auto *net = new emt6_mlp();
  net->device = device;
  net->max_batch = max_batch;
  const int H = HID;
  bool ok = cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) == cudaSuccess;
  for (int l = 0; l < 3 && ok; ++l) {
    const size_t n = static_cast<size_t>(rows_of(l)) * cols_of(l);
    ok = net->w[l].alloc(n) && net->m[l].alloc(n) && net->v[l].alloc(n) && net->b[l].alloc(H) &&
         net->bm[l].alloc(H) && net->bv[l].alloc(H) && net->wb[l].alloc(n) &&
         (l == 0 || net->wbt[l].alloc(n)) && net->gradw[l].alloc(n);
  }
  const size_t BH = static_cast<size_t>(max_batch) * H;
  ok = ok && net->w4.alloc(H) && net->m4.alloc(H) && net->v4.alloc(H) && net->b4.alloc(1) &&
       net->mb4.alloc(1) && net->vb4.alloc(1) &&
       net->X16.alloc(static_cast<size_t>(max_batch) * INP) && net->dy.alloc(max_batch) &&
       net->loss.alloc(2) && net->err.alloc(1) &&
       cudaHostAlloc(&net->host_err, sizeof(int), cudaHostAllocMapped) == cudaSuccess &&
       cudaHostGetDevicePointer(&net->host_err_dev, net->host_err, 0) == cudaSuccess;
  if (ok) *net->host_err = 0;
  for (int l = 0; l < 3 && ok; ++l)
    ok = net->A[l].alloc(BH) && net->dZ[l].alloc(BH) && net->Z[l].alloc(BH / 8);
  for (int i = 0; i < 5 && ok; ++i) ok = net->gradv[i].alloc(i < 4 ? H : 1);
  if (!ok) {
    if (net->stream) cudaStreamDestroy(net->stream);
    delete net;
    return fail("emt6_mlp_create: out of device memory");
  }
  // He-style initialisation from a seeded generator; biases and moments zero
  std::mt19937_64 rng(seed);
  std::vector<float> host;
  e = cudaSuccess;
  for (int l = 0; l < 4 && e == cudaSuccess; ++l) {
    const int rows = l < 3 ? rows_of(l) : 1, cols = l < 3 ? cols_of(l) : H;
    const int fan_in = l == 0 ? IN : H;
    std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / static_cast<float>(fan_in)));
    host.assign(static_cast<size_t>(rows) * cols, 0.0f);
    for (int r = 0; r < rows; ++r)
      for (int c = 0; c < cols; ++c)
        if (l != 0 || c < IN) host[static_cast<size_t>(r) * cols + c] = nd(rng);
    float *dst = l < 3 ? net->w[l].p : net->w4.p;
    e = cudaMemcpy(dst, host.data(), host.size() * sizeof(float), cudaMemcpyHostToDevice);
  }
  float *zero[] = {net->m[0].p, net->v[0].p, net->m[1].p, net->v[1].p, net->m[2].p, net->v[2].p,
                   net->b[0].p, net->bm[0].p, net->bv[0].p, net->b[1].p, net->bm[1].p,
                   net->bv[1].p, net->b[2].p, net->bm[2].p, net->bv[2].p, net->m4.p, net->v4.p,
                   net->b4.p, net->mb4.p, net->vb4.p};
  const size_t zn[] = {net->m[0].n, net->v[0].n, net->m[1].n, net->v[1].n, net->m[2].n,
                       net->v[2].n, net->b[0].n, net->bm[0].n, net->bv[0].n, net->b[1].n,
                       net->bm[1].n, net->bv[1].n, net->b[2].n, net->bm[2].n, net->bv[2].n,
                       net->m4.n, net->v4.n, net->b4.n, net->mb4.n, net->vb4.n};
  for (size_t i = 0; i < sizeof(zero) / sizeof(zero[0]) && e == cudaSuccess; ++i)
    e = cudaMemset(zero[i], 0, zn[i] * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(net->err.p, 0, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(net->loss.p, 0, 2 * sizeof(float));
  if (e != cudaSuccess) {
    emt6_mlp_destroy(net);
    return cuda_fail(e, "emt6_mlp_create");
  }
  int rc = build_maps(net) ? refresh_bf16(net) : fail("emt6_mlp_create: cuTensorMapEncodeTiled failed");
  if (rc == EMT6_OK) {
    e = cudaStreamSynchronize(net->stream);
    if (e != cudaSuccess) rc = cuda_fail(e, "emt6_mlp_create");
  }
  if (rc != EMT6_OK) {
    emt6_mlp_destroy(net);
    return rc;
  }
  *out = net;
  return EMT6_OK;
}

void emt6_mlp_destroy(emt6_mlp *net) {
  if (!net) return;
  cudaSetDevice(net->device);
  if (net->stream) cudaStreamSynchronize(net->stream);
  if (net->stream) cudaStreamDestroy(net->stream);
  delete net;
}

void *emt6_mlp_stream(emt6_mlp *net) { return net ? net->stream : nullptr; }

int emt6_mlp_set_params(emt6_mlp *net, const float *const *host) {
  if (!net || !host) return fail("emt6_mlp_set_params: null argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  float *dev[8];
  size_t cnt[8];
  param_arrays(net, dev, cnt);
  cudaError_t e = cudaStreamSynchronize(net->stream);
  for (int i = 0; i < 8 && e == cudaSuccess; ++i)
    e = cudaMemcpy(dev[i], host[i], cnt[i] * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_mlp_set_params");
  int rc = refresh_bf16(net);
  if (rc != EMT6_OK) return rc;
  e = cudaStreamSynchronize(net->stream);
  return e == cudaSuccess ? EMT6_OK : cuda_fail(e, "emt6_mlp_set_params");
}

int emt6_mlp_get_params(emt6_mlp *net, float *const *host) {
  if (!net || !host) return fail("emt6_mlp_get_params: null argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  float *dev[8];
  size_t cnt[8];
  param_arrays(net, dev, cnt);
  cudaError_t e = cudaStreamSynchronize(net->stream);
  for (int i = 0; i < 8 && e == cudaSuccess; ++i)
    e = cudaMemcpy(host[i], dev[i], cnt[i] * sizeof(float), cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? read_err(net) : cuda_fail(e, "emt6_mlp_get_params");
}

int emt6_mlp_predict(emt6_mlp *net, const float *d_x, int B, float *d_y) {
  if (!net || !d_x || !d_y) return fail("emt6_mlp_predict: null argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  const int rc = check_batch(net, B);
  return rc == EMT6_OK ? run_rows(net, d_x, B, nullptr, nullptr, nullptr, d_y) : rc;
}

int emt6_mlp_predict_rows(emt6_mlp *net, const float *d_x, int64_t n, const float *mean,
                          const float *std, float *d_y) {
  if (!net || n < 0 || (n > 0 && (!d_x || !d_y)) || !mean != !std)
    return fail("emt6_mlp_predict_rows: null or negative argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  return run_rows(net, d_x, n, mean, std, nullptr, d_y);
}

int emt6_mlp_train_step(emt6_mlp *net, const float *d_x, const float *d_target, int B, float lr,
                        float *h_loss) {
  if (!net || !d_x || !d_target) return fail("emt6_mlp_train_step: null argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  int rc = check_batch(net, B);
  const int slot = net->slot;
  if (rc == EMT6_OK) rc = run_rows(net, d_x, B, nullptr, nullptr, d_target, nullptr);
  if (rc == EMT6_OK) rc = run_grads(net, B, true, lr);
  if (rc != EMT6_OK) return rc;
  net->slot ^= 1;
  if (!h_loss) return EMT6_OK;
  rc = read_loss(net, B, slot, h_loss);
  return rc == EMT6_OK ? read_err(net) : rc;
}

int emt6_mlp_gradients(emt6_mlp *net, const float *d_x, const float *d_target, int B,
                       float *const *host_grads, float *h_loss) {
  if (!net || !d_x || !d_target || !host_grads)
    return fail("emt6_mlp_gradients: null argument", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  int rc = check_batch(net, B);
  const int slot = net->slot;
  if (rc == EMT6_OK) rc = run_rows(net, d_x, B, nullptr, nullptr, d_target, nullptr);
  if (rc == EMT6_OK) rc = run_grads(net, B, false, 0.0f);
  if (rc != EMT6_OK) return rc;
  net->slot ^= 1;
  if ((rc = read_err(net)) != EMT6_OK) return rc;
  const float *grad[8] = {net->gradw[0].p, net->gradv[0].p, net->gradw[1].p, net->gradv[1].p,
                          net->gradw[2].p, net->gradv[2].p, net->gradv[3].p, net->gradv[4].p};
  float *dev[8];
  size_t cnt[8];
  param_arrays(net, dev, cnt);
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 8 && e == cudaSuccess; ++i)
    e = cudaMemcpy(host_grads[i], grad[i], cnt[i] * sizeof(float), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_mlp_gradients");
  return h_loss ? read_loss(net, B, slot, h_loss) : EMT6_OK;
}

int emt6_mlp_set_splitk(emt6_mlp *net, int splits) {
  if (!net || (splits != 0 && splits != 1 && splits != 2 && splits != 4 && splits != 8))
    return fail("emt6_mlp_set_splitk: splits must be 0 (automatic), 1, 2, 4 or 8",
                EMT6_ERR_INVALID);
  net->split_override = splits;
  return EMT6_OK;
}

int emt6_mlp_status(const emt6_mlp *net) {
  return net ? status(net) : fail("emt6_mlp_status: null", EMT6_ERR_INVALID);
}

int emt6_mlp_sync(emt6_mlp *net) {
  if (!net) return fail("emt6_mlp_sync: null", EMT6_ERR_INVALID);
  cudaSetDevice(net->device);
  return read_err(net);
}

int emt6_test_mlp_stall(emt6_mlp *net, int phase, uint32_t stall_us) {
  if (!net || phase < 0 || phase > kStallGrads || stall_us == 0 || stall_us > 100000)
    return fail("emt6_test_mlp_stall: null handle, phase outside 0..5 or stall outside 1..100000 us",
                EMT6_ERR_INVALID);
  net->stall_phase = phase;
  net->stall_ns = stall_us * 1000u;
  return EMT6_OK;
}

int emt6_test_mlp_gemm(const void *d_a, const void *d_b, float *d_c, int M, int N, int K,
                       void *stream) {
  if (!d_a || !d_b || !d_c) return fail("emt6_test_mlp_gemm: null argument", EMT6_ERR_INVALID);
  if (M <= 0 || N <= 0 || K <= 0 || M % BM || N % BN || K % BK)
    return fail("emt6_test_mlp_gemm: M, N multiples of 128 and K of 64 required", EMT6_ERR_INVALID);
  if (!encode_fn()) return fail("cuTensorMapEncodeTiled unavailable");
  CUtensorMap ma, mb;
  if (!make_map(&ma, d_a, M, K) || !make_map(&mb, d_b, N, K))
    return fail("emt6_test_mlp_gemm: cuTensorMapEncodeTiled failed");
  int *err = nullptr;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMallocAsync(&err, sizeof(int), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_test_mlp_gemm");
  e = launch_test_gemm(ma, mb, d_c, M, N, K, err, 0u, st);
  int h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(err, st);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_test_mlp_gemm");
  if (h) return fail("emt6_test_mlp_gemm: a tensor-core pipeline wait timed out");
  return EMT6_OK;
}

int emt6_test_mlp_gemm_timeout(const void *d_a, const void *d_b, float *d_c, int M, int N,
                               int K, uint32_t stall_us, void *stream) {
  if (!d_a || !d_b || !d_c || stall_us == 0 || stall_us > 100000)
    return fail("emt6_test_mlp_gemm_timeout: null argument or stall outside 1..100000 us",
                EMT6_ERR_INVALID);
  if (M <= 0 || N <= 0 || K <= 0 || M % BM || N % BN || K % BK)
    return fail("emt6_test_mlp_gemm_timeout: M, N multiples of 128 and K of 64 required",
                EMT6_ERR_INVALID);
  if (!encode_fn()) return fail("cuTensorMapEncodeTiled unavailable");
  CUtensorMap ma, mb;
  if (!make_map(&ma, d_a, M, K) || !make_map(&mb, d_b, N, K))
    return fail("emt6_test_mlp_gemm_timeout: cuTensorMapEncodeTiled failed");
  int *err = nullptr;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMallocAsync(&err, sizeof(int), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_test_mlp_gemm_timeout");
  e = launch_test_gemm(ma, mb, d_c, M, N, K, err, stall_us * 1000u, st);
  int h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(err, st);
  if (e != cudaSuccess) return cuda_fail(e, "emt6_test_mlp_gemm_timeout");
  if (h) return fail("emt6_test_mlp_gemm_timeout: a tensor-core pipeline wait timed out");
  return EMT6_OK;
}

}  // extern "C"
