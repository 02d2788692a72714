#pragma once
// Test-only kernel for the bounded-wait path of the attention kernels (not part of the product).
//
// One warp waits, through the same mbar_wait the attention kernels use, on an mbarrier that nothing
// ever arrives on.  No copy, no MMA and no tensor memory is in flight, so when the wait gives up the
// kernel simply returns: the test then reads the sticky status word the wait left behind, checks that
// a later launch returns at entry, and that clearing the status re-arms the library.  The wait's
// cycle budget is cut to about a millisecond for this translation unit.  A second kernel issues one small copy into its own
// shared memory when its wait has given up, and is to stay until it has landed.
#define FRAY_WAIT_LIMIT_CYCLES 2000000LL
#include "flash_attn/host_sm100.cuh"
#include "flash_attn/sm100_ptx.cuh"

namespace fray_test {

static constexpr unsigned int kProbeSite = 0x7E1;   // site code the probe's wait reports
static constexpr int kProbeExtra = 42;

// out[0]: 1 = the wait ran out and the kernel returned normally, 2 = the status was already raised and the
// kernel returned at entry (as every attention kernel does), 3 = the barrier flipped (cannot happen).
__global__ void wait_probe_kernel(int* out) {
  __shared__ uint64_t bar;
  __shared__ uint32_t abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = (*reinterpret_cast<volatile int*>(&fray::sm100::fray_attn_status[0]) != 0) ? 2u : 0u;
    fray::sm100::mbar_init(&bar, 1);
    fray::sm100::fence_barrier_init();
  }
  __syncthreads();
  if (abort_flag != 0) {
    if (threadIdx.x == 0) out[0] = 2;
    return;
  }
  if (threadIdx.x < 32) fray::sm100::mbar_wait(&bar, 0, &abort_flag, kProbeSite, kProbeExtra);
  __syncthreads();
  if (threadIdx.x == 0) out[0] = abort_flag == 1u ? 1 : 3;
}

inline void launch_wait_probe(int* out, cudaStream_t stream, int& rc) {
  wait_probe_kernel<<<1, 64, 0, stream>>>(out);
  rc = cudaGetLastError() == cudaSuccess ? 0 : 8;
}

// The end of a kernel whose wait ran out, with one copy issued just before: the CTA stays until the copy has landed.
// out[0]: as above; out[1]: thousands of cycles the end took; out[2]: 1 when every copied byte was there when the CTA left.
static constexpr int kSettleBytes = 8192;
__global__ void settle_probe_kernel(const uint8_t* src, int* out) {
  __shared__ alignas(128) uint8_t buf[kSettleBytes];
  __shared__ uint64_t bar, landed;
  __shared__ uint32_t abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    fray::sm100::mbar_init(&bar, 1);
    fray::sm100::mbar_init(&landed, 1);
    fray::sm100::fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x < 32) fray::sm100::mbar_wait(&bar, 0, &abort_flag, kProbeSite, kProbeExtra);
  if (threadIdx.x == 0) {
    fray::sm100::mbar_expect_tx(&landed, kSettleBytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     fray::sm100::smem_u32(buf)), "l"(src), "r"(kSettleBytes), "r"(fray::sm100::smem_u32(&landed))
                 : "memory");
  }
  __syncthreads();
  const long long t0 = clock64();
  if (*reinterpret_cast<volatile uint32_t*>(&abort_flag) == 1u) fray::sm100::settle_after_abort();
  __syncthreads();
  if (threadIdx.x == 0) {
    out[0] = abort_flag == 1u ? 1 : 3;
    out[1] = static_cast<int>((clock64() - t0) / 1000);
    out[2] = fray::sm100::mbar_try_wait(&landed, 0) ? 1 : 0;
    if (out[2] == 0) {  // not expected: leave only when it has landed
      uint32_t flag = 0;
      fray::sm100::mbar_wait(&landed, 0, &flag, kProbeSite + 1);
    }
  }
}

inline void launch_settle_probe(const int* src, int* out, cudaStream_t stream, int& rc) {
  settle_probe_kernel<<<1, 64, 0, stream>>>(reinterpret_cast<const uint8_t*>(src), out);
  rc = cudaGetLastError() == cudaSuccess ? 0 : 8;
}

}  // namespace fray_test
