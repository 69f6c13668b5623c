// Helpers of the tcgen05 / TMEM kernels: MMA, commit, fence, TMEM-load and bounded-wait wrappers.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "kernels_mega.cuh"  // mbarrier / TMA helpers
#include "tg_common.cuh"

namespace tg {

constexpr int TC_SPIN_CAP = 1 << 24;

// ------------------------------------------------------------------ tcgen05 helpers
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
	asm volatile(
	    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
	    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
	    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
	    : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
	             "l"(src), "r"(bytes), "r"(smem_u32(bar))
	             : "memory");
}
// 32 lanes x 32 consecutive fp32 columns of TMEM -> 32 registers per thread (completion: tcgen05.wait::ld)
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
	asm volatile(
	    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
	    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
	    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
	      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
	      "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
	      "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
	    : "r"(taddr)
	    : "memory");
}
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, int *err) {
	int spins = 0;
	while (!mbar_try_wait(bar, parity)) {
		if (++spins > TC_SPIN_CAP) {
			*static_cast<volatile int *>(err) = 6;  // (a plain store: the word may lie in host memory)
			return false;
		}
	}
	return true;
}

// A warp that issues tcgen05 or bulk-copy instructions runs converged: all lanes walk its loop and wait, one elected lane
// issues. The operands of these instructions live in uniform registers; inside a single-lane branch with a conditional
// exit they are moved there by a loop around every instruction (measured: 260 clk per MMA against 40).
// one lane of the (converged) warp
__device__ __forceinline__ bool tc_elect() {
	uint32_t p;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
	return p != 0;
}
// Bounded wait without an exit: `cap` polls at most, and none any more once it has run out (cap = 0).
__device__ __forceinline__ void tc_wait_cap(uint64_t *bar, uint32_t parity, int &cap) {
	int z = 0;
	for (; z < cap && !mbar_try_wait(bar, parity); z++) {
	}
	cap = z < cap ? cap : 0;
}
// keys [M] ((value, column) as 64 bits: the larger value, among equal ones the lower column, is the larger key; 0 = no
// candidate) -> maximum (or -inf) and column (or -1) per row
__global__ void top1_unpack_kernel(const unsigned long long *keys, int M, float *max_out, int *idx_out) {
	const int r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r >= M) return;
	const unsigned long long k = keys[r];
	if (k == 0ull) {
		max_out[r] = -INFINITY;
		idx_out[r] = -1;
		return;
	}
	const uint32_t ord = uint32_t(k >> 32);
	max_out[r] = __uint_as_float((ord & 0x80000000u) ? (ord & 0x7FFFFFFFu) : ~ord);
	idx_out[r] = int(0xFFFFFFFFu - uint32_t(k));
}

}  // namespace tg
