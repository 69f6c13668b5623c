// Helpers of the tcgen05 / TMEM kernels: fp32 operands as three bf16 terms (x = hi + mid + lo, 8 + 8 + 8 mantissa bits,
// each residual computed exactly in fp32), packed in the tensor core's shared-memory layout so that a kernel fetches an
// operand tile with one bulk copy; MMA, commit, fence, TMEM-load and bounded-wait wrappers.
//
// Operand layout (K-major, no swizzle): 8 x 8 bf16 "core matrices" of 128 contiguous bytes (8 rows of 16 bytes); byte
// offset of (r, k) in a [128][32] tile = (r/8)*512 + (k/8)*128 + (r%8)*16 + (k%8)*2, i.e. 128 B between the 8-wide K
// groups of an MMA (leading offset), 512 B between groups of 8 rows (stride offset).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "kernels_mega.cuh"  // mbarrier / TMA helpers
#include "tg_common.cuh"

namespace tg {

constexpr int TC_BM = 128, TC_BK = 32;
constexpr int TC_TILE_BYTES = TC_BM * TC_BK * 2;  // 8 KiB: one [128][32] bf16 operand tile
constexpr int TC_SPIN_CAP = 1 << 24;

// ------------------------------------------------------------------ split + pack
// out: [3 terms][m_tiles][k_blocks][TC_TILE_BYTES]; rows >= M are zero.
// fp32 x[8] (8 consecutive k of one row) -> the three bf16 terms, stored at the operand-layout offset
__device__ __forceinline__ void tc_pack8(__nv_bfloat16 *out, size_t term_stride, int k_blocks, int row, int k8, const float (&x)[8]) {
	__align__(16) __nv_bfloat16 hi[8], mid[8], lo[8];
#pragma unroll
	for (int i = 0; i < 8; i++) {
		hi[i] = __float2bfloat16_rn(x[i]);
		const float r1 = x[i] - __bfloat162float(hi[i]);  // exact
		mid[i] = __float2bfloat16_rn(r1);
		const float r2 = r1 - __bfloat162float(mid[i]);   // exact
		lo[i] = __float2bfloat16_rn(r2);
	}
	const int mt = row / TC_BM, r = row % TC_BM, kb = (8 * k8) / TC_BK, kc = ((8 * k8) % TC_BK) / 8;
	const size_t off = (size_t(mt) * k_blocks + kb) * (TC_TILE_BYTES / 2) + (r / 8) * 256 + kc * 64 + (r % 8) * 8;
	*reinterpret_cast<uint4 *>(out + off) = *reinterpret_cast<const uint4 *>(hi);
	*reinterpret_cast<uint4 *>(out + term_stride + off) = *reinterpret_cast<const uint4 *>(mid);
	*reinterpret_cast<uint4 *>(out + 2 * term_stride + off) = *reinterpret_cast<const uint4 *>(lo);
}

// Work item c of a packing kernel -> (row, group of 8 consecutive k). Eight consecutive items are the eight rows
// of a core matrix at the same k group, so that a warp's 16-byte stores fill whole 128-byte lines of the packed
// tile (items in row-major order wrote every other 16 bytes of a line); each thread still reads 32 contiguous
// bytes of its row (one sector).
__device__ __forceinline__ void tc_chunk_to_row_k8(size_t c, int k8s, int &row, int &k8) {
	const size_t g = c / (size_t(8) * k8s);          // group of 8 rows
	const int w = int(c - g * (size_t(8) * k8s));    // item inside the group
	row = int(g) * 8 + (w & 7);
	k8 = w >> 3;
}

__global__ void __launch_bounds__(256) split_pack_kernel(const float *A, __nv_bfloat16 *out, int M, int K, int m_tiles) {
	pdl_trigger();
	pdl_wait();
	const int k_blocks = K / TC_BK;
	A += size_t(blockIdx.y) * M * K;  // blockIdx.y: one of several matrices behind each other
	out += size_t(blockIdx.y) * 3 * m_tiles * k_blocks * (TC_TILE_BYTES / 2);
	const size_t n_chunks = size_t(m_tiles) * TC_BM * (K / 8);  // one thread per (row, 8 consecutive k)
	const size_t term_stride = size_t(m_tiles) * k_blocks * (TC_TILE_BYTES / 2);
	for (size_t c = size_t(blockIdx.x) * blockDim.x + threadIdx.x; c < n_chunks; c += size_t(gridDim.x) * blockDim.x) {
		int row, k8;
		tc_chunk_to_row_k8(c, K / 8, row, k8);
		float x[8];
		if (row < M) {
			const float4 a = *reinterpret_cast<const float4 *>(A + size_t(row) * K + 8 * k8);
			const float4 b = *reinterpret_cast<const float4 *>(A + size_t(row) * K + 8 * k8 + 4);
			x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
		} else {
#pragma unroll
			for (int i = 0; i < 8; i++) x[i] = 0.0f;
		}
		tc_pack8(out, term_stride, k_blocks, row, k8, x);
	}
}

// ------------------------------------------------------------------ tcgen05 helpers
// shared-memory matrix descriptor: K-major, no swizzle, LBO 128 B, SBO 512 B
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t smem_addr) {
	uint64_t d = 0;
	d |= uint64_t((smem_addr & 0x3FFFF) >> 4);   // start address, 16-byte units
	d |= uint64_t(128 >> 4) << 16;               // leading-dimension byte offset (next 8 k)
	d |= uint64_t(512 >> 4) << 32;               // stride-dimension byte offset (next 8 rows)
	d |= uint64_t(1) << 46;                      // descriptor version of this architecture
	return d;                                    // base offset 0, layout type 0 = no swizzle
}
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
