// What the samplers on host buffers work in, and the order of a call's copies and launches (plain host code over the CUDA
// runtime's calls, so that a test can drive its error paths without a GPU).
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "tg_status.h"

namespace {
// A stream, device memory and pinned staging, kept by the calling thread (so no two threads share one) and given back when the
// thread ends. Allocating and freeing these per call took several times the work itself. Kept up to HOST_WS_MAX bytes each; a
// larger call takes and frees its own.
constexpr size_t HOST_WS_MAX = size_t(8) << 20;
constexpr int HOST_WS_CHUNKS = 4;  // copies to and from the caller's pageable memory overlap the transfers in chunks
struct HostWs {
	cudaStream_t st = nullptr;
	cudaEvent_t ev[HOST_WS_CHUNKS] = {};
	uint8_t *dev = nullptr, *pin = nullptr;
	size_t dev_bytes = 0, pin_bytes = 0;
	void release() {
		if (st) cudaStreamSynchronize(st);
		for (cudaEvent_t &e : ev)
			if (e) cudaEventDestroy(e);
		cudaFree(dev);
		cudaFreeHost(pin);
		if (st) cudaStreamDestroy(st);
		cudaGetLastError();
		st = nullptr;
		for (cudaEvent_t &e : ev) e = nullptr;
		dev = pin = nullptr;
		dev_bytes = pin_bytes = 0;
	}
	int reserve(size_t d, size_t p) {
		if (!st) {
			TG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
			for (cudaEvent_t &e : ev) TG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
		}
		if (d > dev_bytes) {
			cudaFree(dev);
			dev = nullptr;
			dev_bytes = 0;
			TG_CUDA(cudaMalloc(reinterpret_cast<void **>(&dev), d));
			dev_bytes = d;
		}
		if (p > pin_bytes) {
			cudaFreeHost(pin);
			pin = nullptr;
			pin_bytes = 0;
			TG_CUDA(cudaMallocHost(reinterpret_cast<void **>(&pin), p));
			pin_bytes = p;
		}
		return TG_OK;
	}
	// the caller's buffer -> dst (enqueued; the caller's memory has been read on return)
	int upload(uint8_t *dst, const void *src, size_t bytes) {
		const size_t ch = (bytes / HOST_WS_CHUNKS + 4095) & ~size_t(4095);
		for (size_t o = 0; o < bytes; o += ch) {
			const size_t n = std::min(ch, bytes - o);
			std::memcpy(pin + o, static_cast<const uint8_t *>(src) + o, n);
			TG_CUDA(cudaMemcpyAsync(dst + o, pin + o, n, cudaMemcpyHostToDevice, st));
		}
		return TG_OK;
	}
	// src -> the pinned buffer (enqueued), and from there into the caller's (complete on return)
	int download(const uint8_t *src, size_t bytes) {
		const size_t ch = (bytes / HOST_WS_CHUNKS + 4095) & ~size_t(4095);
		int k = 0;
		for (size_t o = 0; o < bytes; o += ch, k++) {
			TG_CUDA(cudaMemcpyAsync(pin + o, src + o, std::min(ch, bytes - o), cudaMemcpyDeviceToHost, st));
			TG_CUDA(cudaEventRecord(ev[k], st));
		}
		return TG_OK;
	}
	int deliver(void *dst, size_t bytes) {
		const size_t ch = (bytes / HOST_WS_CHUNKS + 4095) & ~size_t(4095);
		int k = 0;
		for (size_t o = 0; o < bytes; o += ch, k++) {
			TG_CUDA(cudaEventSynchronize(ev[k]));
			std::memcpy(static_cast<uint8_t *>(dst) + o, pin + o, std::min(ch, bytes - o));
		}
		return TG_OK;
	}
	~HostWs() {
		if (st || dev || pin) release();
	}
};

// One row of n logits in host memory through w: [token][uniform count][uniform] .. [key][ticket] ..., the row, the scratch of
// `scratch` bytes. head(w, row) launches what leaves the row's probabilities, walk(w, row) what leaves the token; with out = null there
// are none and head is not called.
template <class Head, class Walk>
int host_row(HostWs &w, const float *in, float *out, int n, size_t scratch, float randf, int *tok, Head head, Walk walk) {
	const size_t row = size_t(n) * 4, row_up = (row + 255) & ~size_t(255), dbytes = 256 + row_up + scratch;
	const bool fresh = dbytes > w.dev_bytes;
	auto steps = [&]() -> int {
		TG_TRY(w.reserve(dbytes, row_up + 256));
		if (fresh) TG_CUDA(cudaMemsetAsync(w.dev, 0, 256, w.st));  // (the kernels leave key and ticket zero)
		struct {
			int tok, count;
			float randf;
		} up = {0, 0, randf};
		uint8_t *pin_words = w.pin + row_up, *dev_row = w.dev + 256;
		std::memcpy(pin_words, &up, sizeof up);
		TG_CUDA(cudaMemcpyAsync(w.dev, pin_words, sizeof up, cudaMemcpyHostToDevice, w.st));
		TG_TRY(w.upload(dev_row, in, row));
		if (out) {
			// the probabilities are copied back before the walk for the token: it runs (28 us) while the host takes them out of the
			// pinned buffer (~18 us less of 270 a call)
			TG_TRY(head(w, dev_row));
			TG_TRY(w.download(dev_row, row));
		}
		TG_TRY(walk(w, dev_row));
		TG_CUDA(cudaMemcpyAsync(pin_words, w.dev, 4, cudaMemcpyDeviceToHost, w.st));
		if (out) TG_TRY(w.deliver(out, row));
		TG_CUDA(cudaStreamSynchronize(w.st));
		std::memcpy(tok, pin_words, 4);
		return TG_OK;
	};
	const int rc = steps();
	// a call that stopped half-way leaves copies in flight in the pinned buffer and key and ticket anywhere: the next one takes
	// a workspace of its own
	if (rc != TG_OK) w.release();
	return rc;
}
}  // namespace
