// Drives the samplers' workspace for host buffers (host_ws.h) over a model of the CUDA runtime: what is enqueued on a stream runs when
// the host waits for it and not before, so whatever a failed call leaves in flight runs into the next one. Every runtime call and launch of
// a call is made to fail in turn; the call after it has to be right.
#include <cstdio>
#include <deque>
#include <functional>
#include <vector>

#include "../tiny-gemma_b200/csrc/host_ws.h"

namespace {
std::deque<std::function<void()>> queue;  // what is enqueued (one stream)
int calls = 0, fail_at = -1, live = 0;
bool fails() { return calls++ == fail_at; }
void run_queue() {
	while (!queue.empty()) {
		queue.front()();
		queue.pop_front();
	}
}
int fail(int code, const std::string &) { return code; }
// launches: the row is doubled and the key counted up; the token is the first value, if the key was left at zero before
int head(HostWs &w, uint8_t *row, int n) {
	if (fails()) return fail(TG_ECUDA, "head");
	uint8_t *dev = w.dev;
	queue.push_back([=] {
		float *v = reinterpret_cast<float *>(row);
		for (int i = 0; i < n; i++) v[i] *= 2.0f;
		++*reinterpret_cast<int *>(dev + 64);
	});
	return TG_OK;
}
int walk(HostWs &w, uint8_t *row, int key_wanted) {
	if (fails()) return fail(TG_ECUDA, "walk");
	uint8_t *dev = w.dev;
	queue.push_back([=] {
		int *key = reinterpret_cast<int *>(dev + 64);
		*reinterpret_cast<int *>(dev) = *key == key_wanted ? int(*reinterpret_cast<float *>(row)) : -1;
		*key = 0;
	});
	return TG_OK;
}
int sample(HostWs &w, std::vector<float> &v, bool probabilities, int *tok) {
	const int n = int(v.size());
	return host_row(
	    w, v.data(), probabilities ? v.data() : nullptr, n, 512, 0.5f, tok, [&](HostWs &x, uint8_t *row) { return head(x, row, n); },
	    [&](HostWs &x, uint8_t *row) { return walk(x, row, probabilities ? 1 : 0); });
}
// one call on its own values and what it has to give
bool right(HostWs &w, int n, float first, bool probabilities) {
	std::vector<float> v(n);
	for (int i = 0; i < n; i++) v[i] = first + float(i);
	int tok = -2;
	if (sample(w, v, probabilities, &tok) != TG_OK || tok != int(probabilities ? 2 * first : first)) return false;
	for (int i = 0; i < n; i++)
		if (v[i] != (probabilities ? 2.0f : 1.0f) * (first + float(i))) return false;
	return queue.empty();
}
}  // namespace

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
	if (fails()) return cudaErrorMemoryAllocation;
	live++;
	*s = reinterpret_cast<cudaStream_t>(8);
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) {
	live--;
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
	const bool f = fails();
	run_queue();
	return f ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
	if (fails()) return cudaErrorMemoryAllocation;
	live++;
	*e = reinterpret_cast<cudaEvent_t>(8);
	return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) {
	live--;
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return fails() || !e ? cudaErrorInvalidResourceHandle : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
	if (fails() || !e) return cudaErrorInvalidResourceHandle;
	run_queue();
	return cudaSuccess;
}
static cudaError_t take(void **p, size_t n) {
	if (fails()) return cudaErrorMemoryAllocation;
	live++;
	*p = ::operator new(n);
	std::memset(*p, 0xA5, n);
	return cudaSuccess;
}
static cudaError_t give(void *p) {
	if (!p) return cudaSuccess;
	live--;
	::operator delete(p);
	return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaMallocHost(void **p, size_t n) { return take(p, n); }
cudaError_t cudaFreeHost(void *p) { return give(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
	if (fails()) return cudaErrorUnknown;
	queue.push_back([=] { std::memcpy(d, s, n); });
	return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
	if (fails()) return cudaErrorUnknown;
	queue.push_back([=] { std::memset(d, v, n); });
	return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
}

int main() {
	int tried = 0;
	for (int n : {4, 8192, 65536})
		for (bool probabilities : {true, false})
			for (bool warm : {true, false})
				for (int at = 0;; at++) {
					HostWs w;
					if (warm && !right(w, n, 3.0f, probabilities)) return std::printf("a call without a failure is wrong\n"), 1;
					std::vector<float> v(n, 100.0f);
					int tok = -2;
					calls = 0;
					fail_at = at;
					const int rc = sample(w, v, probabilities, &tok);
					const bool reached = calls > at;
					fail_at = -1;
					if (!reached) {
						if (rc != TG_OK) return std::printf("error %d without a failure\n", rc), 1;
						break;
					}
					tried++;
					if (rc == TG_OK) return std::printf("failure %d of a call (n %d) is not reported\n", at, n), 1;
					if (!right(w, n, 7.0f, probabilities)) return std::printf("the call after failure %d (n %d, warm %d) is wrong\n", at, n, warm), 1;
				}
	if (live) return std::printf("%d objects are not given back\n", live), 1;
	std::printf("%d\n", tried);
	return 0;
}
