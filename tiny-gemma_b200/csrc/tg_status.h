// Return codes of the host code: what a failed call leaves is in the thread's message (fail).
#pragma once
#include <string>

#include "../../include/tiny_gemma_b200.h"

namespace {
int fail(int code, const std::string &msg);
}

#define TG_CUDA(call)                                                                                   \
	do {                                                                                                \
		cudaError_t e__ = (call);                                                                       \
		if (e__ != cudaSuccess)                                                                         \
			return fail(TG_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e__));                 \
	} while (0)

#define TG_TRY(call)                \
	do {                            \
		int rc__ = (call);          \
		if (rc__ != TG_OK) return rc__; \
	} while (0)
