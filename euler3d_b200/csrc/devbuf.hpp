// Device buffers owned by the engine and the surrogate.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/e3d.h"
#include "mesh.hpp"

namespace e3d {

inline void cuda_ok(cudaError_t e, const char* what) {
	if (e != cudaSuccess) throw Error(E3D_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// n is the length of p, also after a call that threw: buffers that outlive a call
// are tested by n alone, and running out of memory is an error a caller may
// handle and come back from.
template <class T>
struct DevBuf {
	T* p = nullptr;
	size_t n = 0;
	void alloc(size_t count) {
		free();
		if (!count) return;
		T* q = nullptr;
		const cudaError_t e = cudaMalloc(&q, count * sizeof(T));
		if (e != cudaSuccess) cudaGetLastError();  // reported here, not by the next launch's check
		cuda_ok(e, "cudaMalloc");
		p = q;
		n = count;
	}
	// room for count values; what it held is lost when it grows
	void reserve(size_t count) {
		if (n < count) alloc(count);
	}
	void upload(const std::vector<T>& h) {
		alloc(h.size());
		if (h.empty()) return;
		cudaError_t e = cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
		// a copy from pageable memory may return with its last staged part still on the way, and the
		// solver's streams do not wait for the default stream
		if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
		if (e != cudaSuccess) free();
		cuda_ok(e, "upload");
	}
	void free() {
		if (p) cudaFree(p);
		p = nullptr;
		n = 0;
	}
	DevBuf() = default;
	DevBuf(const DevBuf&) = delete;
	DevBuf& operator=(const DevBuf&) = delete;
	~DevBuf() { free(); }
};

}  // namespace e3d
