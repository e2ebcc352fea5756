"""Device buffers after a failed allocation or copy, with a stand-in for the CUDA calls.  Host only.

Buffers that outlive a call are tested by their length, so a length without memory
behind it would send the next call's kernels through a null pointer."""
import os
import shutil
import subprocess

import pytest
from conftest import REPO

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
CSRC = os.path.join(REPO, "euler3d_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "devbuf.hpp"

static bool no_memory = false, no_copy = false;
static cudaError_t last = cudaSuccess;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
	if (no_memory) return last = cudaErrorMemoryAllocation;
	*p = std::malloc(n);
	return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
	if (no_copy) return cudaErrorInvalidValue;
	std::memcpy(d, s, n);
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
	const cudaError_t e = last;
	last = cudaSuccess;
	return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }
}

#define EXPECT(x)                                         \
	do {                                                  \
		if (!(x)) {                                       \
			std::printf("line %d: %s\n", __LINE__, #x);   \
			return 1;                                     \
		}                                                 \
	} while (0)

template <class F>
static bool throws(F f) {
	try {
		f();
	} catch (const e3d::Error& e) {
		return e.code == E3D_ERR_CUDA;
	}
	return false;
}

int main() {
	e3d::DevBuf<double> b;
	const std::vector<double> h{1., 2., 3.};
	// first allocation, growth and upload without memory: empty afterwards, no error left behind, and a retry works
	for (int held : {0, 2}) {
		b.reserve(held);
		no_memory = true;
		EXPECT(throws([&] { b.reserve(4); }));
		EXPECT(b.n == 0 && b.p == nullptr && last == cudaSuccess);
		EXPECT(throws([&] { b.upload(h); }));
		EXPECT(b.n == 0 && b.p == nullptr && last == cudaSuccess);
		no_memory = false;
		b.reserve(4);
		EXPECT(b.n == 4 && b.p != nullptr);
		b.free();
	}
	// a copy that failed leaves no length with undefined values behind
	no_copy = true;
	EXPECT(throws([&] { b.upload(h); }));
	EXPECT(b.n == 0 && b.p == nullptr);
	no_copy = false;
	b.upload(h);
	EXPECT(b.n == 3 && b.p[2] == 3.);
	// room that is there is kept
	double* p = b.p;
	b.reserve(2);
	EXPECT(b.p == p && b.n == 3);
	b.alloc(0);
	EXPECT(b.p == nullptr && b.n == 0);
	return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_length_matches_memory_after_failure(tmp_path):
    src, exe = tmp_path / "devbuf.cpp", tmp_path / "devbuf"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}/include", str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
