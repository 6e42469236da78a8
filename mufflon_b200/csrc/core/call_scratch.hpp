// Device memory that a call needs only while it runs.
#pragma once

#include <cstddef>
#include <cuda_runtime_api.h>

namespace mb {

// Kept for the next call (gradient replays, ray queries): allocating and
// freeing it took longer than many of these calls (64 K ray queries 2.0 ms with
// it, 0.4 without; the gradient of a 512 x 512 texture 23 and 14 ms).
// Grow-only; what exceeds KEEP is given back when the call ends. Used under the
// instance's iterationMutex, on its stream, through CallScratchUse.
struct CallScratch {
	static constexpr size_t KEEP = size_t(512) << 20;
	char* device = nullptr;
	size_t bytes = 0;
	cudaError_t reserve(size_t need) {
		if(need <= bytes) return cudaSuccess;
		release();
		void* p = nullptr;
		const cudaError_t e = cudaMalloc(&p, need);
		if(e != cudaSuccess) return e;
		device = static_cast<char*>(p);
		bytes = need;
		return cudaSuccess;
	}
	void release() {
		cudaFree(device);
		device = nullptr;
		bytes = 0;
	}
};

// One call's use of the scratch memory. However the call ends, with its result
// or by an exception, no copy or kernel of its own is left on the stream (they
// reach into the caller's arrays) and the memory beyond KEEP is given back.
class CallScratchUse {
public:
	CallScratchUse(CallScratch& scratch, cudaStream_t stream) : m_scratch(scratch), m_stream(stream) {}
	CallScratchUse(const CallScratchUse&) = delete;
	CallScratchUse& operator=(const CallScratchUse&) = delete;
	~CallScratchUse() {
		if(!m_idle) cudaStreamSynchronize(m_stream);
		if(m_scratch.bytes > CallScratch::KEEP) m_scratch.release();
	}
	cudaError_t reserve(size_t need) { return m_scratch.reserve(need); }
	char* data() const { return m_scratch.device; }
	// The end of a call that succeeds: waits for the stream.
	cudaError_t finish() {
		const cudaError_t e = cudaStreamSynchronize(m_stream);
		m_idle = e == cudaSuccess;
		return e;
	}
private:
	CallScratch& m_scratch;
	cudaStream_t m_stream;
	bool m_idle = false;
};

} // namespace mb
