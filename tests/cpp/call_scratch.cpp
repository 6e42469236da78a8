// The kept call scratch over a fake of the CUDA runtime's allocation calls.
// Prints a line per check that fails; exits with their number.
#include "../../mufflon_b200/csrc/core/call_scratch.hpp"
#include <cstdio>
#include <stdexcept>

namespace {
size_t g_live = 0;     // bytes allocated
int g_blocks = 0, g_syncs = 0;
bool g_fail = false;   // the next allocation fails
size_t g_size[64];
int g_failures = 0;
void check(bool ok, const char* what) {
	if(!ok) { ++g_failures; std::printf("failed: %s\n", what); }
}
} // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
	if(g_fail) return cudaErrorMemoryAllocation;
	for(int i = 1; i < 64; ++i)
		if(!g_size[i]) {
			g_size[i] = n;
			g_live += n;
			++g_blocks;
			*p = reinterpret_cast<void*>(size_t(i) << 40);
			return cudaSuccess;
		}
	return cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
	if(!p) return cudaSuccess;
	size_t& n = g_size[size_t(p) >> 40];
	check(n > 0, "a block is freed once");
	g_live -= n;
	--g_blocks;
	n = 0;
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++g_syncs; return cudaSuccess; }
}

int main() {
	using namespace mb;
	constexpr size_t MB = size_t(1) << 20;
	CallScratch s;
	{ CallScratchUse u(s, nullptr); u.reserve(MB); u.finish(); }
	check(s.bytes == MB && g_live == MB, "a small call's memory is kept");
	check(g_syncs == 1, "a call that succeeds waits once");
	{ CallScratchUse u(s, nullptr); u.reserve(MB / 2); u.finish(); }
	check(s.bytes == MB && g_blocks == 1, "a smaller call takes what is there");
	{ CallScratchUse u(s, nullptr); u.reserve(CallScratch::KEEP); u.finish(); }
	check(s.bytes == CallScratch::KEEP && g_blocks == 1, "up to the bound it is kept");
	{ CallScratchUse u(s, nullptr); u.reserve(CallScratch::KEEP + 1); u.finish(); }
	check(s.bytes == 0 && s.device == nullptr && g_live == 0, "beyond the bound it is given back");
	g_syncs = 0;
	try {
		CallScratchUse u(s, nullptr);
		u.reserve(CallScratch::KEEP + MB);
		throw std::runtime_error("a CUDA call fails");
	} catch(const std::runtime_error&) {}
	check(s.bytes == 0 && g_live == 0, "a call that throws gives back what exceeds the bound");
	check(g_syncs == 1, "a call that throws waits for its copies");
	try {
		CallScratchUse u(s, nullptr);
		u.reserve(MB);
		throw std::runtime_error("a CUDA call fails");
	} catch(const std::runtime_error&) {}
	check(s.bytes == MB && g_live == MB, "and keeps the rest");
	g_fail = true;
	{ CallScratchUse u(s, nullptr); check(u.reserve(2 * MB) == cudaErrorMemoryAllocation, "the failure is reported"); }
	check(s.bytes == 0 && s.device == nullptr && g_live == 0, "nothing is kept of a failed allocation");
	g_fail = false;
	{ CallScratchUse u(s, nullptr); check(u.reserve(MB) == cudaSuccess && u.data() != nullptr, "the next call allocates again"); }
	s.release();
	check(g_blocks == 0, "released");
	return g_failures;
}
