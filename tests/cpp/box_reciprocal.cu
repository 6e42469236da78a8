// The box test's reciprocal against the correctly rounded one, clamped alike:
// for each exponent, how many of the 2^24 floats of that exponent and either
// sign differ in a bit.
#include "../../mufflon_b200/csrc/trace/wide_traverse.cuh"
#include <cstdio>
#include <cstdlib>

__global__ void compare(unsigned exponent, unsigned* differ) {
	const unsigned mantissa = blockIdx.x * blockDim.x + threadIdx.x; // 2^23 threads
	for(unsigned sign = 0; sign < 2; ++sign) {
		const float x = __uint_as_float(sign << 31 | exponent << 23 | mantissa);
		if(__float_as_uint(mb::box_rcp(x)) != __float_as_uint(mb::slab_rcp(x))) atomicAdd(differ, 1u);
	}
}

int main(int argc, char** argv) {
	unsigned* differ = nullptr;
	if(cudaMalloc(&differ, sizeof(unsigned)) != cudaSuccess) return 2;
	for(int i = 1; i < argc; ++i) {
		unsigned n = 0;
		cudaMemset(differ, 0, sizeof(unsigned));
		compare<<<(1u << 23) / 256, 256>>>(unsigned(std::atoi(argv[i]) + 127), differ);
		if(cudaMemcpy(&n, differ, sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
		std::printf("%u\n", n);
	}
	cudaFree(differ);
	return 0;
}
