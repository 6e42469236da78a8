// GPU conversion of a binary Karras hierarchy into the compressed 8-wide
// format of wide.hpp, one kernel launch per level of the wide tree.
//
// Eight lanes turn one queued binary node into one wide node:
//   1. gather up to eight children by repeatedly opening the gathered binary
//      internal node with the largest surface area,
//   2. children with more than leafMax primitives become wide internal nodes
//      (queued for the next level), the others become leaves,
//   3. children are assigned to slots by direction octant: slot s prefers the
//      child whose centroid offset points along (s&4 ? -x : +x, s&2 ? -y : +y,
//      s&1 ? -z : +z); a greedy maximum of centroid-offset . octant vector,
//   4. boxes are quantised conservatively (see wide.hpp) and the node is
//      written; leaf primitives are copied into the node's primitive block.
#include "wide.hpp"
#include "../trace/dmath.cuh"

#include <cfloat>

namespace mb {
namespace {

enum { CNT_NODES = 0, CNT_PRIMS = 1, CNT_QUEUE = 2 /* 3 rotating counts */, CNT_ERROR = 5 };
constexpr int MAX_WIDE_LEVELS = 512;
constexpr float INV_252 = 1.0f / 252.0f;

__global__ void k_wide_init(uint32_t* counters, int2* queueA) {
	counters[CNT_NODES] = 1;
	counters[CNT_PRIMS] = 0;
	counters[CNT_QUEUE + 0] = 1;
	counters[CNT_QUEUE + 1] = 0;
	counters[CNT_QUEUE + 2] = 0;
	counters[CNT_ERROR] = 0;
	queueA[0] = make_int2(0, 0);
}

MBD void bin_box(const float4* nd, int b, f3& mn, f3& mx) {
	const float4 a = nd[2 * size_t(b)], c = nd[2 * size_t(b) + 1];
	mn = make3(a.x, a.y, a.z);
	mx = make3(c.x, c.y, c.z);
}
MBD float half_area(f3 mn, f3 mx) {
	const f3 d = mx - mn;
	return d.x * d.y + d.y * d.z + d.z * d.x;
}
MBD float comp(f3 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
MBD float pow2f(int e) { return __int_as_float((e + 127) << 23); }

constexpr int WIDE_THREADS = 128;
constexpr unsigned FULL = 0xffffffffu;

// Or of v over the eight lanes of a group.
MBD uint32_t group_or(uint32_t v) {
	for(int off = 4; off > 0; off >>= 1) v |= __shfl_xor_sync(FULL, v, off, 8);
	return v;
}
// Lane of the group with the largest value, the lowest lane of equal ones.
MBD int group_argmax(float& v, int lane8) {
	int i = lane8;
	for(int off = 4; off > 0; off >>= 1) {
		const float ov = __shfl_xor_sync(FULL, v, off, 8);
		const int oi = __shfl_xor_sync(FULL, i, off, 8);
		if(ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
	}
	return i;
}

// One level: eight lanes turn one queued binary node into one wide node, a
// lane holding one gathered child. (With one thread per node, whose opening
// steps and slot assignment are a serial chain of dependent loads and of
// nc * 8 * 8 compares over local arrays, every level took 34-91 us however
// few its nodes: the conversion of 1.31 M triangles 0.58 ms against 0.40, of
// 20 480 0.21 ms against 0.13.)
__global__ void __launch_bounds__(WIDE_THREADS) k_wide_level(WideBuildArgs A, const int2* __restrict__ qin,
                                                             const uint32_t* inCount, int2* qout, uint32_t* outCount,
                                                             uint32_t* zeroCount) {
	__shared__ __align__(16) unsigned char sNode[WIDE_THREADS / 8][sizeof(WideNode)];
	if(blockIdx.x == 0 && threadIdx.x == 0) *zeroCount = 0;
	const uint32_t count = *inCount;
	const int nI = A.numInternal;
	const int lane = int(threadIdx.x & 31u), lane8 = lane & 7;
	unsigned char* node = sNode[threadIdx.x >> 3];
	// Warp-uniform loop over four nodes at a time: their node, primitive and
	// queue allocations are one atomic each per warp.
	const uint32_t warps = gridDim.x * (WIDE_THREADS / 32);
	for(uint32_t first0 = 4u * (blockIdx.x * (WIDE_THREADS / 32) + (threadIdx.x >> 5)); first0 < count; first0 += 4u * warps) {
		const uint32_t item = first0 + uint32_t(lane >> 3);
		const bool valid = item < count;
		const int2 e = valid ? qin[item] : make_int2(0, 0);
		const int b = e.x;
		const uint32_t w = uint32_t(e.y);
		// 1. gather: open the largest internal child while a lane is free
		int ch = -1, nc = 2;
		float area = -1.0f; // leaves, free lanes (and NaN boxes) are not opened
		f3 mn = make3(0.0f, 0.0f, 0.0f), mx = mn;
		auto take = [&](int c) {
			ch = c;
			bin_box(A.nodeData, c, mn, mx);
			const float h = c < nI ? half_area(mn, mx) : -1.0f;
			area = h > -1.0f ? h : -1.0f;
		};
		if(lane8 < 2) take(A.children[2 * b + lane8]);
		for(;;) {
			float best = area;
			const int bi = group_argmax(best, lane8);
			const bool open = best > -1.0f && nc < 8;
			if(!__any_sync(FULL, open)) break;
			const int c = __shfl_sync(FULL, ch, bi, 8);
			if(open) {
				if(lane8 == bi) take(A.children[2 * c]);
				else if(lane8 == nc) take(A.children[2 * c + 1]);
				++nc;
			}
		}
		// 2. classify
		const bool used = lane8 < nc;
		int first = 0, cnt = 0;
		if(used) {
			if(ch >= nI) { first = ch - nI; cnt = 1; }
			else { const int2 r = A.ranges[ch]; first = r.x; cnt = r.y - r.x + 1; }
		}
		const bool inner = used && cnt > A.leafMax;
		// 3. octant slots: repeatedly the largest (centroid offset . octant vector)
		// of a free child and a free slot
		f3 pmn, pmx;
		bin_box(A.nodeData, b, pmn, pmx);
		const f3 off = (mn + mx) * 0.5f - (pmn + pmx) * 0.5f;
		float score[8];
#pragma unroll
		for(int s = 0; s < 8; ++s)
			score[s] = ((s & 4) ? -off.x : off.x) + ((s & 2) ? -off.y : off.y) + ((s & 1) ? -off.z : off.z);
		uint32_t freeSlots = 0xFFu;
		int slot = -1;
		for(int round = 0; round < 8; ++round) {
			float best = -INFINITY;
			int bs = __ffs(int(freeSlots)) - 1; // (every score NaN: the first free slot)
#pragma unroll
			for(int s = 0; s < 8; ++s)
				if((freeSlots >> s & 1u) && score[s] > best) { best = score[s]; bs = s; }
			// assigned children and free lanes lose to every free child
			float key = used && slot < 0 ? (best > -FLT_MAX ? best : -FLT_MAX) : -INFINITY;
			const int bi = group_argmax(key, lane8);
			const int ws = __shfl_sync(FULL, bs, bi, 8);
			if(round < nc) {
				if(lane8 == bi) slot = ws;
				freeSlots &= ~(1u << ws);
			}
		}
		const uint32_t innerSlots = group_or(inner ? 1u << slot : 0u);
		const uint32_t leafCounts = group_or(used && !inner ? uint32_t(cnt) << (2 * slot) : 0u); // two bits a slot
		const uint32_t below = used ? (1u << slot) - 1u : 0u;
		const uint32_t belowLeaf = leafCounts & ((1u << (2 * (used ? slot : 0))) - 1u);
		const uint32_t innerRank = uint32_t(__popc(innerSlots & below));
		const uint32_t primOffset = uint32_t(__popc(belowLeaf & 0x5555u) + 2 * __popc(belowLeaf & 0xAAAAu));
		const uint32_t nInner = valid ? uint32_t(__popc(innerSlots)) : 0u;
		const uint32_t nPrims = valid ? uint32_t(__popc(leafCounts & 0x5555u) + 2 * __popc(leafCounts & 0xAAAAu)) : 0u;
		uint32_t preN = 0, preP = 0, totN = 0, totP = 0;
#pragma unroll
		for(int g = 0; g < 4; ++g) {
			const uint32_t gn = __shfl_sync(FULL, nInner, 8 * g), gp = __shfl_sync(FULL, nPrims, 8 * g);
			if(g < lane >> 3) { preN += gn; preP += gp; }
			totN += gn; totP += gp;
		}
		uint32_t bn = 0, bp = 0, bq = 0;
		if(lane == 0) {
			if(totN) { bn = atomicAdd(A.counters + CNT_NODES, totN); bq = atomicAdd(outCount, totN); }
			if(totP) bp = atomicAdd(A.counters + CNT_PRIMS, totP);
		}
		const uint32_t childBase = __shfl_sync(FULL, bn, 0) + preN;
		const uint32_t primBase = __shfl_sync(FULL, bp, 0) + preP;
		const uint32_t queueBase = __shfl_sync(FULL, bq, 0) + preN;
		bool write = valid;
		if(valid && (childBase + nInner > A.nodeCapacity || primBase + nPrims > uint32_t(A.n) || w >= A.nodeCapacity)) {
			if(lane8 == 0) atomicOr(A.counters + CNT_ERROR, 1u);
			write = false;
		}
		// 4. quantisation grid per axis, then every lane its child's bytes
		uint32_t* words = reinterpret_cast<uint32_t*>(node);
		float pgrid[3], inv[3];
		uint32_t ebytes = 0;
#pragma unroll
		for(int a = 0; a < 3; ++a) {
			const float lo = comp(pmn, a), hi = comp(pmx, a);
			const float ext = __fsub_ru(hi, lo);
			const float amax = fmaxf(fabsf(lo), fabsf(hi));
			const float need = fmaxf(__fmul_ru(ext, INV_252), amax * (1.0f / 1048576.0f));
			int ex = -100;
			if(need > 0.0f) { frexpf(need, &ex); }
			ex = max(-100, min(100, ex));
			const float scale = pow2f(ex);
			pgrid[a] = __fsub_rd(lo, scale);
			inv[a] = pow2f(-ex);
			ebytes |= uint32_t(ex + 127) << (8 * a);
		}
		// words: 0-2 grid origin, 3 exponents and mask, 4 child base, 5 primitive
		// base, 6-7 meta, 8-13 lower planes, 14-19 upper planes; empty slots are
		// lower 255, upper 0
		if(lane8 < 3) words[lane8] = __float_as_uint(lane8 == 0 ? pgrid[0] : (lane8 == 1 ? pgrid[1] : pgrid[2]));
		else if(lane8 == 3) words[3] = ebytes | (innerSlots << 24);
		else if(lane8 == 4) words[4] = childBase;
		else if(lane8 == 5) words[5] = primBase;
		else words[lane8] = 0u;
		if(lane8 < 6) { words[8 + lane8] = 0xFFFFFFFFu; words[14 + lane8] = 0u; }
		__syncwarp();
		bool bad = false;
		if(used && write) {
#pragma unroll
			for(int a = 0; a < 3; ++a) {
				const float l = floorf(__fsub_rd(comp(mn, a), pgrid[a]) * inv[a]) - 1.0f;
				const float h = ceilf(__fsub_ru(comp(mx, a), pgrid[a]) * inv[a]) + 1.0f;
				if(l < 0.0f || h > 255.0f) bad = true; // (NaN boxes of degenerate primitives quantise to slot 0)
				node[32 + 8 * a + slot] = (unsigned char)uint32_t(fminf(fmaxf(l, 0.0f), 255.0f));
				node[56 + 8 * a + slot] = (unsigned char)uint32_t(fminf(fmaxf(h, 0.0f), 255.0f));
			}
			if(inner) {
				node[24 + slot] = (unsigned char)((1 << 5) | (24 + slot));
				const uint32_t q = queueBase + innerRank;
				if(q < A.nodeCapacity) qout[q] = make_int2(ch, int(childBase + innerRank));
				else bad = true;
			} else {
				node[24 + slot] = (unsigned char)((((1 << cnt) - 1) << 5) | primOffset);
				for(int j = 0; j < cnt; ++j) A.prims[primBase + primOffset + uint32_t(j)] = A.sortedIds[first + j];
			}
		}
		if(bad) atomicOr(A.counters + CNT_ERROR, 2u);
		__syncwarp();
		if(write && lane8 < 5)
			reinterpret_cast<float4*>(A.nodes + w)[lane8] = reinterpret_cast<const float4*>(node)[lane8];
		__syncwarp();
	}
}

} // namespace

cudaError_t build_wide(const WideBuildArgs& a, int32_t* numNodesOut, cudaStream_t stream) {
	*numNodesOut = 0;
	if(a.n < 2) return cudaSuccess;
	k_wide_init<<<1, 1, 0, stream>>>(a.counters, a.queueA);
	int dev = 0, sms = 148;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	constexpr int NODES_PER_BLOCK = WIDE_THREADS / 8;
	const unsigned grid = unsigned(std::max(1, std::min(sms * 16, int((a.nodeCapacity + NODES_PER_BLOCK - 1) / NODES_PER_BLOCK))));
	// Levels launched before the queue length is read back: up to eight leaves
	// are one node; launches over an empty queue cost about 2 us each.
	const int levelsPerCheck = a.n <= 8 ? 1 : a.n <= 4096 ? 6 : 12;
	uint32_t host[WIDE_COUNTERS];
	for(int level = 0; level < MAX_WIDE_LEVELS;) {
		for(int k = 0; k < levelsPerCheck; ++k, ++level) {
			const int2* qin = (level & 1) ? a.queueB : a.queueA;
			int2* qout = (level & 1) ? a.queueA : a.queueB;
			uint32_t* cin = a.counters + CNT_QUEUE + level % 3;
			uint32_t* cout = a.counters + CNT_QUEUE + (level + 1) % 3;
			uint32_t* czero = a.counters + CNT_QUEUE + (level + 2) % 3;
			k_wide_level<<<grid, WIDE_THREADS, 0, stream>>>(a, qin, cin, qout, cout, czero);
		}
		cudaError_t e = cudaMemcpyAsync(host, a.counters, sizeof(host), cudaMemcpyDeviceToHost, stream);
		if(e == cudaSuccess) e = cudaStreamSynchronize(stream);
		if(e != cudaSuccess) return e;
		if(host[CNT_ERROR]) return cudaErrorInvalidValue;
		if(host[CNT_QUEUE + level % 3] == 0) {
			if(host[CNT_PRIMS] != uint32_t(a.n)) return cudaErrorInvalidValue;
			*numNodesOut = int32_t(host[CNT_NODES]);
			return cudaSuccess;
		}
	}
	return cudaErrorInvalidValue;
}

} // namespace mb
