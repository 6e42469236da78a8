// Compressed 8-wide BVH for traversal, converted on the GPU from the binary
// Karras hierarchy of an LBVH build (the same tree whose collapsed form is
// exported in the reference's BvhNode layout).
//
// The format follows Ylitie, Karras and Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017): child boxes are
// stored as 8-bit offsets on a per-node power-of-two grid, internal children
// are stored contiguously, leaf primitives of a node are stored contiguously,
// and children are placed in slots by direction octant so that a ray visits
// them roughly near to far without sorting. The meta byte (a unary count above
// an offset, 24 + slot for internal children) and the way a ray turns it into
// its hit masks and its octant's order (wide_node_test) are the paper's too.
// The margin, the rounding, the leaf sizes and the conversion are this
// project's own:
//
//   * 80-byte node, five 16-byte loads;
//   * every quantised box contains its child's exact box with a margin of one
//     grid step on every side (directed rounding), so that the box test,
//     t = (q + 2^15) * (2^e * invDir) + ((p - origin) * invDir - 2^15 * 2^e * invDir)
//     with the second term rounded outwards (wide_traverse.cuh), never culls a
//     box that contains a hit point (the step is far larger than the rounding
//     error of the rest);
//   * leaves hold at most wide_leaf_max primitives of one contiguous range;
//     meta[slot] = (one bit per primitive << 5) | offset, offset relative to
//     the node's primitive base, and (1 << 5) | (24 + slot) for an internal
//     child: shifting the upper three bits by the lower five and or-ing the
//     hit slots gives the node's hit primitives in bits 0-23 and its hit
//     internal children in bits 24-31 of one word.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mb {

constexpr int WIDE_LEAF_MAX = 3;       // primitives per leaf in object hierarchies, at most
// Primitives per leaf of an object of n primitives. Leaves of two hold their
// primitives closer and cost a ray more nodes: per iteration, leaves of 3 / 2 /
// 1, 4 096 instances 720p 12.9 / 12.3 / 12.1 ms, plane 1.50 / 1.45 / 1.47 ms,
// icosphere 1080p 2.89 / 2.85 / 2.90 ms; but the cut-outs' objects of up to two
// dozen primitives, mostly one node each with leaves of three, 1.61 / 1.67 / 1.67.
// The line at 64 keeps those and is no optimum for others: 300 instances of an
// object of scattered triangles, quads and spheres, leaves of 3 / 2: 8
// primitives 3.72 / 3.74 ms, 16 9.2 / 7.0, 24 7.9 / 6.8, 32 6.7 / 6.4, 48 7.2 /
// 6.9, 64 6.6 / 6.4, 96 8.5 / 8.3, 128 8.0 / 7.3, 1 000 9.4 / 8.7.
inline int wide_leaf_max(size_t n) { return n <= 64 ? WIDE_LEAF_MAX : 2; }
constexpr int WIDE_TLAS_LEAF_MAX = 1;  // instances per leaf in the instance hierarchy

// In the second row's w of a primitive's soup: its kind, so that the traversal
// needs no primitive counts of the object.
constexpr int SOUP_TRIANGLE = 1;

struct alignas(16) WideNode {
	float p[3];            // grid origin
	uint32_t eimask;       // biased exponents ex | ey << 8 | ez << 16, internal-slot mask << 24
	uint32_t childBase;    // index of the first internal child
	uint32_t primBase;     // first slot of this node's leaf primitives
	uint32_t meta[2];      // per slot (unary count << 5) | offset, (1 << 5) | (24 + slot) internal, 0 empty
	uint32_t qlo[3][2];    // per axis, 8 slots of 8 bits
	uint32_t qhi[3][2];
};
static_assert(sizeof(WideNode) == 80, "WideNode layout");

// Upper bound on the number of wide nodes for n primitives: every node with
// eight children expands seven binary nodes of its own; the others are
// disjoint subtrees of more than leafMax primitives.
inline size_t wide_node_capacity(size_t n, int leafMax) { return n / 7 + n / size_t(leafMax + 1) + 2; }

struct WideBuildArgs {
	int n;                          // leaves of the binary tree (primitives in use)
	int numInternal;                // n - 1
	int leafMax;
	const int32_t* children;        // 2 per binary internal node
	const int2* ranges;             // first/last sorted leaf per binary internal node
	const float4* nodeData;         // 2 per binary node: min.xyz, max.xyz (exact boxes)
	const int32_t* sortedIds;       // sorted leaf index -> primitive / instance id
	WideNode* nodes;                // capacity wide_node_capacity(n, leafMax)
	int32_t* prims;                 // n: wide leaf slot -> primitive / instance id
	uint32_t nodeCapacity;
	uint32_t* counters;             // device scratch, WIDE_COUNTERS entries
	int2* queueA;                   // device scratch, nodeCapacity entries each
	int2* queueB;
};
constexpr int WIDE_COUNTERS = 8;

// Converts the binary tree into the wide one on `stream`. Reads back the
// node count once (one synchronisation). Returns cudaErrorInvalidValue if
// the capacity was exceeded or the levels did not terminate.
cudaError_t build_wide(const WideBuildArgs& a, int32_t* numNodesOut, cudaStream_t stream);

} // namespace mb
