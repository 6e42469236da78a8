// Traversal of the compressed 8-wide hierarchies (lbvh/wide.hpp) for closest
// hits and shadow rays; the counterpart of intersection.cu:319-492 and
// 624-753 of the reference, over a different hierarchy with the same result.
//
// One loop runs both levels. The state of a ray is
//   * a node group: the child base of the last visited node, its internal-slot
//     mask and the still unvisited hit internal children as bits in
//     traversal order (bit 24 + (slot ^ octant of the ray's direction), so
//     that the highest bit is roughly the nearest child),
//   * a primitive group: the last visited node's primitive base and one bit
//     per primitive of its hit leaves,
//   * a stack of node groups (and, at the instance level, primitive groups of
//     instances not yet entered).
// Entering an instance transforms the ray into object space and remembers the
// stack depth; when the object level's groups are exhausted at that depth the
// world ray is restored. Every step visits one node (eight box tests that do
// the same arithmetic in every lane) and then that node's hit primitives.
//
// What bounds it: divergence and instruction issue (ncu, incoherent bounce of
// the icosphere: 54 % of issue slots, 41 % of the ALU pipe, memory below 10 %
// of its peak; see warp_step), so the step is written for few
// instructions and registers: box planes from biased bytes in packed
// multiply-adds, hit masks by shifts of precomputed bytes, reciprocals without
// special cases for boxes, one record per instance, no world-ray shear
// constants, entering an instance in the step that visits its root. Against a
// form with divisions, a subtraction per plane byte, out-of-line instance
// transforms and the prepared world ray in registers (same box, per iteration,
// both before the votes): trace stage of the 1080p icosphere 2.90 -> 2.12 ms,
// of 4 096 instances at 720p 15.4 -> 14.3 ms.
//
// The box test cannot cull a box that contains a hit point (wide.hpp), so the
// closest hit is the minimum of (world t, instance, primitive) over all
// primitive hits, exactly as with the binary hierarchy.
#pragma once

#include "intersect.cuh"
#include "../lbvh/wide.hpp"

namespace mb {

constexpr int WIDE_STACK = 64;

// The traversal stack of one ray. The node group being visited lives in
// registers (WideTracerT::ngBase/ngMask, pgBase/pgHits); pushed groups
// go to this per-thread array in local memory, which the L1 cache serves.
// (Keeping the first 4, 8 or 16 entries in shared memory instead, thread-
// interleaved, measured 5-7 % slower in the trace kernel on the B200.)
// The closest hit so far lies beside the stack: it is written when a nearer
// one is found and read at the end of the ray (or at equal distances).
struct LocalStack {
	uint2 e[WIDE_STACK];
	int2 hit;     // instance (-1: none yet), primitive
	float2 hitSp; // surface parameters
	MBD void put(int i, uint2 v) { e[i] = v; }
	MBD uint2 get(int i) const { return e[i]; }
};
// A node group is (child base, hit children in bits 24-31 | internal-slot mask
// in bits 0-7), a primitive group (primitive base, primitive bits 0-23): what
// is popped from the stack is a node group exactly when it exceeds PRIM_BITS.
constexpr uint32_t PRIM_BITS = 0x00FFFFFFu;
static_assert(8 * WIDE_LEAF_MAX <= 24 && 8 * WIDE_TLAS_LEAF_MAX <= 24, "primitive mask width");

// Sign bits of the reciprocal direction (of a zero component's as well).
MBD uint32_t ray_octant(f3 d) {
	return (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
}
// The root as the only child, in slot 0, of a virtual parent.
MBD uint32_t root_group(uint32_t oct) { return (1u << (24u + oct)) | 1u; }

// slab_rcp for the box tests: the hardware's approximate reciprocal and one
// Newton-Raphson step, r + r (1 - x r), of a component kept away from zero by
// 2^-64. It has the bits of slab_rcp for components below 2^126 in magnitude
// (above, the box test keeps every box); the approximate reciprocal alone
// differs from them in 13 % of all values, by up to 1.65 units of 2^-24. A
// correctly rounded division calls a routine for its special cases, for which
// the traversal kernels spilled (trace 1080p icosphere 1.90 ms, 1.83 this way;
// instances 720p 11.4 and 10.95 ms; cut-outs 1.30 and 1.19 ms).
MBD float box_rcp(float x) {
	x = copysignf(fmaxf(fabsf(x), 1.0f / 18446744073709551616.0f), x);
	float r;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return __fmaf_rn(r, __fmaf_rn(-x, r, 1.0f), r);
}
MBD f3 box_rcp3(f3 d) { return make3(box_rcp(d.x), box_rcp(d.y), box_rcp(d.z)); }

// Two fused multiply-adds in one instruction (sm_100's packed f32x2 form),
// each rounded like __fmaf_rn.
MBD unsigned long long pack2(float a, float b) {
	unsigned long long v;
	asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
	return v;
}
MBD void fma2(float qa, float qb, unsigned long long s, unsigned long long o, float& ra, float& rb) {
	unsigned long long v;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(pack2(qa, qb)), "l"(s), "l"(o));
	asm("mov.b64 {%0, %1}, %2;" : "=f"(ra), "=f"(rb) : "l"(v));
}

// Byte b (0..3) of w as the float 2^15 + byte: 0x4700bb00. The offset is
// folded into the additive constant of the box test (below), so a byte costs
// one instruction.
constexpr float QBYTE_BIAS = 32768.0f;
MBD float qbyte_biased(uint32_t w, int b) {
	return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7404u | (uint32_t(b) << 4)));
}

// Primitives other than triangles, out of line (rare in large scenes, and
// large code). The quad test's exact reciprocal of the dominant direction
// component is computed here; spheres need none.
struct PrimHit { float t; f2 uv; bool hit; };
MBD FastRay other_ray(const DLod& l, f3 o, f3 d, int p) {
	FastRay r;
	r.o = o; r.d = d;
	r.kx = r.ky = r.kz = 0;
	r.Sx = r.Sy = r.Sz = 0.0f;
	float inv = 0.0f;
	if(uint32_t(p) < l.numTriangles + l.numQuads) {
		const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
		inv = slab_rcp((ax < ay || ax < az) ? (ay >= az ? d.y : d.z) : d.x); // quad_test's axis d0
	}
	r.inv = make3(inv, inv, inv);
	return r;
}
static __device__ __noinline__ PrimHit other_prim_test(const DLod* l, f3 o, f3 d, int p) {
	PrimHit h;
	h.hit = prim_test(*l, other_ray(*l, o, d, p), 0, p, h.t, h.uv);
	return h;
}
// The alpha test's scene in kernels that were compiled with it. Whether it
// applies is the kernel's to say, not S.hasAlpha's: a batch with cut-outs in
// one job's scene runs such kernels over all of them, and the materials of the
// others name no alpha texture.
MBD AlphaCtx alpha_all(const DScene& S) {
	AlphaCtx a;
	a.materials = S.materials;
	a.textures = S.textures;
	return a;
}
static __device__ __noinline__ PrimHit other_prim_test_alpha(const DLod* l, f3 o, f3 d, int p, AlphaCtx alpha) {
	PrimHit h;
	h.hit = prim_test(*l, other_ray(*l, o, d, p), 0, p, h.t, h.uv, alpha);
	return h;
}

// Three-operand minimum and maximum of sm_100 (one instruction each; a NaN
// operand is dropped like fminf/fmaxf drop it).
MBD float min3_(float a, float b, float c) {
	float d;
	asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
	return d;
}
MBD float max3_(float a, float b, float c) {
	float d;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
	return d;
}

// Tests the eight child boxes of node `idx`; returns the child's node group
// and primitive group. A child is hit when
//   max(near planes, 0) <= min(far planes * (1 + 2^-20), tmaxBox).
// With a plane's byte read as q + 2^15, its distance is one multiply-add:
//   (q + 2^15) * s + (o - 2^15 * s),
// near and far plane of an axis in one packed instruction. The additive
// constants are rounded outwards, the near plane's down and the far plane's up,
// so their rounding (at most 2^-8 of a grid step, or 2^-23 of the offset if that
// is larger) only widens a box. That holds
// at any scale: where 2^15 * s overflows (grid steps from 2^49 on, and a ray
// along a coordinate axis), the near constant becomes -inf or stays the largest
// finite number, the far one +inf or stays the smallest, and the box is kept.
// The far-plane tolerance is applied to the per-node scale and offset, not per
// child, which moves a plane by far less than the grid step of margin every
// quantised box carries.
MBD void wide_node_test(const WideNode* nodes, uint32_t idx, f3 org, f3 inv, uint32_t oct, float tmaxBox,
                        uint32_t& ngBase, uint32_t& ngMask, uint32_t& pgBase, uint32_t& pgHits) {
	const float4* q = reinterpret_cast<const float4*>(nodes + idx);
	const float4 n0 = __ldg(q), n1 = __ldg(q + 1), n2 = __ldg(q + 2), n3 = __ldg(q + 3), n4 = __ldg(q + 4);
	const uint32_t eim = __float_as_uint(n0.w);
	auto axis = [](float grid, uint32_t ex, float o, float i, unsigned long long& s2, unsigned long long& o2) {
		const float s = __fmul_rn(__uint_as_float(ex << 23), i);
		const float t = __fmul_rn(__fsub_rn(grid, o), i);
		const float fs = __fmul_rn(s, BOX_FAR_SLACK), ft = __fmul_rn(t, BOX_FAR_SLACK);
		s2 = pack2(s, fs);
		o2 = pack2(__fmaf_rd(-QBYTE_BIAS, s, t), __fmaf_ru(-QBYTE_BIAS, fs, ft));
	};
	unsigned long long sx, sy, sz, ox, oy, oz;
	axis(n0.x, eim & 0xFFu, org.x, inv.x, sx, ox);
	axis(n0.y, (eim >> 8) & 0xFFu, org.y, inv.y, sy, oy);
	axis(n0.z, (eim >> 16) & 0xFFu, org.z, inv.z, sz, oz);
	const bool fx = (oct & 4u) != 0u, fy = (oct & 2u) != 0u, fz = (oct & 1u) != 0u;
	const uint32_t lx0 = __float_as_uint(n2.x), lx1 = __float_as_uint(n2.y);
	const uint32_t ly0 = __float_as_uint(n2.z), ly1 = __float_as_uint(n2.w);
	const uint32_t lz0 = __float_as_uint(n3.x), lz1 = __float_as_uint(n3.y);
	const uint32_t hx0 = __float_as_uint(n3.z), hx1 = __float_as_uint(n3.w);
	const uint32_t hy0 = __float_as_uint(n4.x), hy1 = __float_as_uint(n4.y);
	const uint32_t hz0 = __float_as_uint(n4.z), hz1 = __float_as_uint(n4.w);
	const uint32_t nx[2] = { fx ? hx0 : lx0, fx ? hx1 : lx1 }, fxw[2] = { fx ? lx0 : hx0, fx ? lx1 : hx1 };
	const uint32_t ny[2] = { fy ? hy0 : ly0, fy ? hy1 : ly1 }, fyw[2] = { fy ? ly0 : hy0, fy ? ly1 : hy1 };
	const uint32_t nz[2] = { fz ? hz0 : lz0, fz ? hz1 : lz1 }, fzw[2] = { fz ? lz0 : hz0, fz ? lz1 : hz1 };
	const uint32_t meta[2] = { __float_as_uint(n1.z), __float_as_uint(n1.w) };
	uint32_t hits = 0;
#pragma unroll
	for(int w = 0; w < 2; ++w) {
		// four slots at a time: an internal child's bit position (24 + slot,
		// the only ones with bits 3 and 4 set) is moved into traversal order
		const uint32_t inner = ((meta[w] & (meta[w] << 1)) & 0x10101010u) >> 4;
		const uint32_t pos = meta[w] ^ (oct * inner);
		const uint32_t bits = (meta[w] >> 5) & 0x07070707u;
#pragma unroll
		for(int b = 0; b < 4; ++b) {
			float tnx, tny, tnz, tfx, tfy, tfz;
			fma2(qbyte_biased(nx[w], b), qbyte_biased(fxw[w], b), sx, ox, tnx, tfx);
			fma2(qbyte_biased(ny[w], b), qbyte_biased(fyw[w], b), sy, oy, tny, tfy);
			fma2(qbyte_biased(nz[w], b), qbyte_biased(fzw[w], b), sz, oz, tnz, tfz);
			const float tnear = max3_(tnx, tny, fmax_(tnz, 0.0f));
			const float tfar = min3_(tfx, tfy, fmin_(tfz, tmaxBox));
			// (a funnel shift takes its distance modulo 32: the low five bits of the slot's byte)
			const uint32_t m = __funnelshift_l(0u, __byte_perm(bits, 0u, 0x4440u | uint32_t(b)), pos >> (8 * b));
			if(tnear <= tfar) hits |= m;
		}
	}
	ngBase = __float_as_uint(n1.x);
	ngMask = (hits & ~PRIM_BITS) | (eim >> 24);
	pgBase = __float_as_uint(n1.y);
	pgHits = hits & PRIM_BITS;
}

// Idle lanes of a persistent warp are refilled together once this many are idle
// (or none is busy): waiting for all 32 leaves lanes idle behind the longest
// ray, refilling one by one waits for the queue's loads in most passes. Trace
// per iteration, icosphere at 1080p and 4 096 instances at 720p: 8 lanes 2.01
// and 10.1 ms, 12 lanes 1.95 and 10.3 ms, 24 lanes 1.95 and 11.0 ms, all 32
// 2.11 and 12.4 ms.
constexpr int REFILL_LANES = 12;

// Lanes of every warp of a persistent launch that take work when `items` do
// not fill the launch: fewer rays or paths per warp, over more warps, diverge
// less, and a short queue is bound by the latency of its slowest warp. (64 x
// 64 box: 0.40 -> 0.27 ms an iteration; the light tracer's short late
// generations at 1080p: 3.13 -> 2.86 ms.)
MBD unsigned lanes_per_warp(unsigned items) {
	const unsigned warps = gridDim.x * (blockDim.x / 32u);
	return items >= 32u * warps ? 32u : (items + warps - 1u) / warps;
}

// Resumable traversal of one ray: init() sets it up, every step() enters a
// pending instance, visits at most one node and that node's hit primitives
// and leaves a finished instance, and returns true once the ray is finished. Kernels that refill
// lanes as soon as their ray finishes call step() from one loop shared by the
// whole warp. Alpha mode AM: ALPHA_NEVER, every surface is opaque (scenes
// without alpha textures, and the wireframe renderer's
// first_intersection<CURRENT_DEV, false>, wireframe_common.hpp:108);
// ALPHA_ALWAYS, the materials' alpha textures apply (kernels launched for
// scenes with alpha textures); ALPHA_SCENE, decided per step by the scene.
enum AlphaMode { ALPHA_NEVER = 0, ALPHA_ALWAYS = 1, ALPHA_SCENE = 2 };
template < int AM >
struct WideTracerT {
	f3 wo, wd;            // world ray as given
	f3 o, d, inv;         // ray of the current level (d: object level only)
	uint32_t axes;        // shear axes kx | ky << 2 | kz << 4 and constants of the triangle test (object level)
	float Sx, Sy, Sz;
	float scale;          // object-space length of a world-space unit
	float t;              // closest hit so far, or the incoming tmax; shadow rays: the segment's length
	const WideNode* nodes;
	const float4* soup;
	uint32_t oct, ngBase, ngMask, pgBase, pgHits;
	int inst, sp, instSp, steps; // steps: what is left of the scene's step limit (exceeded)
	bool any, done, occluded;

	template < class Stack >
	MBD HitRec hit(const Stack& stack) const {
		HitRec h;
		h.t = t; h.inst = stack.hit.x; h.prim = stack.hit.y; h.has = h.inst >= 0;
		h.sp = h.has ? make2(stack.hitSp.x, stack.hitSp.y) : make2(0.0f, 0.0f);
		return h;
	}

	template < class Stack >
	MBD void init(const DScene& S, f3 org, f3 dir, float tmax, bool anyHit, Stack& stack) {
		wo = org; wd = dir;
		any = anyHit;
		t = tmax; occluded = false;
		stack.hit = make_int2(-1, -1);
		sp = 0; instSp = -1; steps = S.maxSteps; inst = -1;
		ngBase = 0; ngMask = 0; pgBase = 0; pgHits = 0;
		done = S.activeInstances <= 0;
		if(S.activeInstances == 1) pgHits = 1u; // its instance is entered by the first step
		else if(S.tlasNumWide > 0) { to_world(S); ngMask = root_group(oct); }
		else done = true;
	}

	// The step limit counts node visits, instances taken from the stack (not the
	// one entered from the node that was just visited) and objects without a
	// hierarchy, at the event itself, so that step() and warp_step() abandon the
	// same rays. A visit is refused behind its box tests and an instance from the
	// stack when it is entered: with the checks before the tests and in pop(),
	// which runs in every pass, trace launches of the instanced scene took 11.2
	// instead of 11.0 ms an iteration.
	template < class C >
	MBD bool exceeded(C& cnt) {
		if(steps >= 0) return false;
		++cnt.errors;
		done = true;
		return true;
	}

	// Sets the world ray and the instance level's hierarchy.
	MBD void to_world(const DScene& S) {
		o = wo;
		inv = box_rcp3(wd);
		oct = ray_octant(inv);
		scale = 1.0f;
		nodes = S.tlasWide;
		instSp = -1;
	}

	// Transforms the ray into the object space of the instance in leaf slot
	// `slot` of the instance level (the arithmetic of instance_ray and
	// make_ray) and starts at its hierarchy's root.
	template < class C >
	MBD void enter(const DScene& S, uint32_t slot, C& cnt) {
		++cnt.instances;
		const float4* rec = reinterpret_cast<const float4*>(S.instRecs + slot);
		Mat34 W;
		W.r0 = __ldg(rec); W.r1 = __ldg(rec + 1); W.r2 = __ldg(rec + 2);
		const ulonglong2 ptr = __ldg(reinterpret_cast<const ulonglong2*>(rec + 3));
		const int2 np = __ldg(reinterpret_cast<const int2*>(rec + 4));
		inst = np.y;
		nodes = reinterpret_cast<const WideNode*>(ptr.x);
		soup = reinterpret_cast<const float4*>(ptr.y);
		const f3 dirO = xform_dir(W, wd);
		scale = len(dirO);
		o = xform_point(W, wo);
		d = dirO / scale;
		inv = box_rcp3(d);
		oct = ray_octant(inv);
		int kx, ky, kz;
		shear(d, kx, ky, kz, Sx, Sy, Sz);
		axes = uint32_t(kx) | uint32_t(ky) << 2 | uint32_t(kz) << 4;
		ngBase = 0; ngMask = 0; pgBase = 0; pgHits = 0;
		if(np.x >= 2) ngMask = root_group(oct);
		else {
			--steps;
			if(!exceeded(cnt)) pgHits = np.x == 1 ? 1u : 0u;
		}
		instSp = sp;
	}

	// One step. The hot kernels are compiled once per alpha mode and launched
	// with ALPHA_NEVER for scenes without alpha textures, so their step carries
	// no alpha code (any alpha check in a step shared by both kinds of scenes
	// made the trace stage 5-7 % slower: more registers spilled).
	template < class Stack, class C >
	MBD bool step(const DScene& S, C& cnt, Stack& stack) {
		if constexpr(AM == ALPHA_SCENE) {
			if(S.hasAlpha) return step_impl<true>(S, cnt, stack);
			return step_impl<false>(S, cnt, stack);
		} else {
			return step_impl<AM == ALPHA_ALWAYS>(S, cnt, stack);
		}
	}

	// The parts of a step, for a ray that has something to do there.
	template < class Stack, class C >
	MBD void enter_pending(const DScene& S, C& cnt, Stack& stack) {
		// instance leaves of the top level: enter one, keep the rest
		const uint32_t j = 31u - uint32_t(__clz(int(pgHits)));
		const uint32_t slot = pgBase + j;
		pgHits ^= 1u << j;
		if(sp + 2 > WIDE_STACK || steps < 0) { ++cnt.errors; done = true; return; }
		if(ngMask > PRIM_BITS) stack.put(sp++, make_uint2(ngBase, ngMask));
		if(pgHits) stack.put(sp++, make_uint2(pgBase, pgHits));
		enter(S, slot, cnt);
	}
	template < class Stack, class C >
	MBD void visit_node(C& cnt, Stack& stack) {
		--steps;
		const uint32_t k = 31u - uint32_t(__clz(int(ngMask))); // highest bit first: nearest octant first
		const uint32_t s = (k ^ oct) & 7u;
		const uint32_t child = ngBase + uint32_t(__popc(ngMask & ((1u << s) - 1u)));
		ngMask ^= 1u << k;
		if(ngMask > PRIM_BITS) {
			if(sp >= WIDE_STACK) { ++cnt.errors; done = true; return; }
			stack.put(sp++, make_uint2(ngBase, ngMask));
		}
		++cnt.nodes;
		const float tmaxBox = t * scale * BOX_SLACK;
		wide_node_test(nodes, child, o, inv, oct, tmaxBox, ngBase, ngMask, pgBase, pgHits);
		exceeded(cnt);
	}
	template < bool ALPHA, class Stack, class C >
	MBD void test_prim(const DScene& S, C& cnt, Stack& stack) {
		const uint32_t j = 31u - uint32_t(__clz(int(pgHits)));
		pgHits ^= 1u << j;
		// all three rows at once (every primitive has them), so a
		// triangle costs one round trip to memory, not two
		const float4* s4 = soup + 3 * size_t(pgBase + j);
		const float4 a = __ldg(s4), b = __ldg(s4 + 1), c = __ldg(s4 + 2);
		const int p = __float_as_int(a.w);
		++cnt.prims;
		float to;
		f2 uv;
		bool hit;
		if(__float_as_int(b.w) == SOUP_TRIANGLE) {
			hit = tri_test(o, int(axes & 3u), int(axes >> 2 & 3u), int(axes >> 4), Sx, Sy, Sz, f4to3(a), f4to3(b), f4to3(c), to, uv) && to > 0.0f;
			if(ALPHA && hit) hit = !alpha_cuts_triangle(alpha_all(S), lod(S), p, uv);
		} else {
			const PrimHit ph = ALPHA ? other_prim_test_alpha(&lod(S), o, d, p, alpha_all(S)) : other_prim_test(&lod(S), o, d, p);
			hit = ph.hit; to = ph.t; uv = ph.uv;
		}
		if(hit) {
			if(any) {
				if(to < t * scale) { occluded = true; done = true; }
			} else {
				const float tw = __fdiv_rn(to, scale);
				// better(): with no hit yet (instance -1) equal distances do not count
				if(tw < t || (tw == t && (inst < stack.hit.x || (inst == stack.hit.x && p < stack.hit.y)))) {
					t = tw; stack.hit = make_int2(inst, p); stack.hitSp = make_float2(uv.x, uv.y);
				}
			}
		}
	}
	template < class Stack >
	MBD void pop(const DScene& S, Stack& stack) {
		if(instSp >= 0 && sp == instSp) {
			if(S.activeInstances == 1) { done = true; return; }
			to_world(S);
		}
		if(sp == 0) { done = true; return; }
		const uint2 e = stack.get(--sp);
		if(e.y > PRIM_BITS) { ngBase = e.x; ngMask = e.y; }
		else { pgBase = e.x; pgHits = e.y; --steps; }
	}

	template < bool ALPHA, class Stack, class C >
	MBD bool step_impl(const DScene& S, C& cnt, Stack& stack) {
		if(done) return true;
		if(instSp < 0 && pgHits) enter_pending(S, cnt, stack);
		if(!done && ngMask > PRIM_BITS) visit_node(cnt, stack);
		if(instSp >= 0) while(pgHits && !done) test_prim<ALPHA>(S, cnt, stack);
		if(!done && ngMask <= PRIM_BITS && !pgHits) pop(S, stack);
		return done;
	}

	// One step of every ray of the warp whose lane passes active, called by
	// all 32 lanes together. Every lane's ray waits to enter an instance, to
	// test primitives or to visit a node; the warp does the one that most of
	// its rays wait for, an instance or a primitive counting more than a node
	// so that their results, which shorten the other visits, do not come late.
	// Rays thus collect until a part runs with many lanes. (One step of all
	// three parts a pass ran the node test at 14 and the others at 2-5 lanes;
	// without the votes the compiler besides threads a ray that entered an
	// instance into a copy of the node test of its own, and the lanes drift
	// apart.) ncu, incoherent bounces: 12.7 of 32 lanes per instruction, 9.0
	// before the votes (icosphere, 540p), and 14.2, 5.6 to 9.9 for steps without
	// and with a meeting of the lanes between the parts (4 096 instances, 360p).
	// Weights: instances 3 and primitives 2 measured 10.3 ms of trace per 720p
	// iteration of the instanced scene, 2 and 2 10.7, 1 and 1 11.7, 2 and 3 10.5,
	// no votes 13.1; the icosphere is within 2 % for all.
	// With at most EACH rays left the warp runs all parts in every pass: few
	// rays gain little from company, and a launch's last rays and a short queue
	// wait for each pass (against votes at any number, 64 x 64 box 0.264 -> 0.246
	// ms an iteration, cut-outs 1.65 -> 1.56, bidirectional 1080p 7.43 -> 7.29).
	// 14, 16 and 22 rays: cut-outs 1.600, 1.594, 1.567 ms, 4 096 instances 12.24,
	// 12.24, 12.30, the other scenes within their spread.
	template < class Stack, class C >
	MBD bool warp_step(const DScene& S, C& cnt, Stack& stack, bool active) {
		constexpr int INSTANCE_WEIGHT = 3, PRIM_WEIGHT = 2, EACH = 16;
		const bool go = active && !done;
		const bool top = go && instSp < 0 && pgHits, prim = go && instSp >= 0 && pgHits, node = go && !pgHits;
		const unsigned bt = __ballot_sync(0xffffffffu, top), bp = __ballot_sync(0xffffffffu, prim);
		const unsigned bn = __ballot_sync(0xffffffffu, node);
		const int wt = INSTANCE_WEIGHT * __popc(bt), wp = PRIM_WEIGHT * __popc(bp), wn = __popc(bn);
		const bool each = __popc(bt | bp | bn) <= EACH;
		const bool doTop = each || (wt > wn && wt >= wp), doPrim = each || (!doTop && wp > wn);
		const bool doNode = each || !(doTop || doPrim);
		if(doTop && top) enter_pending(S, cnt, stack);
		__syncwarp();
		if(doNode && go && !done && !pgHits && ngMask > PRIM_BITS) visit_node(cnt, stack);
		__syncwarp();
		if(doPrim && go && !done && instSp >= 0 && pgHits) {
			do {
				if constexpr(AM == ALPHA_SCENE) {
					if(S.hasAlpha) test_prim<true>(S, cnt, stack);
					else test_prim<false>(S, cnt, stack);
				} else {
					test_prim<AM == ALPHA_ALWAYS>(S, cnt, stack);
				}
			} while(pgHits && !done);
		}
		__syncwarp();
		if(go && !done && ngMask <= PRIM_BITS && !pgHits) pop(S, stack);
		return active && done;
	}

	MBD const DLod& lod(const DScene& S) const { return S.lods[__ldg(S.instanceLod + inst)]; }
};

// Closest hit of a world-space ray whose origin is already offset.
template < int AM = ALPHA_SCENE, class Stack, class C >
MBD HitRec closest_hit_wide(const DScene& S, f3 o, f3 dir, float tmax, C& cnt, Stack& stack) {
	++cnt.rays;
	WideTracerT<AM> t;
	t.init(S, o, dir, tmax, false, stack);
	while(!t.step(S, cnt, stack)) {}
	return t.hit(stack);
}

// Occlusion of a prepared shadow ray (origin offset, unit direction, length tmax).
template < class Stack, class C >
MBD bool occluded_wide(const DScene& S, f3 a, f3 dir, float tmax, C& cnt, Stack& stack) {
	++cnt.rays; ++cnt.shadow;
	WideTracerT<ALPHA_SCENE> t;
	t.init(S, a, dir, tmax, true, stack);
	while(!t.step(S, cnt, stack)) {}
	return t.occluded;
}

} // namespace mb
