// Device form of the wide collapse (bvh_core.hpp collapseItem): eight lanes build one wide node, one
// lane per child, four nodes per warp. The host function is its specification: same children, same
// slots, same bytes; only the numbers of the nodes and of the leaf records follow the atomics.
//
// What bounds it is latency, of instructions as much as of loads: a node takes about 8 us from its task to
// its record, up to seven rounds of opening the largest child one after another, then slots, quantisation
// and packing. One thread per node, with the eight children in local arrays, took 33-36 us per depth; here
// every lane holds one child in registers and the choices are shuffles. The children of a child that may
// be opened are prefetched while the choice is made, the slots are given out from one list that all eight
// lanes hold, and a mesh's leaf records are written once all depths are done. Wide nodes are numbered depth
// by depth, so the queue entry of a node sits at its own index and a depth is a range of indices: no queue
// counter.
#pragma once

#include "bvh_core.hpp"

namespace rgl {
namespace collapsedev {

// Work left for a wide node: the two children of its binary subtree's root (left also alone, for a
// tree of one primitive: right = kNoChild).
struct CollapseTask
{
	int32_t left, right;
};
constexpr int32_t kNoChild = 0x7fffffff;

// Per-depth counters: wide nodes allocated for the next depth (low word) and leaf records written by
// this one (high word), so one 64-bit atomic serves both.
using DepthCounter = unsigned long long;

__device__ __forceinline__ void prefetchL1(const void* p)
{
	asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

struct CollapseTarget
{
	WideNode* wide;
	TriRecord* tris;
	Box* wideBoxes;      // optional: float box of every wide node (TLAS refit)
	CollapseTask* queue; // one entry per wide node
};

// Builds the wide nodes of up to four items, one per group of eight lanes; every lane of the warp takes
// part. `valid` is uniform within a group. Nodes of the next depth start at index `nextNodes`, leaf
// records of this depth at `firstTri`; `limit` bounds both (the primitive count): a warp whose
// allocation passes it, as no proper tree's does, writes nothing, and the counter tells the caller.
template<bool TRIANGLES>
__device__ __forceinline__ void collapseGroups(bool valid, uint32_t wideIdx, CollapseTask task, const CollapseInputs& in,
                                               const CollapseTarget& out, DepthCounter* counter, uint32_t nextNodes, uint32_t firstTri,
                                               uint32_t limit)
{
	constexpr uint32_t kAll = 0xffffffffu;
	const int lane = (int) (threadIdx.x & 31u), sub = lane & 7, group = lane >> 3;

	// This lane's child: reference, box, primitives, first sorted position, children.
	int32_t c = sub == 0 ? task.left : task.right;
	bool has = valid && sub < 2 && c != kNoChild;
	Box b = emptyBox();
	int cnt = 0, first = 0;
	int32_t left = 0, right = 0;
	auto load = [&]() {
		if (c >= 0) {
			const float4* p = reinterpret_cast<const float4*>(in.bin + c);
			const float4 lo = p[0], hi = p[1];
			first = in.rangeFirst[c];
			cnt = in.rangeLast[c] - first + 1;
			b = Box{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
			left = __float_as_int(lo.w);
			right = __float_as_int(hi.w);
		} else {
			first = ~c;
			const int32_t id = in.sortedIds[first];
			const float4 lo = in.triLo[id], hi = in.triHi[id];
			cnt = 1;
			b = Box{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
		}
	};
	if (has) {
		load();
	}
	float area = has ? halfArea(b) : -1.0f;
	// An inner child that may be opened has a key: its area's bits (areas are not negative, their bits are
	// ordered; a NaN is never opened).
	auto openKey = [&]() { return has && c >= 0 && cnt > in.leafMax && area >= 0.0f ? __float_as_uint(area + 0.0f) + 1u : 0u; };
	uint32_t open = openKey();
	// Its children are likely to be held next: asked for while the choice is made.
	auto prefetch = [&]() {
		if (TRIANGLES && open != 0u) {
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				const int32_t k = q == 0 ? left : right;
				if (k >= 0) {
					prefetchL1(in.bin + k);
					prefetchL1(in.rangeFirst + k);
					prefetchL1(in.rangeLast + k);
				} else {
					prefetchL1(in.sortedIds + ~k);
				}
			}
		}
	};
	prefetch();

	// Open the largest inner child until eight children are held or none is left (ties: the lowest).
	int n = valid ? (task.right == kNoChild ? 1 : 2) : kWideArity;
	for (;;) {
		uint32_t best = open;
#pragma unroll
		for (int d = 1; d < 8; d <<= 1) {
			best = max(best, __shfl_xor_sync(kAll, best, d));
		}
		const bool go = n < kWideArity && best != 0u;
		const uint32_t holders = __ballot_sync(kAll, go && open == best) >> (8 * group) & 0xffu;
		if (__ballot_sync(kAll, go) == 0u) {
			break;
		}
		const int bestK = holders != 0u ? (int) lowestBit(holders) : 0;
		const int32_t l = __shfl_sync(kAll, left, bestK, 8), r = __shfl_sync(kAll, right, bestK, 8);
		const bool mine = go && (sub == bestK || sub == n);
		if (mine) {
			c = sub == bestK ? l : r;
			has = true;
			load();
			area = halfArea(b);
			open = openKey();
			prefetch();
		}
		n += go ? 1 : 0;
	}

	// Box of the node.
	Box nb = b;
#pragma unroll
	for (int d = 1; d < 8; d <<= 1) {
		const Box o{__shfl_xor_sync(kAll, nb.lox, d), __shfl_xor_sync(kAll, nb.loy, d), __shfl_xor_sync(kAll, nb.loz, d),
		            __shfl_xor_sync(kAll, nb.hix, d), __shfl_xor_sync(kAll, nb.hiy, d), __shfl_xor_sync(kAll, nb.hiz, d)};
		nb = unite(nb, o);
	}

	// Slots by octant (see collapseItem): children in order of falling area, each to the free slot
	// nearest to its octant in Hamming distance, the lowest among equals.
	const uint32_t key = has ? __float_as_uint(area) : 0u; // areas are not negative: their bits are ordered
	int rank = 0;
#pragma unroll
	for (int d = 1; d < 8; ++d) {
		const uint32_t ok = __shfl_xor_sync(kAll, key, d);
		const bool oh = __shfl_xor_sync(kAll, has ? 1 : 0, d) != 0;
		rank += (oh && (ok > key || (ok == key && (sub ^ d) < sub))) ? 1 : 0;
	}
	const float ncx = 0.5f * (nb.lox + nb.hix), ncy = 0.5f * (nb.loy + nb.hiy), ncz = 0.5f * (nb.loz + nb.hiz);
	const uint32_t oct = ((0.5f * (b.lox + b.hix) >= ncx) ? 1u : 0u) | ((0.5f * (b.loy + b.hiy) >= ncy) ? 2u : 0u) |
	                     ((0.5f * (b.loz + b.hiz) >= ncz) ? 4u : 0u);
	// Octants and lanes by rank, one word each for the whole group: every lane then walks the same list.
	uint32_t octs = has ? oct << (3 * rank) : 0u, lanes = has ? (uint32_t) sub << (3 * rank) : 0u;
#pragma unroll
	for (int d = 1; d < 8; d <<= 1) {
		octs |= __shfl_xor_sync(kAll, octs, d);
		lanes |= __shfl_xor_sync(kAll, lanes, d);
	}
	const int children = __popc(__ballot_sync(kAll, has) >> (8 * group) & 0xffu);
	uint32_t freeSlots = 0xffu;
	int from = -1; // the lane whose child takes this lane's slot
#pragma unroll
	for (int r = 0; r < kWideArity; ++r) {
		const uint32_t o = (octs >> (3 * r)) & 7u;
		// slots at distance 1 and 2 of octant o: byte o of the eight
		const uint32_t near1 = __byte_perm(0x86492916u, 0x68949261u, o), near2 = __byte_perm(0x61929468u, 0x16294986u, o);
		const uint32_t d0 = freeSlots & (1u << o), d1 = freeSlots & near1, d2 = freeSlots & near2;
		const uint32_t pick = d0 != 0u ? d0 : (d1 != 0u ? d1 : (d2 != 0u ? d2 : freeSlots));
		const uint32_t bit = r < children ? pick & (0u - pick) : 0u;
		freeSlots ^= bit;
		from = bit == (1u << sub) ? (int) ((lanes >> (3 * r)) & 7u) : from;
	}

	// From here on a lane is a slot.
	const int src = from < 0 ? 0 : from;
	const bool filled = from >= 0;
	c = __shfl_sync(kAll, c, src, 8);
	cnt = __shfl_sync(kAll, cnt, src, 8);
	first = __shfl_sync(kAll, first, src, 8);
	left = __shfl_sync(kAll, left, src, 8);
	right = __shfl_sync(kAll, right, src, 8);
	b = Box{__shfl_sync(kAll, b.lox, src, 8), __shfl_sync(kAll, b.loy, src, 8), __shfl_sync(kAll, b.loz, src, 8),
	        __shfl_sync(kAll, b.hix, src, 8), __shfl_sync(kAll, b.hiy, src, 8), __shfl_sync(kAll, b.hiz, src, 8)};
	const bool internal = filled && c >= 0 && cnt > in.leafMax;
	const int leafCnt = filled && !internal ? cnt : 0;
	const uint32_t internals = __ballot_sync(kAll, internal);
	const uint32_t imask = (internals >> (8 * group)) & 0xffu;

	// Leaf records before this slot in the warp, and the warp's totals.
	int leafIncl = leafCnt;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const int o = __shfl_up_sync(kAll, leafIncl, d);
		leafIncl += lane >= d ? o : 0;
	}
	const int leafBefore = __shfl_sync(kAll, leafIncl - leafCnt, 0, 8); // before the group's first slot
	const uint32_t warpLeaves = (uint32_t) __shfl_sync(kAll, leafIncl, 31), warpInternals = (uint32_t) __popc(internals);
	DepthCounter base = 0;
	if (lane == 0 && (warpLeaves | warpInternals) != 0u) {
		base = atomicAdd(counter, ((DepthCounter) warpLeaves << 32) | warpInternals);
	}
	base = __shfl_sync(kAll, base, 0);
	const uint32_t nodeBase = nextNodes + (uint32_t) base, leafBase = firstTri + (uint32_t) (base >> 32);
	if (nodeBase + warpInternals > limit || leafBase + warpLeaves > limit) {
		return;
	}
	const uint32_t groupLt = (1u << (8 * group)) - 1u;
	const uint32_t childBase = imask != 0u ? nodeBase + (uint32_t) __popc(internals & groupLt) : 0u;
	const int triOff = leafIncl - leafCnt - leafBefore;
	const uint32_t groupLeaves = (uint32_t) __shfl_sync(kAll, triOff + leafCnt, 7, 8);
	const uint32_t triBase = groupLeaves != 0u ? leafBase + (uint32_t) leafBefore : 0u;

	// Quantisation frame: lane a of the group takes axis a.
	const float lo = sub == 0 ? nb.lox : (sub == 1 ? nb.loy : nb.loz), hi = sub == 0 ? nb.hix : (sub == 1 ? nb.hiy : nb.hiz);
	const uint8_t e = quantExponent(hi - lo);
	const float origin = quantOrigin(lo, e);
	const uint32_t ex = __shfl_sync(kAll, (uint32_t) e, 0, 8), ey = __shfl_sync(kAll, (uint32_t) e, 1, 8),
	               ez = __shfl_sync(kAll, (uint32_t) e, 2, 8);
	const float px = __shfl_sync(kAll, origin, 0, 8), py = __shfl_sync(kAll, origin, 1, 8), pz = __shfl_sync(kAll, origin, 2, 8);
	uint8_t q[6] = {255, 255, 255, 0, 0, 0}; // an empty slot
	if (filled) {
		quantizeAxis(px, exp2Byte((uint8_t) ex), b.lox, b.hix, q[0], q[3]);
		quantizeAxis(py, exp2Byte((uint8_t) ey), b.loy, b.hiy, q[1], q[4]);
		quantizeAxis(pz, exp2Byte((uint8_t) ez), b.loz, b.hiz, q[2], q[5]);
	}
	const uint32_t meta = leafCnt != 0 ? (uint32_t) ((leafCnt << 5) | triOff) : 0u;
	// The slots' bytes packed into words (slots 0..3 and 4..7), then lane j stores 16-byte word j.
	uint32_t wl[7], wh[7];
#pragma unroll
	for (int a = 0; a < 7; ++a) {
		uint32_t v = (a < 6 ? (uint32_t) q[a < 6 ? a : 0] : meta) << (8 * (sub & 3));
		v |= __shfl_xor_sync(kAll, v, 1);
		v |= __shfl_xor_sync(kAll, v, 2);
		const uint32_t o = __shfl_xor_sync(kAll, v, 4);
		wl[a] = sub < 4 ? v : o;
		wh[a] = sub < 4 ? o : v;
	}
	if (valid) {
		uint4 w;
		if (sub == 0) {
			w = make_uint4(__float_as_uint(px), __float_as_uint(py), __float_as_uint(pz), ex | (ey << 8) | (ez << 16) | (imask << 24));
		} else if (sub == 1) {
			w = make_uint4(childBase, triBase, wl[6], wh[6]);
		} else if (sub == 2) {
			w = make_uint4(wl[0], wh[0], wl[1], wh[1]);
		} else if (sub == 3) {
			w = make_uint4(wl[2], wh[2], wl[3], wh[3]);
		} else {
			w = make_uint4(wl[4], wh[4], wl[5], wh[5]);
		}
		if (sub < 5) {
			reinterpret_cast<uint4*>(out.wide + wideIdx)[sub] = w;
		}
		if (sub == 5 && out.wideBoxes != nullptr) {
			out.wideBoxes[wideIdx] = nb;
		}
	}
	if (internal) {
		out.queue[childBase + (uint32_t) __popc(imask & ((1u << sub) - 1u))] = CollapseTask{left, right};
	}
	for (int m = 0; m < leafCnt; ++m) {
		float4* rec = reinterpret_cast<float4*>(out.tris + triBase + (uint32_t) (triOff + m));
		if (TRIANGLES) {
			rec[0].w = __int_as_float(first + m); // the sorted position: writeTriangle turns it into the record
		} else { // TLAS leaf: the instance index only
			rec[0] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(in.sortedIds[first + m]));
			rec[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			rec[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
		}
	}
}

// Leaf record i of a mesh, once every depth is done: all records at once, so the chain from position to
// triangle to indices to vertices is walked once, not once per depth.
__device__ __forceinline__ void writeTriangle(const CollapseInputs& in, TriRecord* tris, uint32_t i)
{
	float4* rec = reinterpret_cast<float4*>(tris + i);
	const int32_t id = in.sortedIds[__float_as_int(rec[0].w)];
	const int32_t* ix = in.indices + 3 * (size_t) id;
	const float* va = in.vertices + 3 * (size_t) ix[0];
	const float* vb = in.vertices + 3 * (size_t) ix[1];
	const float* vc = in.vertices + 3 * (size_t) ix[2];
	rec[0] = make_float4(va[0], va[1], va[2], __int_as_float(id));
	rec[1] = make_float4(vb[0], vb[1], vb[2], 0.0f);
	rec[2] = make_float4(vc[0], vc[1], vc[2], 0.0f);
}

// The root's task.
__device__ __forceinline__ CollapseTask rootTask(const BinNode* bin, int n)
{
	return n == 1 ? CollapseTask{~0, kNoChild} : CollapseTask{bin[0].left, bin[0].right};
}

} // namespace collapsedev
} // namespace rgl
