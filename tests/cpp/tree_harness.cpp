// Trees as the library's builders leave them on the device, linked with the library's own objects: read back
// and written out from the root in slot order, so that two trees are the same when the bytes are, whatever
// the order in which their nodes were numbered. The host's trees come from the CPU harness.
#include "bvh_harness.cpp"

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "kernels.hpp"

namespace {

std::vector<uint8_t> written;
std::string failure;

void check(cudaError_t e)
{
	if (e != cudaSuccess) {
		throw std::runtime_error(cudaGetErrorString(e));
	}
}

template<class T>
T* upload(const T* host, size_t count)
{
	T* d = nullptr;
	check(cudaMalloc(&d, sizeof(T) * count));
	check(cudaMemcpy(d, host, sizeof(T) * count, cudaMemcpyHostToDevice));
	return d;
}

template<class T>
std::vector<T> download(const T* device, size_t count)
{
	std::vector<T> h(count);
	check(cudaMemcpy(h.data(), device, sizeof(T) * count, cudaMemcpyDeviceToHost));
	return h;
}

void put(const void* p, size_t bytes) { written.insert(written.end(), static_cast<const uint8_t*>(p), static_cast<const uint8_t*>(p) + bytes); }

// Throws for a reference outside the arrays or more nodes than there are.
void write(const std::vector<WideNode>& nodes, const std::vector<TriRecord>& records, bool triangles)
{
	written.clear();
	std::vector<uint32_t> stack(1, 0u);
	size_t visited = 0;
	while (!stack.empty()) {
		const uint32_t at = stack.back();
		stack.pop_back();
		if (at >= nodes.size() || ++visited > nodes.size()) {
			throw std::runtime_error("a child outside the tree");
		}
		const WideNode& w = nodes[at];
		put(&w.px, 12);
		put(&w.ex, 4);
		put(w.meta, sizeof(w.meta));
		put(w.qlox, 48);
		for (int k = 0; k < kWideArity; ++k) {
			if ((w.imask >> k) & 1u) {
				continue;
			}
			for (int m = 0; m < (w.meta[k] >> 5); ++m) {
				const size_t r = (size_t) w.triBase + (w.meta[k] & 31u) + (size_t) m;
				if (r >= records.size()) {
					throw std::runtime_error("a leaf outside the records");
				}
				const TriRecord& t = records[r];
				put(&t.primId, 4);
				if (triangles) {
					put(&t.v0x, 12);
					put(&t.v1x, 12);
					put(&t.v2x, 12);
				}
			}
		}
		const uint32_t children = (uint32_t) __builtin_popcount(w.imask);
		for (uint32_t c = children; c-- > 0;) {
			stack.push_back(w.childBase + c);
		}
	}
}

template<class Build>
int64_t guarded(Build&& build)
{
	try {
		build();
		return (int64_t) written.size();
	}
	catch (std::exception& e) {
		failure = e.what();
		return -1;
	}
}

void triangleBoxes(const float* v, const int32_t* idx, int n, std::vector<float4>& lo, std::vector<float4>& hi)
{
	for (int t = 0; t < n; ++t) {
		float l[3], h[3];
		for (int a = 0; a < 3; ++a) {
			const float x = v[3 * idx[3 * t] + a], y = v[3 * idx[3 * t + 1] + a], z = v[3 * idx[3 * t + 2] + a];
			l[a] = std::min(x, std::min(y, z));
			h[a] = std::max(x, std::max(y, z));
		}
		lo.push_back(make_float4(l[0], l[1], l[2], 0.0f));
		hi.push_back(make_float4(h[0], h[1], h[2], 0.0f));
	}
}

} // namespace

// Each returns the bytes written, or -1.
extern "C" int64_t device_mesh_tree(const float* v, int nv, const int32_t* idx, int nt, int sah)
{
	return guarded([&] {
		const float* dv = upload(v, 3 * (size_t) nv);
		const int32_t* di = upload(idx, 3 * (size_t) nt);
		BlasBuild b;
		buildBlas(dv, nv, di, nt, b, nullptr, sah != 0);
		write(download(b.nodes, b.nodeCount), download(b.tris, (size_t) nt), true);
		freeBlas(b);
		check(cudaFree(const_cast<float*>(dv)));
		check(cudaFree(const_cast<int32_t*>(di)));
	});
}

extern "C" int64_t host_mesh_tree(const float* v, int, const int32_t* idx, int nt, int sah)
{
	return guarded([&] {
		std::vector<float4> lo, hi;
		triangleBoxes(v, idx, nt, lo, hi);
		const Blas b = sah != 0 ? buildBlasSah(lo, hi, v, idx) : buildWideHost(lo, hi, v, idx, kLeafMaxTris);
		write(b.wide, b.tris, true);
	});
}

// boxes: lo xyz, hi xyz of every instance.
extern "C" int64_t device_instance_tree(const float* boxes, int n)
{
	return guarded([&] {
		std::vector<InstanceRec> inst((size_t) n, InstanceRec{});
		for (int i = 0; i < n; ++i) {
			std::memcpy(&inst[i].lox, boxes + 6 * (size_t) i, 24);
		}
		InstanceRec* d = upload(inst.data(), inst.size());
		TlasBuild t;
		buildTlas(inst.data(), d, n, t, nullptr);
		check(cudaDeviceSynchronize());
		int32_t depths = 0, nodes = 0;
		check(cudaMemcpy(&depths, t.nLevels, sizeof(depths), cudaMemcpyDeviceToHost));
		check(cudaMemcpy(&nodes, t.levelStarts + depths, sizeof(nodes), cudaMemcpyDeviceToHost));
		write(download(t.nodes, (size_t) nodes), download(t.leaves, (size_t) n), false);
		const auto enter = download(t.enter, (size_t) n);
		const auto leaves = download(t.leaves, (size_t) n);
		for (int i = 0; i < n; ++i) {
			if (enter[i].inst != leaves[i].primId) {
				throw std::runtime_error("an enter record of another instance");
			}
		}
		freeTlas(t);
		check(cudaFree(d));
	});
}

extern "C" int64_t host_instance_tree(const float* boxes, int n)
{
	return guarded([&] {
		std::vector<float4> lo, hi;
		std::vector<Box> all;
		for (int i = 0; i < n; ++i) {
			const float* b = boxes + 6 * (size_t) i;
			lo.push_back(make_float4(b[0], b[1], b[2], 0.0f));
			hi.push_back(make_float4(b[3], b[4], b[5], 0.0f));
			all.push_back(Box{b[0], b[1], b[2], b[3], b[4], b[5]});
		}
		const SahTree t = buildBinnedSahTree(all);
		std::vector<WideNode> wide((size_t) n);
		std::vector<TriRecord> leaves((size_t) n);
		uint32_t nodes = 1, records = 0, qa = 1, qb = 0;
		std::vector<int2> a((size_t) n), b((size_t) n);
		a[0] = make_int2(n == 1 ? ~0 : 0, 0);
		CollapseInputs in{t.bin.data(), t.rangeFirst.data(), t.rangeLast.data(), t.sortedIds.data(), lo.data(), hi.data(), nullptr, nullptr, 1};
		while (qa > 0) {
			qb = 0;
			CollapseOutputs o{wide.data(), leaves.data(), &nodes, &records, b.data(), &qb, nullptr};
			for (uint32_t i = 0; i < qa; ++i) {
				collapseItem(a[i].x, (uint32_t) a[i].y, in, o);
			}
			std::swap(a, b);
			qa = qb;
		}
		wide.resize(nodes);
		write(wide, leaves, false);
	});
}

extern "C" void tree_bytes(uint8_t* out) { std::memcpy(out, written.data(), written.size()); }
extern "C" const char* tree_failure() { return failure.c_str(); }
