// CPU harness of csrc/build_memory.cpp: the CUDA runtime calls it makes, over a device of a given size whose
// pools keep what is freed into them until they are trimmed, as cudaMemPoolAttrReleaseThreshold has it.
#include <cuda_runtime.h>

#include <cstdlib>
#include <map>
#include <set>
#include <string>

#include "build_memory.hpp"
#include "common.hpp"
#include "kernels.hpp"

namespace {

struct FakePool
{
	size_t reserved = 0, used = 0;
};
struct Block
{
	size_t bytes;
	FakePool* pool;
};
size_t deviceBytes = 0, plainBytes = 0;
std::set<FakePool*> allPools;
std::map<void*, Block> blocks;
std::string calls; // E<event> an event waited for, F a free, D a device synchronisation

bool fits(size_t more)
{
	size_t sum = plainBytes + more;
	for (FakePool* p : allPools) {
		sum += p->reserved;
	}
	return sum <= deviceBytes;
}

void reset(size_t bytes)
{
	deviceBytes = bytes;
	calls.clear();
}

} // namespace

extern "C" {

cudaError_t cudaGetDevice(int* d)
{
	*d = 0;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n)
{
	*n = 1;
	return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceSynchronize()
{
	calls += "D";
	return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
	*s = reinterpret_cast<cudaStream_t>(std::malloc(1));
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
	calls += "E" + std::to_string(reinterpret_cast<uintptr_t>(e));
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
	*p = std::calloc(1, n);
	return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p)
{
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
	*d = h;
	return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*)
{
	auto* p = new FakePool();
	allPools.insert(p);
	*pool = reinterpret_cast<cudaMemPool_t>(p);
	return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t)
{
	auto* p = reinterpret_cast<FakePool*>(pool);
	p->reserved = p->used;
	return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** out, size_t bytes, cudaMemPool_t pool, cudaStream_t)
{
	auto* p = reinterpret_cast<FakePool*>(pool);
	const size_t more = p->used + bytes > p->reserved ? p->used + bytes - p->reserved : 0;
	if (!fits(more)) {
		return cudaErrorMemoryAllocation;
	}
	p->reserved += more;
	p->used += bytes;
	*out = std::malloc(1);
	blocks[*out] = Block{bytes, p};
	return cudaSuccess;
}
cudaError_t cudaMalloc(void** out, size_t bytes)
{
	if (!fits(bytes)) {
		return cudaErrorMemoryAllocation;
	}
	plainBytes += bytes;
	*out = std::malloc(1);
	blocks[*out] = Block{bytes, nullptr};
	return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
	if (p == nullptr) {
		return cudaSuccess;
	}
	const auto it = blocks.find(p);
	if (it == blocks.end()) {
		return cudaErrorInvalidValue;
	}
	(it->second.pool != nullptr ? it->second.pool->used : plainBytes) -= it->second.bytes;
	blocks.erase(it);
	std::free(p);
	calls += "F";
	return cudaSuccess;
}

} // extern "C"

namespace {

constexpr size_t MB = 1000 * 1000;

bool complete(const rgl::TlasBuild& t, int n)
{
	return t.capacity == n && t.levelCapacity == n + 2 && t.nodes != nullptr && t.leaves != nullptr && t.enter != nullptr &&
	       t.boxes != nullptr && t.levelStarts != nullptr && t.nLevels != nullptr &&
	       (n > rgl::kSahSmallMax || (t.smallCapacity == n && t.lo != nullptr && t.hi != nullptr && t.bin != nullptr &&
	                                  t.rangeFirst != nullptr && t.rangeLast != nullptr && t.sortedIds != nullptr));
}

bool throws(rgl::TlasBuild& t, int n)
{
	try {
		rgl::allocateTlas(t, n);
	}
	catch (std::exception&) {
		return true;
	}
	return false;
}

} // namespace

// Each returns 0, or the number of the expectation that does not hold.
extern "C" int kept_memory_serves_other_allocations()
{
	reset(1000 * MB);
	rgl::freeStorage(rgl::allocateStorage(700 * MB));
	if (fits(600 * MB)) {
		return 1; // the pool keeps it
	}
	rgl::TlasBuild t;
	const int n = 2000000; // 236 bytes each
	if (throws(t, n) || !complete(t, n)) {
		return 2;
	}
	rgl::freeTlas(t);
	{
		rgl::BuildScratch scratch(nullptr);
		uint8_t* p = nullptr;
		scratch.carve([&](rgl::BuildScratch::Carver& place) { place(p, 700 * MB); });
	}
	rgl::DeviceBuffer plain;
	if (plain.ensure(600 * MB) == nullptr) {
		return 3;
	}
	plain.release();
	rgl::freeStorage(rgl::allocateStorage(500 * MB));
	rgl::BuildScratch scratch(nullptr);
	uint8_t* p = nullptr;
	scratch.carve([&](rgl::BuildScratch::Carver& place) { place(p, 900 * MB); }); // one pool out of the other's
	return blocks.size() == 1 ? 0 : 4;
}

// `fitting` of the arrays for n instances fit the device; then there is room for all.
extern "C" int a_failed_tlas_allocation_starts_over(int n, int fitting)
{
	const size_t sizes[] = {sizeof(rgl::WideNode), sizeof(rgl::TriRecord), sizeof(rgl::EnterRec), 24, 4};
	size_t room = 0;
	for (int k = 0; k < fitting; ++k) {
		room += sizes[k] * (size_t) n;
	}
	rgl::trimBuildMemory();
	reset(plainBytes + room);
	rgl::TlasBuild t;
	if (!throws(t, n)) {
		return 1;
	}
	reset(1000 * MB);
	if (throws(t, n) || !complete(t, n)) {
		return 2;
	}
	rgl::freeTlas(t);
	return blocks.empty() ? 0 : 3;
}

extern "C" int frees_wait_for_the_readers_alone()
{
	reset(1000 * MB);
	auto event = [](uintptr_t k) { return reinterpret_cast<cudaEvent_t>(k); };
	rgl::StorageReader a, b;
	auto* c = new rgl::StorageReader();
	void* p[4];
	for (auto& q : p) {
		q = rgl::allocateStorage(MB);
	}
	a.enqueued(event(1));
	c->enqueued(event(3));
	rgl::freeStorage(p[0]);
	if (calls != "E1E3F") {
		return 1;
	}
	rgl::freeStorage(p[1]); // both were waited for
	b.enqueued(event(2));
	b.enqueued(event(4)); // behind the one before
	c->enqueued(event(3));
	c->finish();
	delete c;
	rgl::freeStorage(p[2]);
	if (calls != "E1E3FFE3E4F") {
		return 2;
	}
	rgl::freeStorage(nullptr);
	rgl::trimBuildMemory();
	rgl::freeStorage(p[3]);
	return calls == "E1E3FFE3E4FF" ? 0 : 3;
}
