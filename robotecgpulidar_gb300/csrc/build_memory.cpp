#include "build_memory.hpp"

#include <algorithm>
#include <mutex>
#include <vector>

#include "common.hpp"
#include "kernels.hpp"

namespace rgl {

namespace {

// A pool keeps this much unused memory over a synchronisation. With the default pool, which returns
// everything at every synchronisation, each build mapped its memory anew: an allocation, its release and
// the synchronisation after it cost 86 us against 2 us from a pool that keeps it. The bound holds the
// temporaries of a build of 3 million triangles (about 160 bytes each).
constexpr uint64_t kKeepBytes = 512ull << 20;

// Two pools: scene storage stays in use and would count against what the temporaries may keep. Made at the
// first use and never destroyed: storage of static objects is freed during exit. The allocator serialises
// threads and orders streams itself.
enum Pool { kStorage, kScratch, kPools };
std::mutex poolMutex;
cudaMemPool_t pools[kPools] = {};

cudaMemPool_t makePool()
{
	int device = 0;
	RGL_CHECK_CUDA(cudaGetDevice(&device));
	cudaMemPoolProps props{};
	props.allocType = cudaMemAllocationTypePinned;
	props.handleTypes = cudaMemHandleTypeNone;
	props.location.type = cudaMemLocationTypeDevice;
	props.location.id = device;
	cudaMemPool_t pool = nullptr;
	RGL_CHECK_CUDA(cudaMemPoolCreate(&pool, &props));
	uint64_t keep = kKeepBytes;
	RGL_CHECK_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
	return pool;
}

cudaMemPool_t poolOf(Pool which)
{
	std::lock_guard<std::mutex> g(poolMutex);
	if (pools[which] == nullptr) {
		pools[which] = makePool();
	}
	return pools[which];
}

// Allocations of the first form: a stream of their own, so that they neither wait for nor disturb the legacy
// stream.
cudaStream_t storageStream()
{
	static cudaStream_t stream = [] {
		cudaStream_t s = nullptr;
		RGL_CHECK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
		return s;
	}();
	return stream;
}

// Held while their events are waited for, so that no owner destroys one meanwhile.
std::mutex readerMutex;
std::vector<StorageReader*>& readers()
{
	static auto* all = new std::vector<StorageReader*>(); // never destroyed, as the pools
	return *all;
}

// Report blocks not in use; as many exist as builds ever ran at the same time.
std::mutex reportMutex;
std::vector<BuildReport*>& freeReports()
{
	static auto* reports = new std::vector<BuildReport*>(); // never destroyed, as the pools
	return *reports;
}

void* allocate(Pool which, size_t bytes, cudaStream_t s)
{
	const cudaMemPool_t pool = poolOf(which);
	void* p = nullptr;
	RGL_CHECK_CUDA(trimAndRetry([&] { return cudaMallocFromPoolAsync(&p, bytes, pool, s); }));
	return p;
}

// A plain allocation of `count` elements.
template<class T>
void allocateArray(T*& p, size_t count)
{
	RGL_CHECK_CUDA(trimAndRetry([&] { return cudaMalloc(reinterpret_cast<void**>(&p), sizeof(T) * count); }));
}

template<class T>
void freeArray(T*& p)
{
	cudaFree(p);
	p = nullptr;
}

void freeTlasScratch(TlasBuild& t)
{
	t.smallCapacity = 0;
	freeArray(t.lo);
	freeArray(t.hi);
	freeArray(t.bin);
	freeArray(t.rangeFirst);
	freeArray(t.rangeLast);
	freeArray(t.sortedIds);
}

} // namespace

StorageReader::StorageReader()
{
	std::lock_guard<std::mutex> g(readerMutex);
	readers().push_back(this);
}

StorageReader::~StorageReader()
{
	std::lock_guard<std::mutex> g(readerMutex);
	readers().erase(std::find(readers().begin(), readers().end(), this));
}

void StorageReader::finish()
{
	std::lock_guard<std::mutex> g(readerMutex);
	wait();
}

void StorageReader::wait()
{
	if (cudaEvent_t e = last_.exchange(nullptr)) {
		cudaEventSynchronize(e);
	}
}

void* allocateStorage(size_t bytes)
{
	void* p = allocate(kStorage, bytes, storageStream());
	RGL_CHECK_CUDA(cudaStreamSynchronize(storageStream()));
	return p;
}

void* allocateStorage(size_t bytes, cudaStream_t s) { return allocate(kStorage, bytes, s); }

void freeStorage(void* p)
{
	if (p == nullptr) {
		return;
	}
	{
		std::lock_guard<std::mutex> g(readerMutex);
		for (StorageReader* r : readers()) {
			r->wait();
		}
	}
	cudaFree(p); // of a pool's block: waits for nothing
}

uintptr_t BuildScratch::allocate(size_t bytes)
{
	base_ = rgl::allocate(kScratch, bytes, stream_);
	return reinterpret_cast<uintptr_t>(base_);
}

BuildScratch::~BuildScratch()
{
	if (base_ != nullptr) {
		// Freed for good, so that trimBuildMemory finds it free: one that is queued on a stream counts as in
		// use until the host has waited for it.
		if (!waited_) {
			cudaStreamSynchronize(stream_);
		}
		cudaFree(base_);
	}
}

HostReport::HostReport()
{
	BuildReport* report = nullptr;
	{
		std::lock_guard<std::mutex> g(reportMutex);
		if (!freeReports().empty()) {
			report = freeReports().back();
			freeReports().pop_back();
		}
	}
	if (report == nullptr) {
		void* p = nullptr;
		RGL_CHECK_CUDA(cudaHostAlloc(&p, sizeof(BuildReport), cudaHostAllocMapped | cudaHostAllocPortable));
		report = static_cast<BuildReport*>(p);
	}
	*report = BuildReport{};
	host_ = report;
	void* d = nullptr;
	RGL_CHECK_CUDA(cudaHostGetDevicePointer(&d, report, 0));
	device_ = static_cast<BuildReport*>(d);
}

HostReport::~HostReport()
{
	std::lock_guard<std::mutex> g(reportMutex);
	freeReports().push_back(const_cast<BuildReport*>(host_));
}

bool trimBuildMemory()
{
	bool made = false;
	{
		std::lock_guard<std::mutex> g(poolMutex);
		for (cudaMemPool_t p : pools) {
			if (p != nullptr) {
				cudaMemPoolTrimTo(p, 0);
				made = true;
			}
		}
	}
	std::lock_guard<std::mutex> g(reportMutex);
	for (BuildReport* r : freeReports()) {
		cudaFreeHost(r);
	}
	freeReports().clear();
	return made;
}

// The capacities are set once all arrays are there: after an allocation that failed, the next build of that
// size starts over instead of using the ones that are missing.
void allocateTlas(TlasBuild& t, int n)
{
	if (n > t.capacity) {
		freeTlas(t);
		allocateArray(t.nodes, (size_t) n);
		allocateArray(t.leaves, (size_t) n);
		allocateArray(t.enter, (size_t) n);
		allocateArray(t.boxes, 6 * (size_t) n);
		allocateArray(t.levelStarts, (size_t) n + 2);
		allocateArray(t.nLevels, 1);
		t.levelCapacity = n + 2;
		t.capacity = n;
	}
	// The one-block rebuild's scratch has a size of its own: a scene that shrinks from above
	// kSahSmallMax instances keeps its node storage but has no scratch yet.
	if (n <= kSahSmallMax && n > t.smallCapacity) {
		freeTlasScratch(t);
		allocateArray(t.lo, (size_t) n);
		allocateArray(t.hi, (size_t) n);
		allocateArray(t.bin, (size_t) n);
		allocateArray(t.rangeFirst, (size_t) n);
		allocateArray(t.rangeLast, (size_t) n);
		allocateArray(t.sortedIds, (size_t) n);
		t.smallCapacity = n;
	}
}

void freeTlas(TlasBuild& t)
{
	freeTlasScratch(t);
	freeArray(t.nodes);
	freeArray(t.leaves);
	freeArray(t.enter);
	freeArray(t.boxes);
	freeArray(t.levelStarts);
	freeArray(t.nLevels);
	t = TlasBuild{};
}

} // namespace rgl
