// Device memory that comes and goes with scene objects: temporaries of acceleration-structure builds,
// and the storage of meshes and their structures.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace rgl {

// Scene storage (mesh vertices, indices, BLAS nodes), from a pool that keeps up to kKeepBytes for the
// next mesh. The first form is usable on every stream at once, the second once `s` has reached the call's
// point. A freed block is handed out again at once, on any stream, so freeing first waits for all
// StorageReaders.
void* allocateStorage(size_t bytes);
void* allocateStorage(size_t bytes, cudaStream_t s);
void freeStorage(void* p);

// Device work that may read scene storage (a graph's runs, a batch's frames, a server slot's batches). Its
// owner names an event behind the work it has just enqueued; freeStorage waits for the events named last.
// It does not wait for the device as a whole, which is not allowed while any stream of the process is being
// captured, by this library on another thread or by another one, and would end that capture.
class StorageReader
{
public:
	StorageReader();
	StorageReader(const StorageReader&) = delete;
	StorageReader& operator=(const StorageReader&) = delete;
	~StorageReader();
	// `behind` is recorded (not in a capture) after everything enqueued so far; it is the owner's.
	void enqueued(cudaEvent_t behind) { last_.store(behind); }
	// Waits for that event, which the owner is about to destroy.
	void finish();

private:
	friend void freeStorage(void* p);
	void wait();
	std::atomic<cudaEvent_t> last_{nullptr};
};

// Temporaries of one build on one stream: one allocation, given back when the object goes, after the stream.
class BuildScratch
{
public:
	explicit BuildScratch(cudaStream_t s) : stream_(s) {}
	BuildScratch(const BuildScratch&) = delete;
	BuildScratch& operator=(const BuildScratch&) = delete;
	~BuildScratch();

	// Places arrays in the order in which `layout` names them, each on a 256-byte boundary; called once.
	class Carver
	{
	public:
		template<class T>
		void operator()(T*& p, size_t count)
		{
			used_ = (used_ + 255) & ~(size_t) 255;
			p = reinterpret_cast<T*>(base_ + used_);
			used_ += sizeof(T) * (count > 0 ? count : 1);
		}

	private:
		friend class BuildScratch;
		uintptr_t base_ = 0;
		size_t used_ = 0;
	};
	template<class Layout>
	void carve(Layout&& layout)
	{
		Carver size;
		layout(size);
		Carver place;
		place.base_ = allocate(size.used_);
		layout(place);
	}

	// The host has waited for the stream since the last use of the arrays.
	void waited() { waited_ = true; }

private:
	uintptr_t allocate(size_t bytes);
	cudaStream_t stream_;
	void* base_ = nullptr;
	bool waited_ = false;
};

// What a device build tells the host: written by the build's last kernel straight into mapped pinned
// memory and read after the stream has been synchronised, without a copy.
struct BuildReport
{
	int32_t done;               // 1 once written
	int32_t sortFailed;         // the radix sort's look-back did not complete
	uint32_t nodes, leaves;     // wide nodes and leaf records written
	uint32_t sahNodes, sahError; // binary nodes of the SAH topology, an index left its range
	float box[6];               // root box lo xyz, hi xyz
};
class HostReport
{
public:
	HostReport();
	HostReport(const HostReport&) = delete;
	HostReport& operator=(const HostReport&) = delete;
	~HostReport();
	volatile BuildReport* host() const { return host_; }
	BuildReport* device() const { return device_; }

private:
	volatile BuildReport* host_ = nullptr;
	BuildReport* device_ = nullptr;
};

// Returns what the pools and the report list keep beyond what is in use; false when nothing was ever kept.
bool trimBuildMemory();

// Every device allocation of the library that may be large goes through this: memory may be out only
// because of what the pools keep, so the allocation runs once more without it.
template<class Allocate>
cudaError_t trimAndRetry(Allocate&& allocate)
{
	cudaError_t e = allocate();
	if (e == cudaErrorMemoryAllocation && trimBuildMemory()) {
		cudaGetLastError();
		e = allocate();
	}
	return e;
}

} // namespace rgl
