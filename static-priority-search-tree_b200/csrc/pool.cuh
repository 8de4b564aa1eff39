// Device memory of the library's own objects (trees, engines, scratch): freed blocks are
// kept, up to a bound, for the next object of about their size.
#pragma once

#include <map>
#include <mutex>

#include "common.cuh"

namespace pst {

// Memory on the current device, ready for any stream; fails with PST_ERR_NOMEM, naming
// `what`.
void *pool_alloc(size_t bytes, const char *what);
// Frees p of `device`, which no work queued anywhere may still use.  p may be null.
void pool_release(void *p, int device) noexcept;
// The same for pinned host memory (mapped, as cudaMallocHost gives it).
void *pinned_alloc(size_t bytes, const char *what);
void pinned_release(void *p, int device) noexcept;
// Gives the blocks kept on the current device back.
void pool_trim() noexcept;

// The result of `allocate`, called again without the kept blocks where it first runs out of
// memory: what the library keeps counts as free for its own allocations.
template <typename F>
cudaError_t allocate_or_trim(F &&allocate)
{
	const cudaError_t e = allocate();
	if (e != cudaErrorMemoryAllocation)
		return e;
	cudaGetLastError();
	pool_trim();
	return allocate();
}

// Unique id of the calling thread's current context on device `dev`, made current when
// the thread has none.
unsigned long long current_context_id(int dev);

// Waits for all the work of a device, whichever is current.
void wait_for_device(int device) noexcept;

// The asynchronous passes over one tree that may still be running, one event per
// engine.  The tree and its engines share it, so either may be destroyed first: an
// engine waits for its own pass, a tree for all of them, before its memory is freed.
class InFlight {
  public:
	// Marks the end of the work queued on `s`, of the current device, for `owner` (after its
	// earlier mark, which may lie on another stream).  Work captured into a graph of the
	// caller's may run at any time: from then on the owner waits for the whole device.
	void mark(const void *owner, cudaStream_t s);
	void wait(const void *owner) noexcept;  // and forget it
	void wait_all() noexcept;
	~InFlight();

  private:
	std::mutex mu;
	struct Mark {
		cudaEvent_t event = nullptr;
		bool captured = false;
		int device = 0;
	};
	static void wait_for(const Mark &m) noexcept;
	std::map<const void *, Mark> ev;
};

}  // namespace pst
