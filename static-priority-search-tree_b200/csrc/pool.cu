// The block pool of pool.cuh.
#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include <cuda.h>

#include "pool.cuh"

namespace pst {

namespace {

// Freed memory kept per device: 1/KEEP_SHARE of its memory (5.6 of 179 GiB), enough for
// the build of a 2^26-point tree beside the tree that it replaces (3.6 GiB); of a larger
// one, as of 2^28 points, the scratch is mapped and unmapped at each build.  cudaMalloc
// and cudaFree map and unmap pages, and cudaFree waits for the whole device: 19 and 20 of
// them took 2.1 of the 4.4 ms of an isosurface pass over a 384^3 volume, and 1.2 of the
// 1.9 ms of a build of 2^21 points.  A stream-ordered CUDA pool did as well while the
// blocks stayed in it, but grows by about 8 ms a GB (cudaMalloc: 0.2 ms), which made the
// build of a 2^28-point tree 117 ms slower.
constexpr size_t KEEP_SHARE = 32;
// Pinned host memory kept per device, for the control block and the staged queries of
// engines: cudaMallocHost and cudaFreeHost took 3.1 and 0.6 ms a call in a process that
// holds little pinned memory, more than the rest of a 384^3 isosurface pass.
constexpr size_t KEEP_PINNED = size_t(8) << 20;
// Requests are rounded up to an eighth of their power of two, so that objects of about
// one size share blocks, and from BIG on to whole pages only: a tree that just fits the
// device has to go on fitting it.
constexpr size_t BIG = size_t(64) << 20, PAGE = size_t(2) << 20;

size_t block_bytes(size_t bytes)
{
	if (bytes >= BIG)
		return (bytes + PAGE - 1) / PAGE * PAGE;
	size_t step = 512;
	while (step * 16 <= bytes)
		step *= 2;
	return (std::max<size_t>(bytes, 1) + step - 1) / step * step;
}

struct Block {
	void *ptr;
	size_t bytes;
};

// One context's blocks.
struct Pool {
	const bool pinned;
	size_t keep = 0, kept = 0;
	std::vector<Block> idle;                    // oldest first
	std::unordered_map<void *, size_t> live;

	explicit Pool(bool host) : pinned(host)
	{
		size_t fr = 0, total = 0;
		check_cuda(cudaMemGetInfo(&fr, &total), "cudaMemGetInfo");
		keep = pinned ? KEEP_PINNED : total / KEEP_SHARE;
	}
	cudaError_t get(void **ptr, size_t bytes) const { return pinned ? cudaMallocHost(ptr, bytes) : cudaMalloc(ptr, bytes); }
	void give_back(const std::vector<Block> &blocks) const noexcept
	{
		for (const Block &b : blocks)
			if ((pinned ? cudaFreeHost(b.ptr) : cudaFree(b.ptr)) != cudaSuccess)
				cudaGetLastError();
	}

	// The smallest idle block that holds `bytes` and is at most an eighth larger.
	void *take(size_t bytes)
	{
		size_t best = idle.size();
		for (size_t i = 0; i < idle.size(); i++)
			if (idle[i].bytes >= bytes && idle[i].bytes <= bytes + bytes / 8 &&
			    (best == idle.size() || idle[i].bytes < idle[best].bytes))
				best = i;
		if (best == idle.size())
			return nullptr;
		const Block b = idle[best];
		idle.erase(idle.begin() + (ptrdiff_t) best);
		kept -= b.bytes;
		live[b.ptr] = b.bytes;
		return b.ptr;
	}

	// Takes the oldest blocks out until at most `most` bytes are kept.
	std::vector<Block> shrink(size_t most)
	{
		std::vector<Block> out;
		while (kept > most) {
			out.push_back(idle.front());
			kept -= idle.front().bytes;
			idle.erase(idle.begin());
		}
		return out;
	}
};

// The pools of one device, by the id of their context.  A block belongs to the context it
// was made in, and programs may switch between several; cudaDeviceReset ends one, whose
// pool is then never entered again (ids are not used twice).
struct Pools {
	const bool pinned;
	std::mutex mu;
	std::map<unsigned long long, Pool> of;

	explicit Pools(bool host) : pinned(host) {}
	// (with mu held)
	Pool &enter(unsigned long long ctx)
	{
		const auto it = of.find(ctx);
		return it != of.end() ? it->second : of.emplace(ctx, pinned).first->second;
	}
};
struct DevicePools {
	Pools mem{false}, pinned{true};
};
DevicePools g_pools[64];

DevicePools &pools_of(int dev)
{
	if (dev < 0 || dev >= 64)
		fail(PST_ERR_CUDA, "device index out of range");
	return g_pools[dev];
}

int current_device()
{
	int dev = 0;
	check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
	return dev;
}

}  // namespace

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

// (The library does not link the driver library itself: the two driver calls come from
// the runtime's entry points.)
unsigned long long current_context_id(int dev)
{
	static CtxGetCurrentFn get_cur = nullptr;
	static CtxGetIdFn get_id = nullptr;
	static std::once_flag once;
	std::call_once(once, [] {
		void *p = nullptr;
		cudaDriverEntryPointQueryResult q{};
		if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
		    q == cudaDriverEntryPointSuccess)
			get_cur = reinterpret_cast<CtxGetCurrentFn>(p);
		p = nullptr;
		if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
		    q == cudaDriverEntryPointSuccess)
			get_id = reinterpret_cast<CtxGetIdFn>(p);
		cudaGetLastError();
	});
	if (!get_cur || !get_id)
		fail(PST_ERR_CUDA, "driver entry points cuCtxGetCurrent / cuCtxGetId are unavailable");
	CUcontext c = nullptr;
	if (get_cur(&c) == CUDA_SUCCESS && !c) {
		// a thread that has made no other CUDA call: cudaSetDevice makes the device's
		// primary context current on it
		check_cuda(cudaSetDevice(dev), "cudaSetDevice");
		get_cur(&c);
	}
	unsigned long long id = 0;
	if (!c || get_id(c, &id) != CUDA_SUCCESS)
		fail(PST_ERR_CUDA, "no current CUDA context");
	return id;
}

namespace {

void *alloc_in(Pools &pools, int dev, size_t bytes, const char *what)
{
	const unsigned long long ctx = current_context_id(dev);
	const size_t want = block_bytes(bytes);
	Pool *p = nullptr;
	void *ptr = nullptr;
	std::vector<Block> out;
	{
		std::lock_guard<std::mutex> lk(pools.mu);
		p = &pools.enter(ctx);  // (a map's elements stay where they are)
		ptr = p->take(want);
		out = p->shrink(p->keep);  // (what was released under another context)
	}
	p->give_back(out);
	if (ptr)
		return ptr;
	const cudaError_t e = allocate_or_trim([&] { return p->get(&ptr, want); });
	if (e == cudaErrorMemoryAllocation) {
		cudaGetLastError();
		fail(PST_ERR_NOMEM, std::string(what) + " allocation of " + std::to_string(bytes) + " B failed");
	}
	check_cuda(e, "cudaMalloc");
	std::lock_guard<std::mutex> lk(pools.mu);
	p->live[ptr] = want;
	return ptr;
}

void release_in(Pools &pools, int dev, void *ptr)
{
	std::vector<Block> out;
	Pool *p = nullptr;
	{
		const unsigned long long ctx = current_context_id(dev);
		std::lock_guard<std::mutex> lk(pools.mu);
		Pool &here = pools.enter(ctx);
		p = &here;
		if (here.live.find(ptr) == here.live.end())
			for (auto &x : pools.of)
				if (x.second.live.find(ptr) != x.second.live.end())
					p = &x.second;
		const auto it = p->live.find(ptr);
		if (it == p->live.end())
			return;
		const Block b{ptr, it->second};
		p->live.erase(it);
		if (p == &here && b.bytes > p->keep) {
			out.push_back(b);
		} else {
			p->idle.push_back(b);
			p->kept += b.bytes;
			// another context's blocks are given back from there (it may be gone, too)
			if (p == &here)
				out = p->shrink(p->keep);
		}
	}
	p->give_back(out);
}

void trim(Pools &pools, int dev)
{
	std::vector<Block> out;
	Pool *p = nullptr;
	{
		const unsigned long long ctx = current_context_id(dev);
		std::lock_guard<std::mutex> lk(pools.mu);
		p = &pools.enter(ctx);
		out = p->shrink(0);
	}
	p->give_back(out);
}

void release_on(bool pinned, void *ptr, int device) noexcept
{
	if (!ptr)
		return;
	try {
		const int cur = current_device();
		if (cur != device)
			check_cuda(cudaSetDevice(device), "cudaSetDevice");
		release_in(pinned ? pools_of(device).pinned : pools_of(device).mem, device, ptr);
		if (cur != device)
			cudaSetDevice(cur);
	} catch (...) {
		cudaGetLastError();
	}
}

}  // namespace

void *pool_alloc(size_t bytes, const char *what)
{
	const int dev = current_device();
	return alloc_in(pools_of(dev).mem, dev, bytes, what);
}

void *pinned_alloc(size_t bytes, const char *what)
{
	const int dev = current_device();
	return alloc_in(pools_of(dev).pinned, dev, bytes, what);
}

void pool_release(void *ptr, int device) noexcept { release_on(false, ptr, device); }
void pinned_release(void *ptr, int device) noexcept { release_on(true, ptr, device); }

void pool_trim() noexcept
{
	try {
		const int dev = current_device();
		trim(pools_of(dev).mem, dev);
		trim(pools_of(dev).pinned, dev);
	} catch (...) {
		cudaGetLastError();
	}
}

void InFlight::mark(const void *owner, cudaStream_t s)
{
	std::lock_guard<std::mutex> lk(mu);
	Mark &m = ev[owner];
	cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
	check_cuda(cudaStreamIsCapturing(s, &st), "cudaStreamIsCapturing");
	if (st != cudaStreamCaptureStatusNone) {
		check_cuda(cudaGetDevice(&m.device), "cudaGetDevice");
		m.captured = true;  // an earlier mark's event does not belong in the caller's graph
		return;
	}
	if (!m.event)
		check_cuda(cudaEventCreateWithFlags(&m.event, cudaEventDisableTiming), "cudaEventCreate");
	else
		check_cuda(cudaStreamWaitEvent(s, m.event, 0), "cudaStreamWaitEvent");
	check_cuda(cudaEventRecord(m.event, s), "cudaEventRecord");
}

void wait_for_device(int device) noexcept
{
	int cur = 0;
	cudaGetDevice(&cur);
	if (cur != device)
		cudaSetDevice(device);
	cudaDeviceSynchronize();
	if (cur != device)
		cudaSetDevice(cur);
	cudaGetLastError();
}

void InFlight::wait_for(const Mark &m) noexcept
{
	if (m.captured)
		wait_for_device(m.device);
	else if (m.event)
		cudaEventSynchronize(m.event);
	cudaGetLastError();
}

void InFlight::wait(const void *owner) noexcept
{
	std::lock_guard<std::mutex> lk(mu);
	auto it = ev.find(owner);
	if (it == ev.end())
		return;
	wait_for(it->second);
	if (it->second.event)
		cudaEventDestroy(it->second.event);
	cudaGetLastError();
	ev.erase(it);
}

void InFlight::wait_all() noexcept
{
	std::lock_guard<std::mutex> lk(mu);
	for (auto &x : ev)
		wait_for(x.second);
}

InFlight::~InFlight()
{
	for (auto &x : ev)
		if (x.second.event)
			cudaEventDestroy(x.second.event);
	cudaGetLastError();
}

}  // namespace pst
