// The block pool under contexts that alternate and end, with the few runtime calls it makes
// replaced by host memory that keeps book: a block goes back to the context it came from, and
// is neither lost nor freed under another.
#include <cstdio>
#include <map>
#include <string>

#include "pool.cuh"

// (fake_runtime.cpp)
extern unsigned long long g_ctx;
extern std::map<void *, unsigned long long> g_blocks;  // every block that the runtime has handed out
extern int g_bad;                                      // blocks freed twice or under another context

namespace pst {
void fail(pst_status st, const std::string &msg) { throw Error{st, msg}; }
void check_cuda(cudaError_t e, const char *what)
{
	if (e != cudaSuccess)
		fail(PST_ERR_CUDA, what);
}
}  // namespace pst

#define EXPECT(x)                                              \
	do {                                                       \
		if (!(x))                                              \
			return printf("line %d: %s\n", __LINE__, #x), 1;   \
	} while (0)

int main()
{
	using namespace pst;
	// objects of two contexts, made and given up in turn
	for (int i = 0; i < 50; i++) {
		g_ctx = 1;
		void *a = pool_alloc(1000, "a"), *ha = pinned_alloc(500, "ha");
		g_ctx = 2;
		void *b = pool_alloc(1000, "b"), *hb = pinned_alloc(500, "hb");
		EXPECT(g_blocks.at(a) == 1 && g_blocks.at(ha) == 1 && g_blocks.at(b) == 2 && g_blocks.at(hb) == 2);
		g_ctx = 1;
		pool_release(a, 0);
		pinned_release(ha, 0);
		g_ctx = 2;
		pool_release(b, 0);
		pinned_release(hb, 0);
		EXPECT(g_blocks.size() == 4 && g_bad == 0);
	}
	// given up while the other context is current: it stays the first one's
	g_ctx = 1;
	void *a = pool_alloc(1000, "a");
	void *big = pool_alloc(size_t(3) << 20, "big");  // more than a context may keep
	g_ctx = 2;
	pool_release(a, 0);
	pool_release(big, 0);
	void *b = pool_alloc(1000, "b");
	EXPECT(a != b && g_blocks.at(b) == 2);
	pool_release(b, 0);
	g_ctx = 1;
	EXPECT(g_blocks.count(big) == 1);
	EXPECT(pool_alloc(1000, "a") == a);
	EXPECT(g_blocks.count(big) == 0);  // back over the bound, so back to the device
	pool_release(a, 0);
	// a context that ended: its blocks are gone with it and nobody frees them
	g_ctx = 3;
	void *c = pool_alloc(2000, "c");
	g_ctx = 4;  // cudaDeviceReset, and a new primary context
	void *d = pool_alloc(2000, "d");
	pool_release(c, 0);  // an object that outlived its context
	EXPECT(pool_alloc(2000, "e") != c);
	pool_release(d, 0);
	pool_trim();
	EXPECT(g_bad == 0 && g_blocks.count(c) == 1);
	// everything kept can be given back
	for (unsigned long long x : {1, 2}) {
		g_ctx = x;
		pool_trim();
	}
	std::map<unsigned long long, int> left;
	for (auto &x : g_blocks)
		left[x.second]++;
	EXPECT(g_bad == 0 && left[1] == 0 && left[2] == 0 && left[4] == 1);
	printf("ok\n");
	return 0;
}
