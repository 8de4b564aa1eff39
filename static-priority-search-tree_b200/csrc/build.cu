// Construction of the static priority search tree on the GPU.
//
// The tree is the one the reference's StaticPSTCPUIter builds, node for node
// (pst/static-pst-cpu-iter.tpp:18-177, pst/static-pst-cpu-iter-populate-tree.tpp:11-114,
// constructNode at pst/static-pst-cpu-iter.tpp:491-598):
//   - a node of c points holds the point that is largest in the dim2 order
//     (value, then id, then input index: helpers/point-struct.h:62-92, :154-188);
//   - its median is the dim1 value of the floor(c/2)-th of the remaining points in
//     dim1 order, and those floor(c/2) points form the left subtree;
//   - the rest form the right subtree.
// The reference finds each node's point with a binary search, then shifts and
// partitions index arrays one node at a time (pst/static-pst-gpu.tu:678-806; one
// thread per node, one block, dynamic parallelism).  This build works level by level
// instead:
//   1. every point gets a tiebreak rank tb (its place in (id, input index) order) and
//      a 64-bit dim2 key whose order is the dim2 order: (dim2 key << 32 | tb + 1) for
//      4-byte values, (dim2 rank << 32 | tb + 1) for doubles (one extra sort finds
//      the ranks).  One radix sort by dim1 key carries these keys along, so position
//      i of the sorted arrays is the i-th point in dim1 order;
//   2. for the wide top levels, one kernel a level: a warp (or, while nodes are few, a
//      CTA) per node finds the largest dim2 key of its positions from a maximum per
//      512-position tile and per 32 tiles and the positions of the tiles that its bounds
//      cut, takes it out (its key becomes 0), brings the maxima up to date and places
//      the median;
//   3. once every node of a level holds at most ST_CAP points, one CTA per node
//      builds the whole remaining subtree in shared memory.
#include <algorithm>
#include <limits>
#include <type_traits>
#include <vector>

#include "scan_sort.cuh"
#include "tree.cuh"

namespace pst {

size_t value_size(pst_dtype dt) { return dt == PST_F64 ? 8 : 4; }

size_t point_size(pst_dtype dt, pst_idtype it)
{
	if (dt != PST_F32 && dt != PST_F64 && dt != PST_I32)
		return 0;
	if (it == PST_ID_NONE)
		return 2 * value_size(dt);
	if (it == PST_ID_U32)
		return dt == PST_F64 ? 24 : 12;
	return 0;
}

namespace {

constexpr size_t ALIGN = 256;
inline size_t align_up(size_t v) { return (v + ALIGN - 1) / ALIGN * ALIGN; }

struct TreeLayout {
	size_t off_dim1, off_dim2, off_med, off_id, off_occ, total;
};

TreeLayout tree_layout(pst_dtype dt, pst_idtype it, uint64_t n)
{
	TreeLayout L{};
	if (n == 0)
		return L;
	const uint32_t D = tree_levels(n);
	const uint64_t S = 1ull << D;
	const size_t vs = value_size(dt);
	size_t o = 0;
	L.off_dim1 = o;
	o = align_up(o + S * vs);
	L.off_dim2 = o;
	o = align_up(o + S * vs);
	L.off_med = o;
	o = align_up(o + (S / 2) * vs);
	L.off_id = o;
	if (it == PST_ID_U32)
		o = align_up(o + S * 4);
	L.off_occ = o;
	o = align_up(o + std::max<uint64_t>(S / 32, 1) * 4);
	L.total = o;
	return L;
}

// Subtree builder capacity: nodes of at most ST_CAP points are finished by one CTA.
constexpr uint32_t ST_CAP = 512;
constexpr int ST_THREADS = 128;
// Arg-max tiles, and the tiles a second maximum covers.
constexpr uint32_t TM_TILE = 512, TM_SUPER = 32;
constexpr int LV_THREADS = 256;

// First level whose largest node holds at most ST_CAP points.  Counts within a
// level take at most two consecutive values (m, m+1).
uint32_t subtree_level(uint64_t n)
{
	uint64_t hi = n;
	uint32_t d = 0;
	while (hi > ST_CAP) {
		hi = hi / 2;  // largest child of the largest node
		d++;
	}
	return d;
}

// Sorted arrays, position i = i-th point in dim1 order:
//   k1s[i]  dim1 key, c2s[i] 64-bit dim2 key (low 32 bits = tb + 1, so never 0) until
//   the point is stored in a node, then 0.
template <typename T, bool HAS_ID>
struct BuildCtx {
	using K = typename KeyOf<T>::K;
	const Point<T, HAS_ID> *pts;
	const uint32_t *P;  // tiebreak rank -> input index (null: identity)
	const K *k1s;
	uint64_t *c2s;
	uint64_t *tmax;     // per TM_TILE tile: max c2s
	uint64_t *smax;     // per TM_SUPER tiles: max c2s
	T *dim1;
	T *dim2;
	T *med;
	uint32_t *id;
	uint32_t *occ;
	uint32_t *top_pos;  // heap position -> dim1-sorted position of its point (levels < L0)
	uint32_t *err;
	uint64_t n;
	uint32_t D;
	// Points are rebuilt from their sorted keys instead of gathered from the input:
	// set for 4-byte values when no value is -0.0 (the only value the keys do not
	// keep: it shares +0.0's key) and the ids, if any, equal the input indices (so
	// the id is the tiebreak rank the dim2 key carries).
	bool recon;

	__device__ __forceinline__ Point<T, HAS_ID> point_of_tb(uint32_t tb) const { return pts[P ? P[tb] : tb]; }
	__device__ __forceinline__ static uint32_t tb_of(uint64_t key2) { return (uint32_t) key2 - 1u; }
	// The point of dim1 key k1 and 64-bit dim2 key c2 (recon only).
	__device__ __forceinline__ static Point<T, HAS_ID> point_from_keys(K k1, uint64_t c2)
	{
		Point<T, HAS_ID> p;
		p.dim1 = KeyOf<T>::value(k1);
		p.dim2 = KeyOf<T>::value((K) (c2 >> 32));
		if constexpr (HAS_ID)
			p.id = tb_of(c2);
		return p;
	}
	// The point at position pos, whose dim2 key is (or was) c2.
	__device__ __forceinline__ Point<T, HAS_ID> point_of(uint32_t pos, uint64_t c2) const
	{
		if constexpr (sizeof(K) == 4) {
			if (recon)
				return point_from_keys(k1s[pos], c2);
		}
		return point_of_tb(tb_of(c2));
	}
	__device__ __forceinline__ void write_node(uint32_t h, const Point<T, HAS_ID> &p) const
	{
		dim1[h] = p.dim1;
		dim2[h] = p.dim2;
		if constexpr (HAS_ID)
			id[h] = p.id;
	}
};

template <typename K>
__device__ __forceinline__ void atomic_min_key(K *p, K v)
{
	if constexpr (sizeof(K) == 4)
		atomicMin(reinterpret_cast<unsigned int *>(p), (unsigned int) v);
	else
		atomicMin(reinterpret_cast<unsigned long long *>(p), (unsigned long long) v);
}

template <typename K>
__device__ __forceinline__ void atomic_max_key(K *p, K v)
{
	if constexpr (sizeof(K) == 4)
		atomicMax(reinterpret_cast<unsigned int *>(p), (unsigned int) v);
	else
		atomicMax(reinterpret_cast<unsigned long long *>(p), (unsigned long long) v);
}

// Block-wide min and max of (lo, hi), folded into range[0] / range[1] with atomics.
template <typename K>
__device__ void block_range_fold(K lo, K hi, K *range)
{
	__shared__ K s_lo[32], s_hi[32];
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		const K a = __shfl_xor_sync(0xFFFFFFFFu, lo, o), b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
		lo = a < lo ? a : lo;
		hi = b > hi ? b : hi;
	}
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
	if (lane == 0) {
		s_lo[warp] = lo;
		s_hi[warp] = hi;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int w = 1; w < nw; w++) {
			lo = s_lo[w] < lo ? s_lo[w] : lo;
			hi = s_hi[w] > hi ? s_hi[w] : hi;
		}
		atomic_min_key<K>(&range[0], lo);
		atomic_max_key<K>(&range[1], hi);
	}
}

// ---------------------------------------------------------------------------
// Preparation kernels.

// What the key pass finds, in the construction's flag words.
template <typename K>
struct BuildFlags {
	uint32_t id_order;     // bits of k_prep_keys' idflag
	uint32_t err;          // error bits
	uint32_t id_range[2];  // [min, max]
	uint32_t negzero;      // -0.0 seen
	uint32_t unused[11];
	K range[4];  // [k1 min, k1 max, k2 min, k2 max]
};
static_assert(sizeof(BuildFlags<uint64_t>) <= 256 && offsetof(BuildFlags<uint64_t>, range) == 64, "flag words");

// The flag words as k_prep_keys wants them, and the bounds of the root.  (A copy of each
// from the host, and one back for each group of flags: 349 us for a build of 2^21
// metacells, with the search index made behind another wait; now 314.)
template <typename K>
__global__ void k_build_init(uint32_t *flag, uint32_t *bounds, uint32_t n)
{
	BuildFlags<K> *f = reinterpret_cast<BuildFlags<K> *>(flag);
	if (threadIdx.x < 16)
		flag[threadIdx.x] = threadIdx.x == 2 ? 0xFFFFFFFFu : 0u;
	if (threadIdx.x < 4)
		f->range[threadIdx.x] = threadIdx.x & 1 ? K(0) : ~K(0);
	if (threadIdx.x < 2)
		bounds[threadIdx.x] = threadIdx.x ? n : 0u;
}

template <typename T, bool HAS_ID>
__global__ void k_id_keys(const Point<T, HAS_ID> *pts, uint64_t n, uint32_t *keys)
{
	if constexpr (HAS_ID) {
		for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
			keys[i] = pts[i].id;
	}
}

// Copies of the digit histogram a block of k_prep_keys keeps in shared memory (a
// quarter of its warps on each), so that keys sharing a digit meet on fewer counters.
constexpr int PK_HIST_COPIES = 4;
constexpr int PK_THREADS = 512, PK_CTAS = 2, PK_ITEMS = 4;  // points in flight per thread

// Keys in tiebreak-rank order r (input index P[r]): k1[r] = dim1 key and either the
// final 64-bit dim2 key (4-byte values) or the raw dim2 key k2[r] (doubles).
// range = [min k1, max k1, min k2, max k2]; *negzero |= 1 when a value is -0.0 (the
// one value its key does not keep).
// SCAN_IDS (P null, points with ids): the same pass checks the ids, idflag |= 1 when
// they decrease somewhere and |= 2 when some id differs from its input index,
// id_range = [min id, max id].  hist (non-null): the pass also counts the 8-bit
// digits of the dim1 keys, hist[d * 256 + v] += keys whose digit d is v, for every
// digit of the key (the radix sort's histogram, which the order of the keys does
// not change); dynamic shared memory PK_HIST_COPIES * sizeof(K) * 256 words.
// Bound by memory at 2^26 points (1.61 GB: 246 us), below some 10 M by the atomics that
// end a CTA: up to 256 counters per digit and the ranges, all CTAs' on the same words.
// So two CTAs of 512 threads to an SM and no more, which keep four points a thread in
// flight, in place of up to 16 of 256 with one: 2^21 metacells 31.6 -> 13.5 us, 5 M
// doubles 56.9 -> 35.2, 2^26 points 305 -> 282 (eight points 18, 61, 379; two 13.7, 37,
// 322).
template <typename T, bool HAS_ID, bool SCAN_IDS>
__global__ void __launch_bounds__(PK_THREADS, PK_CTAS) k_prep_keys(const Point<T, HAS_ID> *pts, const uint32_t *P, uint64_t n,
                            typename KeyOf<T>::K *k1, uint64_t *c2, typename KeyOf<T>::K *k2,
                            typename KeyOf<T>::K *range, uint32_t *negzero, uint32_t *idflag,
                            uint32_t *id_range, uint32_t *hist)
{
	using K = typename KeyOf<T>::K;
	constexpr int ND = (int) sizeof(K);  // 8-bit digits of a key
	extern __shared__ uint32_t pk_hist[];
	uint32_t *myh = pk_hist + ((threadIdx.x >> 5) % PK_HIST_COPIES) * (ND * 256);
	if (hist) {
		for (int i = threadIdx.x; i < PK_HIST_COPIES * ND * 256; i += blockDim.x)
			pk_hist[i] = 0;
		__syncthreads();
	}
	K lo1 = ~K(0), hi1 = 0, lo2 = ~K(0), hi2 = 0;
	bool nz = false;
	uint32_t ilo = 0xFFFFFFFFu, ihi = 0;
	bool dec = false, other = false;
	const uint64_t step = (uint64_t) gridDim.x * PK_THREADS * PK_ITEMS;
	for (uint64_t base = (uint64_t) blockIdx.x * PK_THREADS * PK_ITEMS + threadIdx.x; base < n; base += step) {
		Point<T, HAS_ID> p[PK_ITEMS];
		uint32_t after[PK_ITEMS];  // the next point's id
#pragma unroll
		for (int u = 0; u < PK_ITEMS; u++) {
			const uint64_t r = base + u * PK_THREADS;
			if (r < n) {
				p[u] = pts[P ? P[r] : r];
				if constexpr (SCAN_IDS && HAS_ID)
					after[u] = r + 1 < n ? pts[r + 1].id : 0xFFFFFFFFu;
			}
		}
#pragma unroll
		for (int u = 0; u < PK_ITEMS; u++) {
			const uint64_t r = base + u * PK_THREADS;
			if (r >= n)
				break;
			if constexpr (SCAN_IDS && HAS_ID) {
				const uint32_t v = p[u].id;
				ilo = min(ilo, v);
				ihi = max(ihi, v);
				dec |= v > after[u];
				other |= (uint64_t) v != r;
			}
			const K a = KeyOf<T>::key(p[u].dim1), b = KeyOf<T>::key(p[u].dim2);
			if constexpr (!std::is_integral<T>::value)
				nz |= (p[u].dim1 == T(0) && signbit(p[u].dim1)) || (p[u].dim2 == T(0) && signbit(p[u].dim2));
			k1[r] = a;
			if constexpr (sizeof(K) == 4)
				c2[r] = ((uint64_t) b << 32) | (uint64_t) (r + 1);
			else
				k2[r] = b;
			if (hist) {
#pragma unroll
				for (int d = 0; d < ND; d++)
					atomicAdd(&myh[d * 256 + rs_digit(a, 8 * d)], 1u);
			}
			lo1 = a < lo1 ? a : lo1;
			hi1 = a > hi1 ? a : hi1;
			lo2 = b < lo2 ? b : lo2;
			hi2 = b > hi2 ? b : hi2;
		}
	}
	if (__any_sync(0xFFFFFFFFu, nz) && (threadIdx.x & 31) == 0)
		atomicOr(negzero, 1u);
	if constexpr (SCAN_IDS && HAS_ID) {
		if (__any_sync(0xFFFFFFFFu, dec) && (threadIdx.x & 31) == 0)
			atomicOr(idflag, 1u);
		if (__any_sync(0xFFFFFFFFu, other) && (threadIdx.x & 31) == 0)
			atomicOr(idflag, 2u);
		block_range_fold<uint32_t>(ilo, ihi, id_range);
		__syncthreads();
	}
	block_range_fold<K>(lo1, hi1, range);
	__syncthreads();
	block_range_fold<K>(lo2, hi2, range + 2);
	if (hist) {
		__syncthreads();
		for (int i = threadIdx.x; i < ND * 256; i += blockDim.x) {
			uint32_t t = 0;
#pragma unroll
			for (int c = 0; c < PK_HIST_COPIES; c++)
				t += pk_hist[c * ND * 256 + i];
			if (t)
				atomicAdd(&hist[i], t);
		}
	}
}

// Doubles: S2 = dim2-sorted position -> tb (null: identity); c2[tb] = rank << 32 | tb + 1.
__global__ void k_rank_keys(const uint32_t *S2, uint64_t n, uint64_t *c2)
{
	for (uint64_t j = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t) gridDim.x * blockDim.x) {
		const uint32_t tb = S2 ? S2[j] : (uint32_t) j;
		c2[tb] = (j << 32) | (uint64_t) (tb + 1);
	}
}

// Point count of the node at level d, index j within the level (trees hold fewer than
// 2^31 points).  Construction gives a node of c points a left child of floor(c/2) and a
// right child of c - 1 - floor(c/2) points (pst/static-pst-cpu-iter.tpp:512-541), so
// counts depend on n and the node's path only.
__device__ __forceinline__ uint32_t node_count32(uint32_t n, uint32_t d, uint32_t j)
{
	uint32_t c = n;
	for (int b = (int) d - 1; b >= 0 && c != 0; b--)
		c = ((j >> b) & 1u) ? c - 1u - (c >> 1) : c >> 1;
	return c;
}

// ---------------------------------------------------------------------------
// Wide levels.

// The largest of the lanes' 64-bit keys.
__device__ __forceinline__ uint64_t warp_max_key(uint64_t k)
{
	const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t) (k >> 32));
	const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t) (k >> 32) == hi ? (uint32_t) k : 0u);
	return (uint64_t) hi << 32 | lo;
}

// Keys of tile t, lane + 32 k at v[k] (0 past n), all in flight together.
__device__ __forceinline__ void load_tile(const uint64_t *c2s, uint64_t n, uint64_t t, uint64_t (&v)[TM_TILE / 32])
{
	const uint64_t i = t * TM_TILE + lane_id();
#pragma unroll
	for (uint32_t k = 0; k < TM_TILE / 32; k++)
		v[k] = i + 32 * k < n ? c2s[i + 32 * k] : 0ull;
}

// First maxima: a CTA per TM_SUPER tiles.
__global__ void __launch_bounds__(LV_THREADS) k_tile_max(const uint64_t *__restrict__ c2s, uint64_t n, uint64_t *tmax,
                                                         uint64_t *smax)
{
	__shared__ uint64_t s_m[LV_THREADS / 32];
	const uint64_t ntiles = (n + TM_TILE - 1) / TM_TILE;
	const uint32_t warp = threadIdx.x >> 5;
	uint64_t best = 0;
	for (uint32_t k = warp; k < TM_SUPER; k += LV_THREADS / 32) {
		const uint64_t t = (uint64_t) blockIdx.x * TM_SUPER + k;
		if (t >= ntiles)
			break;
		uint64_t v[TM_TILE / 32], m = 0;
		load_tile(c2s, n, t, v);
#pragma unroll
		for (uint32_t i = 0; i < TM_TILE / 32; i++)
			m = max(m, v[i]);
		m = warp_max_key(m);
		best = max(best, m);
		if (lane_id() == 0)
			tmax[t] = m;
	}
	if (lane_id() == 0)
		s_m[warp] = best;
	__syncthreads();
	if (warp == 0) {
		best = warp_max_key(lane_id() < LV_THREADS / 32 ? s_m[lane_id()] : 0ull);
		if (lane_id() == 0)
			smax[blockIdx.x] = best;
	}
}

// Where a node's largest key was seen: a position, a tile, or TM_SUPER tiles.
constexpr uint32_t AT_TILE = 0x80000000u, AT_SUPER = 0xC0000000u, AT_INDEX = 0x3FFFFFFFu;

// Level d of the wide levels: GROUP threads (32 or LV_THREADS) per node.  Bounds are
// dim1-sorted positions that still include points taken by ancestors; those (each the
// point of one ancestor) are skipped when counting to the median.
//
// A tile (or 32) is only asked for its maximum while it lies inside one node, so it is
// only that node's warp that changes it, and a tile that a bound cuts is never asked
// again: no maximum is brought up to date for it.  A level waits on a chain of some six
// loads, not on bandwidth, until its nodes get down to a few tiles; then it reads the
// keys of the tiles that bounds cut, about 6 kB a node.  In place of three kernels a level
// (arg-max by tiles, a binary search for the winner's position by a thread per node, a
// second reduction of the tiles that lost a point): 450 -> 69 us for the 12 levels of
// 2^21 points with the first maxima, 1.15 -> 0.38 ms for the 17 of 2^26.
template <typename T, bool HAS_ID, int GROUP>
__global__ void __launch_bounds__(LV_THREADS) k_level(BuildCtx<T, HAS_ID> c, uint32_t d, const uint32_t *B, uint32_t *Bn)
{
	// a programmatic dependent of the level before it
	asm volatile("griddepcontrol.wait;" ::: "memory");
	__shared__ uint64_t s_key[LV_THREADS / 32];
	__shared__ uint32_t s_at[LV_THREADS / 32];
	const uint32_t nseg = 1u << d;
	const uint32_t j = blockIdx.x * (LV_THREADS / GROUP) + threadIdx.x / GROUP;
	if (j >= nseg)
		return;
	const uint32_t lane = lane_id(), t = threadIdx.x % GROUP;
	const uint32_t h = nseg + j;
	const uint32_t lo = B[j], hi = B[j + 1];
	const bool err = __any_sync(0xFFFFFFFFu, *c.err != 0);
	// the ancestors' positions, wanted for the median
	const uint32_t anc = lane < d ? c.top_pos[h >> (lane + 1)] : 0u;
	const uint32_t cnt = node_count32((uint32_t) c.n, d, j);
	// after an error the bounds may hold unwritten entries (a CTA's warps find out together,
	// below: one that returned alone would leave its words of s_key unwritten)
	if (GROUP == 32 && err)
		return;
	if (cnt < 2 || lo >= hi || hi > c.n) {
		if (t == 0)
			atomicOr(c.err, 1u);
		return;
	}
	uint64_t key = 0;
	uint32_t at = 0;
	auto see = [&](uint64_t k, uint32_t a) {
		if (k > key) {
			key = k;
			at = a;
		}
	};
	// whole tiles [tf, tl), and the positions before and after them
	const uint32_t tf = (uint32_t) (((uint64_t) lo + TM_TILE - 1) / TM_TILE), tl = hi / TM_TILE;
	const bool tiles = tf < tl;
	const uint32_t head = tiles ? tf * TM_TILE - lo : hi - lo, rest = tiles ? tl * TM_TILE : 0u;
	const uint32_t np = tiles ? head + (hi - rest) : head;
	constexpr int U = 8;  // loads in flight
	for (uint32_t i0 = t; i0 < np; i0 += GROUP * U) {
		uint64_t v[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint32_t i = i0 + u * GROUP;
			v[u] = i < np ? c.c2s[i < head ? lo + i : rest + (i - head)] : 0ull;
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint32_t i = i0 + u * GROUP;
			see(v[u], i < head ? lo + i : rest + (i - head));
		}
	}
	if (tiles) {
		// whole groups of tiles [sf, sl), and the tiles before and after them
		const uint32_t sf = (tf + TM_SUPER - 1) / TM_SUPER, sl = tl / TM_SUPER;
		const bool supers = sf < sl;
		const uint32_t th = supers ? sf * TM_SUPER : tl, tr = supers ? sl * TM_SUPER : tl;
		for (uint32_t i = tf + t; i < th; i += GROUP)
			see(c.tmax[i], AT_TILE | i);
		for (uint32_t i = tr + t; i < tl; i += GROUP)
			see(c.tmax[i], AT_TILE | i);
		if (supers) {
#pragma unroll 4
			for (uint32_t i = sf + t; i < sl; i += GROUP)
				see(c.smax[i], AT_SUPER | i);
		}
	}
	uint64_t best = warp_max_key(key);
	at = __shfl_sync(0xFFFFFFFFu, at, __ffs(__ballot_sync(0xFFFFFFFFu, key == best)) - 1);
	if constexpr (GROUP > 32) {
		if (lane == 0) {
			s_key[threadIdx.x >> 5] = best;
			s_at[threadIdx.x >> 5] = at;
		}
		if (__syncthreads_or(err) || threadIdx.x >= 32)
			return;
		key = lane < LV_THREADS / 32 ? s_key[lane] : 0ull;
		best = warp_max_key(key);
		at = s_at[(__ffs(__ballot_sync(0xFFFFFFFFu, key == best)) - 1) % (LV_THREADS / 32)];
	}
	// from here on one warp; every value below is the same in all its lanes, or a lane's own
	if (best == 0) {
		if (lane == 0)
			atomicOr(c.err, 8u);
		return;
	}
	uint32_t tp = at;
	if (at >= AT_TILE) {
		uint64_t other = 0;  // maxima of the other tiles of the group
		uint32_t tile = at & AT_INDEX;
		if (at >= AT_SUPER) {
			const uint64_t m = c.tmax[tile * TM_SUPER + lane];
			const uint32_t w = __ffs(__ballot_sync(0xFFFFFFFFu, m == best)) - 1;
			other = lane == w ? 0ull : m;
			tile = tile * TM_SUPER + (w & 31u);
		}
		uint64_t v[TM_TILE / 32], m = 0;
		load_tile(c.c2s, c.n, tile, v);
		uint32_t k = TM_TILE / 32;
#pragma unroll
		for (uint32_t i = 0; i < TM_TILE / 32; i++) {
			if (v[i] == best)
				k = i;
			else
				m = max(m, v[i]);
		}
		const uint32_t w = __ffs(__ballot_sync(0xFFFFFFFFu, k < TM_TILE / 32));
		if (w == 0) {
			if (lane == 0)
				atomicOr(c.err, 8u);
			return;
		}
		tp = tile * TM_TILE + 32 * __shfl_sync(0xFFFFFFFFu, k, w - 1) + w - 1;
		m = warp_max_key(m);
		if (lane == 0)
			c.tmax[tile] = m;
		if (at >= AT_SUPER) {
			m = max(m, warp_max_key(other));
			if (lane == 0)
				c.smax[at & AT_INDEX] = m;
		}
	}
	if (tp < lo || tp >= hi) {
		if (lane == 0)
			atomicOr(c.err, 8u);
		return;
	}
	// the median: the floor(cnt / 2)-th position of [lo, hi) that no ancestor's point, nor
	// this node's, holds: the smallest pos = first + (positions taken up to pos)
	const uint32_t mine = lane == 31 ? tp : anc;
	const bool inside = (lane == 31 || lane < d) && mine >= lo && mine < hi;
	const uint32_t first = lo + cnt / 2 - 1;
	uint32_t pos = first;
	for (;;) {
		const uint32_t p = first + __popc(__ballot_sync(0xFFFFFFFFu, inside && mine <= pos));
		if (p == pos)
			break;
		pos = p;
	}
	if (pos >= hi) {
		if (lane == 0)
			atomicOr(c.err, 4u);
		return;
	}
	if (lane == 0) {
		Bn[2 * j] = lo;
		Bn[2 * j + 1] = pos + 1;
		if (j == nseg - 1)
			Bn[2 * nseg] = hi;
		c.top_pos[h] = tp;
		c.write_node(h, c.point_of(tp, best));
		c.c2s[tp] = 0;
		// every node of a wide level exists
		if (nseg < 32)
			atomicOr(&c.occ[0], 1u << h);
		else if (j % 32 == 0)
			c.occ[h >> 5] = 0xFFFFFFFFu;
	}
	if (lane == 1)
		c.med[h] = c.point_of(pos, c.c2s[pos]).dim1;
}

// ---------------------------------------------------------------------------
// Subtree builder: one CTA per node of level L0 finishes its whole subtree.
//
// The CTA gathers the 64-bit dim2 keys of its free points in dim1 order into shared
// memory.  Sub-levels whose nodes hold more than 32 points are built in place, a warp per
// node, as the wide levels are: from the maxima of 32 positions and the positions that a
// node's bounds cut, a taken key becoming 0.  Then a warp takes each node of at most 32
// points, a point a lane, and builds all of its sub-levels in registers: a lane knows the
// lanes of its node (a mask) and the node's place; the largest key of a node is a scan over
// its lanes; the lane that holds it writes the node, the lane next to the left half's end
// its median, and every other lane goes down to a child.  No key moves, no lane waits for
// another warp.
//
// Bound by instruction issue (81 % of the cycles at 2^24 points).  With a compaction of all
// keys per sub-level (each a pass for the maxima, one for the node writes and one to move the
// keys, with barriers between) the kernel took 2654 us at 2^26 points, 92 at 2^21 and 463 at 5 M doubles; now 1896, 68 and
// 258.  Of the 1896, a copy that stops early puts some 400 in the gather, 500 in the
// sub-levels of large nodes and 300 before the first sub-level of the small ones.  CTAs of
// 256 threads took 2184 us (more wait at the barriers), of 64 1836 (but 0.5 % more in all at
// 2^21 points and 5 M doubles), of 32 no less; 256 points a CTA 1957 us and a wide level more.

constexpr uint32_t ST_ROWS = ST_CAP / 32;           // positions of a warp-wide row
constexpr uint32_t ST_TOP = ST_ROWS;                // nodes of at most 32 points, at most
constexpr int ST_WARPS = ST_THREADS / 32;
static_assert(ST_CAP == 512 && ST_TOP <= 32, "rows and top nodes are counted in lanes");

// Chunks of ST_THREADS positions the key gather reads: a node's range holds its
// cN <= ST_CAP free points and at most one point taken by each ancestor (< 32).
constexpr int ST_GATHER = (ST_CAP + ST_THREADS - 1) / ST_THREADS + 1;

// A lane of a warp that builds a node of at most 32 points: its point and dim2 key, whether
// the point is still free, the lanes of its node that are, and the node's place.
template <typename T, bool HAS_ID>
struct SubtreeLane {
	Point<T, HAS_ID> pt;
	uint32_t hi, lo;  // the dim2 key's words
	bool alive;
	bool right;       // its node is a right child
	uint32_t seg, h;
};

// The largest value of the lanes of the lane's node, at its last lane: a scan over the
// lanes from its first on, which lie within the node's points (32 >> U at most) and one
// lane for each ancestor in the warp.
template <int U>
__device__ __forceinline__ uint32_t node_max(uint32_t v, uint32_t past_start)
{
	constexpr uint32_t SPAN = (32u >> U) + U;
#pragma unroll
	for (uint32_t o = 1; o < SPAN && o < 32; o <<= 1) {
		const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, v, o);
		if (past_start >= o)
			v = max(v, x);
	}
	return v;
}

// Sub-levels U .. 5 of the warp's node, `left` of them below sub-level 0.
template <typename T, bool HAS_ID, int U>
__device__ __forceinline__ void subtree_levels(const BuildCtx<T, HAS_ID> &c, SubtreeLane<T, HAS_ID> &me, uint32_t left,
                                               uint32_t half, uint32_t first, uint32_t *s_occ)
{
	const uint32_t below = lanemask_lt(), seg = me.seg;
	// the largest key's high word, then, where a node has several of it, its low word
	bool win;
	if constexpr (U == 5) {
		win = me.alive;  // one point a node
	} else {
		const uint32_t start = __ffs(seg) - 1, end = (31 - __clz(seg)) & 31, past = lane_id() - start;
		// (a dead lane's past may wrap round: its value is never read)
		const uint32_t v = me.alive ? me.hi : 0u;
		uint32_t top;
		if constexpr (U == 0) {
			top = __reduce_max_sync(0xFFFFFFFFu, v);
		} else if constexpr (U == 1) {
			const uint32_t l = __reduce_max_sync(0xFFFFFFFFu, me.right ? 0u : v),
			               r = __reduce_max_sync(0xFFFFFFFFu, me.right ? v : 0u);
			top = me.right ? r : l;
		} else {
			top = __shfl_sync(0xFFFFFFFFu, node_max<U>(v, past), end);
		}
		win = me.alive && me.hi == top;
		const uint32_t many = __ballot_sync(0xFFFFFFFFu, win) & seg;
		if (__any_sync(0xFFFFFFFFu, win && (many & (many - 1)) != 0)) {
			const uint32_t low = __shfl_sync(0xFFFFFFFFu, node_max<U>(win ? me.lo : 0u, past), end);
			win = win && me.lo == low;
		}
	}
	const uint32_t rest = seg & ~__ballot_sync(0xFFFFFFFFu, win);
	const uint32_t ct = __popc(seg), r = __popc(rest & below), lh = ct / 2;
	if (win) {
		c.write_node(me.h, me.pt);
		if (ct == 1 && me.h < half)
			c.med[me.h] = me.pt.dim1;  // a node of one point: its own dim1
		if (U == left)
			atomicOr(&s_occ[(me.h - first) >> 5], 1u << ((me.h - first) & 31));
		me.alive = false;
	}
	if constexpr (U < 5) {
		if (U == left)
			return;
		// the left child's lanes end with the median's
		const bool med = me.alive && r + 1 == lh;
		if (med)
			c.med[me.h] = me.pt.dim1;
		const uint32_t mm = __ballot_sync(0xFFFFFFFFu, med) & seg;
		const uint32_t lm = mm ? rest & (2u * mm - 1u) : 0u;
		me.right = r >= lh;
		me.seg = me.right ? rest & ~lm : lm;
		me.h = 2 * me.h + (me.right ? 1u : 0u);
		subtree_levels<T, HAS_ID, U + 1>(c, me, left, half, first, s_occ);
	}
}

template <typename T, bool HAS_ID>
__global__ void __launch_bounds__(ST_THREADS) k_subtree(BuildCtx<T, HAS_ID> c, uint32_t L0,
                                                       const uint32_t *__restrict__ B)
{
	using Ctx = BuildCtx<T, HAS_ID>;
	using K = typename Ctx::K;
	using Pt = Point<T, HAS_ID>;
	constexpr bool KEYS4 = sizeof(K) == 4;
	__shared__ uint64_t s_key[ST_CAP];            // 0 once taken
	__shared__ K s_k1[KEYS4 ? ST_CAP : 1];        // dim1 keys (with rebuilt points)
	__shared__ uint64_t s_row[ST_ROWS];           // largest key of 32 positions
	__shared__ uint16_t s_b[2][ST_TOP + 1];       // bounds of the sub-level's nodes
	__shared__ uint16_t s_top[ST_TOP];            // position of the point of sub-node 1, 2, 3, ..
	__shared__ uint16_t s_list[ST_WARPS][32];
	__shared__ uint32_t s_occ[2 * ST_CAP / 32];   // occupied nodes of the last level
	__shared__ uint32_t s_pre[ST_GATHER][ST_WARPS];
	__shared__ uint32_t s_n;

	const uint32_t j = blockIdx.x;
	const uint32_t cN = node_count32((uint32_t) c.n, L0, j);
	const bool err = *c.err != 0;
	if (cN == 0)
		return;
	const uint32_t lo0 = L0 ? B[j] : 0u;
	const uint32_t hi0 = L0 ? B[j + 1] : (uint32_t) c.n;
	if (lo0 >= hi0 || hi0 > c.n || cN > ST_CAP || hi0 - lo0 > (uint32_t) (ST_GATHER * ST_THREADS)) {
		if (threadIdx.x == 0)
			atomicOr(c.err, 16u);
		return;
	}
	const uint32_t warp = threadIdx.x >> 5, lane = lane_id();

	// Gather the keys of the points still free in [lo0, hi0), in dim1 order: every
	// read in flight at once, then one prefix over (chunk, warp).
	{
		uint64_t v[ST_GATHER];
		K v1[ST_GATHER];
		uint32_t m[ST_GATHER];
#pragma unroll
		for (int u = 0; u < ST_GATHER; u++) {
			const uint32_t i = lo0 + (uint32_t) u * ST_THREADS + threadIdx.x;
			const bool in = i < hi0;
			v[u] = in ? c.c2s[i] : 0;
			v1[u] = (KEYS4 && c.recon && in) ? c.k1s[i] : K(0);
		}
#pragma unroll
		for (int u = 0; u < ST_GATHER; u++) {
			m[u] = __ballot_sync(0xFFFFFFFFu, v[u] != 0);
			if (lane == 0)
				s_pre[u][warp] = __popc(m[u]);
		}
		for (uint32_t i = threadIdx.x; i < 2 * ST_CAP / 32; i += ST_THREADS)
			s_occ[i] = 0;
		// (together: a warp that returned alone would leave its counts and keys unwritten)
		if (__syncthreads_or(err))
			return;
		if (warp == 0) {
			// (chunk, warp) pairs in order, a lane each
			constexpr int PAIRS = ST_GATHER * ST_WARPS;
			static_assert(PAIRS <= 32, "a pair a lane");
			uint32_t *flat = &s_pre[0][0];
			const uint32_t n = lane < PAIRS ? flat[lane] : 0u;
			const uint32_t inc = warp_incl_scan(n);
			if (lane < PAIRS)
				flat[lane] = inc - n;
			if (lane == 31)
				s_n = inc;
		}
		__syncthreads();
#pragma unroll
		for (int u = 0; u < ST_GATHER; u++) {
			if ((m[u] >> lane) & 1u) {
				const uint32_t pos = s_pre[u][warp] + __popc(m[u] & lanemask_lt());
				if (pos < ST_CAP) {
					s_key[pos] = v[u];
					if (KEYS4 && c.recon)
						s_k1[pos] = v1[u];
				}
			}
		}
	}
	if (threadIdx.x == 0) {
		s_b[0][0] = 0;
		s_b[0][1] = (uint16_t) cN;
	}
	__syncthreads();
	if (s_n != cN) {
		if (threadIdx.x == 0)
			atomicOr(c.err, 2u);
		return;
	}
	// the point at position pos, whose key is (or was) `key`
	auto point_at = [&](uint32_t pos, uint64_t key) -> Pt {
		if constexpr (KEYS4) {
			if (c.recon)
				return Ctx::point_from_keys(s_k1[pos], key);
		}
		return c.point_of_tb(Ctx::tb_of(key));
	};
	const uint32_t h0 = (1u << L0) + j;
	const uint32_t last_s = c.D - 1 - L0;
	const uint32_t half = 1u << (c.D - 1);  // med exists for positions < half
	// sub-levels whose largest node (cN >> s points) holds more than 32
	uint32_t S = 0;
	while ((cN >> S) > 32)
		S++;
	if (S) {
		for (uint32_t r = warp; r < (cN + 31) / 32; r += ST_WARPS) {
			const uint64_t k = 32 * r + lane < cN ? s_key[32 * r + lane] : 0ull;
			const uint64_t m = warp_max_key(k);
			if (lane == 0)
				s_row[r] = m;
		}
		__syncthreads();
	}
	for (uint32_t s = 0; s < S; s++) {
		const uint16_t *b = s_b[s & 1];
		uint16_t *bn = s_b[(s + 1) & 1];
		for (uint32_t t = warp; t < (1u << s); t += ST_WARPS) {
			const uint32_t lo = b[t], hi = b[t + 1];
			const uint32_t h = (h0 << s) + t;
			const uint32_t anc = lane < s ? s_top[((1u << s) + t) >> (lane + 1)] : 0u;
			// the node's points: its positions without those that its ancestors took
			const bool took = lane < s && anc >= lo && anc < hi;
			const uint32_t ct = hi - lo - __popc(__ballot_sync(0xFFFFFFFFu, took));
			// whole rows [rf, rl), and the positions before and after them (a node without
			// whole rows spans fewer than 64 positions)
			const uint32_t rf = (lo + 31) / 32, rl = hi / 32;
			const bool rows = rf < rl;
			const uint32_t p0 = lo + lane, p1 = rows ? 32 * rl + lane : lo + 32 + lane;
			const uint64_t k0 = p0 < (rows ? 32 * rf : hi) ? s_key[p0] : 0ull, k1 = p1 < hi ? s_key[p1] : 0ull,
			               kr = rows && rf + lane < rl ? s_row[rf + lane] : 0ull;
			const uint64_t best = warp_max_key(max(max(k0, k1), kr));
			const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, k0 == best), b1 = __ballot_sync(0xFFFFFFFFu, k1 == best),
			               br = __ballot_sync(0xFFFFFFFFu, kr == best);
			uint32_t tp;
			if (b0) {
				tp = lo + __ffs(b0) - 1;
			} else if (b1) {
				tp = (rows ? 32 * rl : lo + 32) + __ffs(b1) - 1;
			} else {
				const uint32_t r = rf + __ffs(br) - 1;
				const uint64_t k = s_key[32 * r + lane];
				tp = 32 * r + __ffs(__ballot_sync(0xFFFFFFFFu, k == best)) - 1;
				const uint64_t m = warp_max_key(k == best ? 0ull : k);
				if (lane == 0)
					s_row[r] = m;
			}
			if (best == 0 && lane == 0)
				atomicOr(c.err, 8u);
			// the median, as on the wide levels
			const uint32_t first = lo + ct / 2 - 1;
			uint32_t pos = first;
			for (;;) {
				const uint32_t p = first + (tp <= pos) + __popc(__ballot_sync(0xFFFFFFFFu, took && anc <= pos));
				if (p == pos)
					break;
				pos = p;
			}
			if (pos >= hi) {
				if (lane == 0)
					atomicOr(c.err, 4u);
				pos = hi - 1;
			}
			if (lane == 0) {
				bn[2 * t] = (uint16_t) lo;
				bn[2 * t + 1] = (uint16_t) (pos + 1);
				if (t + 1 == (1u << s))
					bn[2 * t + 2] = (uint16_t) hi;
				s_top[(1u << s) + t] = (uint16_t) tp;
				c.write_node(h, point_at(tp, best));
				s_key[tp] = 0;
			}
			if (lane == 1)
				c.med[h] = point_at(pos, s_key[pos]).dim1;
		}
		__syncthreads();
	}
	for (uint32_t t = warp; t < (1u << S); t += ST_WARPS) {
		const uint32_t lo = s_b[S & 1][t], hi = s_b[S & 1][t + 1];
		// the free positions of the node, in order: at most 32 among its own and its
		// ancestors'
		const uint32_t p0 = lo + lane, p1 = p0 + 32;
		const bool f0 = p0 < hi && s_key[p0] != 0, f1 = p1 < hi && s_key[p1] != 0;
		const uint32_t a0 = __ballot_sync(0xFFFFFFFFu, f0), a1 = __ballot_sync(0xFFFFFFFFu, f1);
		const uint32_t n0 = __popc(a0), cnt = n0 + __popc(a1);
		if (cnt > 32) {
			if (lane == 0)
				atomicOr(c.err, 2u);
			continue;
		}
		const uint32_t below = lanemask_lt();
		if (f0)
			s_list[warp][__popc(a0 & below)] = (uint16_t) p0;
		if (f1)
			s_list[warp][n0 + __popc(a1 & below)] = (uint16_t) p1;
		__syncwarp();
		bool alive = lane < cnt;
		uint64_t key = 0;
		Pt pt;
		if (alive) {
			const uint32_t pos = s_list[warp][lane];
			key = s_key[pos];
			pt = point_at(pos, key);
		}
		__syncwarp();  // the list is rewritten by the warp's next node
		// the lane's node: its lanes that are left, and its place
		SubtreeLane<T, HAS_ID> me{pt, (uint32_t) (key >> 32), (uint32_t) key, alive, false,
		                          cnt < 32 ? (1u << cnt) - 1u : 0xFFFFFFFFu, (h0 << S) + t};
		const uint32_t first = h0 << last_s;  // the CTA's first place on the last level
		subtree_levels<T, HAS_ID, 0>(c, me, last_s - S, half, first, s_occ);
	}
	__syncthreads();
	// occupancy: every node above the last level exists
	for (uint32_t s = threadIdx.x; s <= last_s; s += ST_THREADS) {
		const uint32_t base = h0 << s;
		if (s < 5) {
			const uint32_t bits = s == last_s ? s_occ[0] : (1u << (1u << s)) - 1u;
			atomicOr(&c.occ[base >> 5], bits << (base & 31));
		}
	}
	for (uint32_t s = 5; s <= last_s; s++)
		for (uint32_t w = threadIdx.x; w < (1u << (s - 5)); w += ST_THREADS)
			c.occ[((h0 << s) >> 5) + w] = s == last_s ? s_occ[w] : 0xFFFFFFFFu;
}

template <typename T>
T *as(void *p)
{
	return static_cast<T *>(p);
}

// All construction scratch lives in one device allocation.
struct ScratchLayout {
	size_t k1, kalt, c2, valt, k2, v32a, v32b, P, rs_status, rs_misc, hist1, flags, Ba, Bb, top, tmax, smax;
	size_t total;
};

ScratchLayout scratch_layout(pst_dtype dt, pst_idtype it, uint64_t n)
{
	ScratchLayout L{};
	const size_t ks = value_size(dt);
	const bool wide_key = dt == PST_F64;
	const uint32_t D = tree_levels(n);
	const uint32_t L0 = n ? std::min(subtree_level(n), D - 1) : 0;
	const uint64_t nodes_wide = 1ull << L0;
	const uint64_t rs_tiles = rs_num_tiles(n);
	const uint64_t ntiles = (n + TM_TILE - 1) / TM_TILE;
	size_t o = 0;
	auto take = [&](size_t bytes) {
		const size_t r = o;
		o = align_up(o + bytes);
		return r;
	};
	L.k1 = take(n * ks);
	L.kalt = take(n * ks);
	L.c2 = take(n * 8);
	L.valt = take(n * 8);
	L.k2 = take(wide_key ? n * 8 : 0);
	L.v32a = take(wide_key ? n * 4 : 0);
	L.v32b = take(wide_key ? n * 4 : 0);
	L.P = take(it == PST_ID_U32 ? n * 4 : 0);
	L.rs_status = take(256 * rs_tiles * 8);
	L.rs_misc = take(rs_misc_words() * 4);
	L.hist1 = take(RS_MAX_PASSES * 256 * 4);
	L.flags = take(256);
	L.Ba = take((nodes_wide + 1) * 4);
	L.Bb = take((nodes_wide + 1) * 4);
	L.top = take(nodes_wide * 4);
	L.tmax = take(L0 ? ntiles * 8 : 0);
	L.smax = take(L0 ? (ntiles + TM_SUPER - 1) / TM_SUPER * 8 : 0);
	L.total = o;
	return L;
}

struct Scratch {
	cudaStream_t s;
	char *base;
	Scratch(size_t bytes, cudaStream_t stream)
	    : s(stream), base(static_cast<char *>(pool_alloc(bytes, "construction scratch")))
	{
	}
	~Scratch()
	{
		cudaStreamSynchronize(s);  // the construction's work
		pool_release(base, device_info().device);
	}
	Scratch(const Scratch &) = delete;
	Scratch &operator=(const Scratch &) = delete;
	template <typename T>
	T *at(size_t off) const
	{
		return reinterpret_cast<T *>(base + off);
	}
};

inline unsigned grid_for(uint64_t n, int threads)
{
	const uint64_t want = (n + threads - 1) / threads;
	const uint64_t cap = (uint64_t) device_info().sms * 16;
	return (unsigned) std::max<uint64_t>(1, std::min(want, cap));
}

// Scratch bytes of build_impl beyond the tree itself.
uint64_t build_scratch_bytes(pst_dtype dt, pst_idtype it, uint64_t n) { return scratch_layout(dt, it, n).total; }

// The tree's memory (one allocation; its occupancy bitmap cleared on `s`).  Called
// with the builder's sorts already queued on `s`: mapping several GB takes the host
// milliseconds, which then overlap the sorts instead of preceding them.
void alloc_tree(TreeStorage &t, cudaStream_t s)
{
	const TreeLayout L = tree_layout(t.dtype, t.idtype, t.n);
	attach_tree_memory(t, pool_alloc(L.total, "tree"));
	PST_CUDA(cudaMemsetAsync(t.occ, 0, L.total - L.off_occ, s));
}

template <typename T, bool HAS_ID>
void build_impl(TreeStorage &t, const void *pts_d, uint64_t n, cudaStream_t s)
{
	using K = typename KeyOf<T>::K;
	using Pt = Point<T, HAS_ID>;
	constexpr bool WIDE_KEY = sizeof(K) == 8;  // doubles: dim2 ranks from their own sort
	const Pt *pts = static_cast<const Pt *>(pts_d);
	const uint32_t D = t.levels;

	// ---- scratch
	const ScratchLayout SL = scratch_layout(t.dtype, t.idtype, n);
	Scratch scr(SL.total, s);
	void *k1 = scr.at<void>(SL.k1), *kalt = scr.at<void>(SL.kalt);
	uint64_t *c2 = scr.at<uint64_t>(SL.c2);
	void *valt = scr.at<void>(SL.valt);
	uint32_t *flag = scr.at<uint32_t>(SL.flags);  // the words of BuildFlags
	K *krange = reinterpret_cast<K *>(scr.at<unsigned char>(SL.flags) + 64);  // [k1 min, k1 max, k2 min, k2 max]
	// one SortScratch for every sort of this build: its epoch tags the look-back
	// status of each pass, which is cleared only here
	SortScratch sc;
	sc.status = scr.at<uint64_t>(SL.rs_status);
	sc.hist = scr.at<uint32_t>(SL.rs_misc);
	sc.counters = sc.hist + RS_MAX_PASSES * 256;
	sc.err = flag + 1;
	sc.cleared = true;
	uint32_t *B = scr.at<uint32_t>(SL.Ba), *Bn = scr.at<uint32_t>(SL.Bb);
	// the sorts' status, counters and the digit counts, which lie side by side
	PST_CUDA(cudaMemsetAsync(sc.status, 0, SL.flags - SL.rs_status, s));
	k_build_init<K><<<1, 64, 0, s>>>(flag, B, (uint32_t) n);
	PST_CUDA(cudaGetLastError());

	const unsigned g = grid_for(n, 256);
	// ---- keys, made in input order; the same pass checks the ids and counts the
	// dim1 keys' digits for their sort
	uint32_t *hist1 = scr.at<uint32_t>(SL.hist1);
	const unsigned pk_g = (unsigned) std::min<uint64_t>((n + PK_THREADS * PK_ITEMS - 1) / (PK_THREADS * PK_ITEMS),
	                                                    (uint64_t) device_info().sms * PK_CTAS);
	const size_t pk_smem = (size_t) PK_HIST_COPIES * sizeof(K) * 256 * 4;
	k_prep_keys<T, HAS_ID, HAS_ID><<<pk_g, PK_THREADS, pk_smem, s>>>(pts, nullptr, n, static_cast<K *>(k1), c2,
	                                                       scr.at<K>(SL.k2), krange, flag + 4, flag, flag + 2,
	                                                       hist1);
	PST_CUDA(cudaGetLastError());
	BuildFlags<K> seen;
	PST_CUDA(cudaMemcpyAsync(&seen, flag, sizeof(seen), cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	const K *range = seen.range;
	const bool negzero = seen.negzero != 0;
	// ---- tiebreak order (id, input index): the input order unless the ids decrease
	// somewhere, then the keys are made again in the order of one sort of the ids
	const uint32_t *P = nullptr;
	bool ids_are_indices = true;
	if constexpr (HAS_ID) {
		ids_are_indices = !(seen.id_order & 2u);
		if (seen.id_order & 1u) {
			uint32_t *idk = static_cast<uint32_t *>(k1);  // k1 holds at least n u32
			k_id_keys<T, HAS_ID><<<g, 256, 0, s>>>(pts, n, idk);
			sc.keys_alt = kalt;
			sc.vals_alt = valt;  // n u32 fit in the u64 buffers
			sc.vals_tmp = c2;
			uint32_t *kres, *vres;
			radix_sort<uint32_t, uint32_t>(idk, nullptr, n, rs_passes<uint32_t>(seen.id_range[0], seen.id_range[1]), sc,
			                               &kres, &vres, s);
			// ids decrease somewhere, so they are not all equal and the sort ran
			PST_CUDA(cudaMemcpyAsync(scr.at<uint32_t>(SL.P), vres, n * 4, cudaMemcpyDeviceToDevice, s));
			P = scr.at<uint32_t>(SL.P);
			// the same keys in the new order: ranges and digit counts stand, so neither
			// is made again (the sort's error bits in flag[1] are kept)
			k_prep_keys<T, HAS_ID, false><<<pk_g, PK_THREADS, 0, s>>>(pts, P, n, static_cast<K *>(k1), c2, scr.at<K>(SL.k2),
			                                                krange, flag + 4, nullptr, nullptr, nullptr);
			PST_CUDA(cudaGetLastError());
		}
	}
	if constexpr (WIDE_KEY) {
		// dim2 ranks: stable sort of the dim2 keys in tiebreak order
		sc.keys_alt = kalt;
		sc.vals_alt = scr.at<void>(SL.v32a);
		sc.vals_tmp = scr.at<void>(SL.v32b);
		K *kres;
		uint32_t *S2;
		radix_sort<K, uint32_t>(scr.at<K>(SL.k2), nullptr, n, rs_passes<K>(range[2], range[3]), sc, &kres, &S2, s);
		k_rank_keys<<<g, 256, 0, s>>>(S2, n, c2);
		PST_CUDA(cudaGetLastError());
	}
	// ---- dim1 order, carrying the dim2 keys
	K *k1s;
	uint64_t *c2s;
	{
		sc.keys_alt = kalt;
		sc.vals_alt = valt;
		sc.vals_tmp = nullptr;
		radix_sort<K, uint64_t>(static_cast<K *>(k1), c2, n, rs_passes<K>(range[0], range[1]), sc, &k1s, &c2s, s,
		                        hist1);
	}
	alloc_tree(t, s);

	// ---- levels
	const uint32_t L0 = std::min(subtree_level(n), D - 1);
	const uint64_t nodes_wide = 1ull << L0;
	const uint64_t ntiles = (n + TM_TILE - 1) / TM_TILE;
	BuildCtx<T, HAS_ID> c;
	c.pts = pts;
	c.P = P;
	// points rebuilt from the keys: 4-byte values, no -0.0, ids (if any) = input indices
	c.recon = !WIDE_KEY && !negzero && ids_are_indices && P == nullptr;
	c.k1s = k1s;
	c.c2s = c2s;
	c.tmax = scr.at<uint64_t>(SL.tmax);
	c.smax = scr.at<uint64_t>(SL.smax);
	c.dim1 = as<T>(t.dim1);
	c.dim2 = as<T>(t.dim2);
	c.med = as<T>(t.med);
	c.id = t.id;
	c.occ = t.occ;
	c.top_pos = scr.at<uint32_t>(SL.top);
	c.err = flag + 1;
	c.n = n;
	c.D = D;
	if (L0) {
		k_tile_max<<<(unsigned) ((ntiles + TM_SUPER - 1) / TM_SUPER), LV_THREADS, 0, s>>>(c2s, n, c.tmax, c.smax);
		PST_CUDA(cudaGetLastError());
		for (uint32_t d = 0; d < L0; d++) {
			const uint32_t nseg = 1u << d;
			// a CTA per node while the device holds them all at once, a warp per node below
			const bool ctas = nseg <= (uint32_t) device_info().sms * 4;
			cudaLaunchConfig_t cfg{};
			cudaLaunchAttribute attr[1];
			attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
			attr[0].val.programmaticStreamSerializationAllowed = 1;
			cfg.gridDim = dim3(ctas ? nseg : (nseg + LV_THREADS / 32 - 1) / (LV_THREADS / 32));
			cfg.blockDim = dim3(LV_THREADS);
			cfg.stream = s;
			cfg.attrs = attr;
			cfg.numAttrs = 1;
			PST_CUDA(ctas ? cudaLaunchKernelEx(&cfg, k_level<T, HAS_ID, LV_THREADS>, c, d, (const uint32_t *) B, Bn)
			              : cudaLaunchKernelEx(&cfg, k_level<T, HAS_ID, 32>, c, d, (const uint32_t *) B, Bn));
			std::swap(B, Bn);
		}
	}
	k_subtree<T, HAS_ID><<<(unsigned) nodes_wide, ST_THREADS, 0, s>>>(c, L0, B);
	PST_CUDA(cudaGetLastError());
	finish_tree_aux(t, s);  // its reads stay inside the tree whatever the check below finds
	uint32_t errs[2] = {0, 0};
	PST_CUDA(cudaMemcpyAsync(errs, flag, 8, cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (errs[1])
		fail(PST_ERR_INTERNAL, "construction consistency check failed (code " + std::to_string(errs[1]) + ")");
}

}  // namespace

uint64_t tree_bytes(pst_dtype dt, pst_idtype it, uint64_t n) { return tree_layout(dt, it, n).total; }

void attach_tree_memory(TreeStorage &t, void *mem)
{
	const TreeLayout L = tree_layout(t.dtype, t.idtype, t.n);
	t.mem = mem;
	t.bytes = L.total;
	char *b = static_cast<char *>(mem);
	t.dim1 = b + L.off_dim1;
	t.dim2 = b + L.off_dim2;
	t.med = b + L.off_med;
	t.id = t.idtype == PST_ID_U32 ? reinterpret_cast<uint32_t *>(b + L.off_id) : nullptr;
	t.occ = reinterpret_cast<uint32_t *>(b + L.off_occ);
}

// The separately allocated search indexes of finish_tree_aux.
static uint64_t aux_bytes(pst_dtype dt, uint64_t n)
{
	const uint32_t D = tree_levels(n);
	if (D < 8)
		return 0;
	const uint64_t last_par = align_up(((1ull << (D - 2)) / 64 + 31) / 32 * 4);
	return last_par + (1ull << (D - 1)) / 64 * value_size(dt);
}

uint64_t build_bytes_needed(pst_dtype dt, pst_idtype it, uint64_t n)
{
	return tree_bytes(dt, it, n) + build_scratch_bytes(dt, it, n) + aux_bytes(dt, n);
}

void build_tree(TreeStorage &t, const void *pts_d, uint64_t n, cudaStream_t s)
{
	if (n >= (1ull << 31))
		fail(PST_ERR_INVALID, "at most 2^31 - 1 points per tree");
	t.n = n;
	t.levels = tree_levels(n);
	if (n == 0)
		return;
	if (!pts_d)
		fail(PST_ERR_INVALID, "null point array");
	try {
		// the tree's own memory is allocated by build_impl once its sorts are queued
		switch (t.dtype) {
		case PST_F32:
			t.idtype == PST_ID_U32 ? build_impl<float, true>(t, pts_d, n, s) : build_impl<float, false>(t, pts_d, n, s);
			break;
		case PST_F64:
			t.idtype == PST_ID_U32 ? build_impl<double, true>(t, pts_d, n, s) : build_impl<double, false>(t, pts_d, n, s);
			break;
		case PST_I32:
			t.idtype == PST_ID_U32 ? build_impl<int32_t, true>(t, pts_d, n, s) : build_impl<int32_t, false>(t, pts_d, n, s);
			break;
		}
	} catch (...) {
		cudaStreamSynchronize(s);
		free_tree(t);
		throw;
	}
}

namespace {

// Minimum of two dim2 values that keeps a NaN (so that no query's min2 compares
// at most the minimum of a block with a NaN below it).
__device__ __forceinline__ float min_keep_nan(float a, float b)
{
	float r;
	asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ int32_t min_keep_nan(int32_t a, int32_t b) { return min(a, b); }
__device__ __forceinline__ double min_keep_nan(double a, double b) { return a != a || a < b ? a : b; }

// A block without descendants holds nothing to test: the largest value.
template <typename T>
__device__ __forceinline__ T min_of_none()
{
	if constexpr (std::is_floating_point<T>::value)
		return std::numeric_limits<T>::infinity();
	else
		return std::numeric_limits<T>::max();
}

// sub_min of the 64-slot blocks of levels e, e - 1, .. e - depth + 1, and (where e is level
// D - 2) one bit per block of level e: does any of its children exist (last_par).  A block's
// value is the smallest dim2 of its 128 children on the level below it (positions
// 2^(level + 1) + 128 j ..; only the occupied ones on the last level) and of the two child
// blocks' values.  A CTA owns 2^(depth - 1) consecutive blocks of level e and all their
// ancestors down to one: the minima of their own children are independent reads, whatever
// the level, and the blocks' values are then folded up in shared memory.  SM_DEPTH levels a
// launch in place of one each: 2^26 points 256 us in 21 launches, 134 in 3; 2^21 40, 19.  (Level by
// level inside the CTA, with a barrier between them: 189 us.)
constexpr int SM_DEPTH = 7, SM_THREADS = 256, SM_WARPS = SM_THREADS / 32;

template <typename T>
__global__ void __launch_bounds__(SM_THREADS) k_sub_min(const T *__restrict__ dim2, const uint32_t *__restrict__ occ,
                                                        T *sub_min, uint32_t *last_par, uint32_t D, uint32_t e,
                                                        uint32_t depth)
{
	// the blocks in order of their level, e first, and of their place: block b of n is the
	// (2^(l + 1) - 1 - r)-th of 2^l blocks on level e - depth + 1 + l, r = n - b, l = log2 r
	__shared__ T s_min[1 << SM_DEPTH];
	__shared__ uint32_t s_any[2];
	constexpr int U = sizeof(T) == 4 ? 4 : 2;  // blocks in flight per warp
	const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
	const uint32_t n = (1u << depth) - 1, nb = 1u << (depth - 1);
	const bool last = e + 2 == D;
	if (threadIdx.x < 2)
		s_any[threadIdx.x] = 0;
	__syncthreads();
	for (uint32_t b0 = warp * U; b0 < n; b0 += SM_WARPS * U) {
		T v[U][4];
		uint32_t om[U];
		uint64_t p[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint32_t b = b0 + u, r = b < n ? n - b : 1u, l = 31 - __clz(r), lv = e - depth + 1 + l;
			const uint64_t j = ((uint64_t) blockIdx.x << l) + (2u << l) - 1 - r;
			p[u] = (1ull << (lv + 1)) + 128 * j + 4 * lane;
			om[u] = b >= n ? 0u : last && b < nb ? (occ[p[u] >> 5] >> (p[u] & 31)) & 0xFu : 0xFu;
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (!om[u])
				continue;  // a last level is often almost empty
			if constexpr (sizeof(T) == 4) {
				const uint4 x = *reinterpret_cast<const uint4 *>(dim2 + p[u]);
				memcpy(&v[u][0], &x.x, 4);
				memcpy(&v[u][1], &x.y, 4);
				memcpy(&v[u][2], &x.z, 4);
				memcpy(&v[u][3], &x.w, 4);
			} else {
				const double2 a = reinterpret_cast<const double2 *>(dim2 + p[u])[0];
				const double2 c = reinterpret_cast<const double2 *>(dim2 + p[u])[1];
				v[u][0] = a.x;
				v[u][1] = a.y;
				v[u][2] = c.x;
				v[u][3] = c.y;
			}
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (b0 + u >= n)
				break;
			T m = min_of_none<T>();
			if (__any_sync(0xFFFFFFFFu, om[u])) {
#pragma unroll
				for (int q = 0; q < 4; q++)
					m = (om[u] >> q) & 1u ? min_keep_nan(m, v[u][q]) : m;
#pragma unroll
				for (int o = 16; o > 0; o >>= 1)
					m = min_keep_nan(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
				if (last && b0 + u < nb && lane == 0)
					atomicOr(&s_any[(b0 + u) >> 5], 1u << ((b0 + u) & 31));
			}
			if (lane == 0)
				s_min[b0 + u] = m;
		}
	}
	__syncthreads();
	// the child blocks' values: of the launch before, then of the level just folded
	for (uint32_t l = depth; l-- > 0;) {
		const uint32_t on = 1u << l, at = n + 1 - (2u << l);  // blocks of the level, and their place
		for (uint32_t i = threadIdx.x; i < on; i += SM_THREADS) {
			T m = s_min[at + i];
			const uint64_t j = ((1ull << (e - depth + 1 + l)) >> 6) + ((uint64_t) blockIdx.x << l) + i;
			if (l + 1 < depth)
				m = min_keep_nan(m, min_keep_nan(s_min[at - 2 * on + 2 * i], s_min[at - 2 * on + 2 * i + 1]));
			else if (!last)
				m = min_keep_nan(m, min_keep_nan(sub_min[2 * j], sub_min[2 * j + 1]));
			s_min[at + i] = m;
			sub_min[j] = m;
		}
		__syncthreads();
	}
	// the CTA's bits: whole words of last_par, or (below 32 blocks in all) the start of one
	if (last && threadIdx.x < (nb + 31) / 32)
		last_par[(uint64_t) blockIdx.x * nb / 32 + threadIdx.x] = s_any[threadIdx.x];
}
static_assert(SM_DEPTH <= 7, "two words of last_par bits per CTA");

template <typename T>
void sub_min_launch(const TreeStorage &t, cudaStream_t s)
{
	// from the bottom up; a run ends at level 6, whose one block is level 6's
	for (uint32_t e = t.levels - 2; e >= 6;) {
		const uint32_t depth = std::min<uint32_t>(SM_DEPTH, e - 5);
		const uint64_t ctas = ((1ull << e) / 64) >> (depth - 1);
		k_sub_min<T><<<(unsigned) ctas, SM_THREADS, 0, s>>>(static_cast<const T *>(t.dim2), t.occ,
		                                                    static_cast<T *>(t.sub_min), t.last_par, t.levels, e, depth);
		PST_CUDA(cudaGetLastError());
		e -= depth;
	}
}

}  // namespace

void finish_tree_aux(TreeStorage &t, cudaStream_t s)
{
	if (t.levels < 8)  // level D-2 spans less than one 64-slot block
		return;
	const uint32_t L = t.levels - 2;
	const uint64_t nb = (1ull << L) / 64;
	const uint64_t words = (nb + 31) / 32;
	const size_t vs = value_size(t.dtype);
	const size_t par_bytes = align_up(words * 4);
	t.aux = pool_alloc(par_bytes + ((1ull << (t.levels - 1)) / 64) * vs, "search index");
	t.last_par = static_cast<uint32_t *>(t.aux);
	t.sub_min = static_cast<char *>(t.aux) + par_bytes;
	// sub_min: one value per 64-slot block of positions [64, 2^(D-1)), levels 6..D-2
	switch (t.dtype) {
	case PST_F32: sub_min_launch<float>(t, s); break;
	case PST_F64: sub_min_launch<double>(t, s); break;
	case PST_I32: sub_min_launch<int32_t>(t, s); break;
	}
}

namespace {

// Zeros for the places of a field that hold no node: place 0, and those of the last level
// without one.
template <typename T>
__global__ void k_clear_absent(T *dim1, T *dim2, T *med, uint32_t *id, const uint32_t *occ, uint64_t slots)
{
	const uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
	const uint64_t h = i == 0 ? 0 : slots / 2 + i - 1;
	if (h >= slots || ((occ[h >> 5] >> (h & 31)) & 1u))
		return;
	dim1[h] = dim2[h] = T(0);
	if (h == 0)
		med[0] = T(0);
	if (id)
		id[h] = 0;
}

template <typename T>
void clear_absent_t(const TreeStorage &t, cudaStream_t s)
{
	const uint64_t slots = 1ull << t.levels;
	k_clear_absent<T><<<(unsigned) ((slots / 2 + 1 + 255) / 256), 256, 0, s>>>(as<T>(t.dim1), as<T>(t.dim2), as<T>(t.med),
	                                                                        t.id, t.occ, slots);
	PST_CUDA(cudaGetLastError());
}

}  // namespace

void clear_absent(const TreeStorage &t, cudaStream_t s)
{
	if (!t.n)
		return;
	// the gaps behind the fields of a small tree
	const TreeLayout L = tree_layout(t.dtype, t.idtype, t.n);
	const size_t vs = value_size(t.dtype), S = size_t(1) << t.levels;
	const size_t ends[] = {L.off_dim1 + S * vs, L.off_dim2 + S * vs, L.off_med + S / 2 * vs,
	                       L.off_id + (t.id ? S * 4 : 0), L.off_occ + std::max<size_t>(S / 32, 1) * 4};
	for (size_t e : ends)
		if (e % ALIGN)
			PST_CUDA(cudaMemsetAsync(static_cast<char *>(t.mem) + e, 0, ALIGN - e % ALIGN, s));
	switch (t.dtype) {
	case PST_F32: clear_absent_t<float>(t, s); break;
	case PST_F64: clear_absent_t<double>(t, s); break;
	case PST_I32: clear_absent_t<int32_t>(t, s); break;
	}
}

void free_tree(TreeStorage &t)
{
	t.passes->wait_all();  // asynchronous passes may still read the tree
	pool_release(t.mem, t.device);
	t.mem = nullptr;
	pool_release(t.aux, t.device);
	t.aux = nullptr;
	t.last_par = nullptr;
	t.sub_min = nullptr;
}

void export_tree(const TreeStorage &t, void *dim1, void *dim2, void *med, uint32_t *ids, uint8_t *bitcodes)
{
	if (t.n == 0)
		return;
	const uint32_t D = t.levels;
	const uint64_t S = 1ull << D;  // positions 0..S-1, position 0 unused
	const size_t vs = value_size(t.dtype);
	std::vector<unsigned char> h1(S * vs), h2(S * vs), hm((S / 2) * vs);
	std::vector<uint32_t> hid(t.id ? S : 0), hocc(std::max<uint64_t>(S / 32, 1));
	PST_CUDA(cudaMemcpy(h1.data(), t.dim1, S * vs, cudaMemcpyDeviceToHost));
	PST_CUDA(cudaMemcpy(h2.data(), t.dim2, S * vs, cudaMemcpyDeviceToHost));
	PST_CUDA(cudaMemcpy(hm.data(), t.med, (S / 2) * vs, cudaMemcpyDeviceToHost));
	if (t.id)
		PST_CUDA(cudaMemcpy(hid.data(), t.id, S * 4, cudaMemcpyDeviceToHost));
	PST_CUDA(cudaMemcpy(hocc.data(), t.occ, hocc.size() * 4, cudaMemcpyDeviceToHost));
	auto occ = [&](uint64_t h) { return h < S && ((hocc[h >> 5] >> (h & 31)) & 1u); };
	unsigned char *o1 = static_cast<unsigned char *>(dim1), *o2 = static_cast<unsigned char *>(dim2),
	              *om = static_cast<unsigned char *>(med);
	for (uint64_t h = 1; h < S; h++) {
		const uint64_t slot = h - 1;
		if (!occ(h)) {
			memset(o1 + slot * vs, 0, vs);
			memset(o2 + slot * vs, 0, vs);
			memset(om + slot * vs, 0, vs);
			if (ids)
				ids[slot] = 0;
			bitcodes[slot] = 0;
			continue;
		}
		memcpy(o1 + slot * vs, &h1[h * vs], vs);
		memcpy(o2 + slot * vs, &h2[h * vs], vs);
		// last-level nodes are leaves; a leaf's median is its own dim1
		// (pst/static-pst-cpu-iter.tpp:512-517)
		memcpy(om + slot * vs, h < S / 2 ? &hm[h * vs] : &h1[h * vs], vs);
		if (ids)
			ids[slot] = t.id ? hid[h] : 0;
		bitcodes[slot] = (uint8_t) ((occ(2 * h) ? 0x2 : 0) | (occ(2 * h + 1) ? 0x1 : 0));
	}
}

}  // namespace pst
