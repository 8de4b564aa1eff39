// Streaming kernels: the interval parallel search comparator and metacell formation.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "scan_kernels.cuh"

namespace pst {

namespace {

// ---------------------------------------------------------------------------
// Interval parallel search (interval-parallel-search/interval-parallel-search.h:76-117):
// report every point with dim1 <= v <= dim2.  A warp owns 256 consecutive records;
// each load instruction reads 32 consecutive records, ranks come from ballots in
// input order, and one atomic per 2048-record tile reserves the output, so the
// results of a tile keep their input order.

constexpr int IPS_THREADS = 256;
constexpr int IPS_PER_LANE = 8;
constexpr uint64_t IPS_WARP_SPAN = 32 * IPS_PER_LANE;
constexpr uint64_t IPS_TILE = IPS_WARP_SPAN * (IPS_THREADS / 32);

// Records of 4-byte values (8 or 12 bytes) would take two or three 4-byte loads per
// lane; a whole, 16-byte aligned warp span is instead copied with 16-byte cp.async
// into shared memory (two buffers per warp: the next tile's span is in flight while
// the current one is tested and written) and the lanes pick their records there.
template <typename Pt>
constexpr bool ips_staged() { return sizeof(Pt) <= 12 && (IPS_WARP_SPAN * sizeof(Pt)) % (16 * 32) == 0; }

// 16-byte copies per lane of one staged warp span, and the dynamic shared memory of
// k_ips (two spans per warp).
template <typename Pt>
constexpr int ips_vec() { return ips_staged<Pt>() ? (int) (IPS_WARP_SPAN * sizeof(Pt) / 16 / 32) : 0; }
template <typename Pt>
constexpr size_t ips_smem() { return (size_t) 2 * (IPS_THREADS / 32) * ips_vec<Pt>() * 32 * 16; }

template <typename T, bool HAS_ID, bool POINTS>
__global__ void __launch_bounds__(IPS_THREADS) k_ips(const Point<T, HAS_ID> *__restrict__ pts, uint64_t n, T v,
                                                    void *out, uint64_t capacity, unsigned long long *counter,
                                                    bool aligned16)
{
	using Pt = Point<T, HAS_ID>;
	constexpr bool STAGED = ips_staged<Pt>();
	constexpr int VEC = ips_vec<Pt>();
	extern __shared__ __align__(16) uint4 s_span[];  // [2][IPS_THREADS / 32][VEC * 32] when STAGED
	__shared__ uint32_t s_warp[IPS_THREADS / 32 + 1];
	__shared__ unsigned long long s_base;
	const int warp = threadIdx.x >> 5;
	const uint32_t lane = lane_id();
	const uint64_t tiles = (n + IPS_TILE - 1) / IPS_TILE;
	const bool staging = STAGED && aligned16;
	// a tile's span of this warp can be staged when it is whole
	auto whole = [&](uint64_t tl) { return tl < tiles && tl * IPS_TILE + (warp + 1) * IPS_WARP_SPAN <= n; };
	auto issue = [&](uint64_t tl, int b) {
		const uint4 *src = reinterpret_cast<const uint4 *>(pts + tl * IPS_TILE + warp * IPS_WARP_SPAN);
		uint4 *dst = s_span + ((size_t) b * (IPS_THREADS / 32) + warp) * (VEC * 32);
#pragma unroll
		for (int j = 0; j < VEC; j++)
			cp_async16(dst + j * 32 + lane, src + j * 32 + lane);
	};
	int cur = 0;
	bool staged_cur = false;
	if (staging) {
		staged_cur = whole(blockIdx.x);
		if (staged_cur)
			issue(blockIdx.x, 0);
		cp_async_commit();
	}
	for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
		const uint64_t wbase = tile * IPS_TILE + warp * IPS_WARP_SPAN;
		uint32_t hit[IPS_PER_LANE];
		Pt rec[IPS_PER_LANE];
		uint32_t wcount = 0;
		bool staged_next = false;
		if (staging) {
			staged_next = whole(tile + gridDim.x);
			if (staged_next)
				issue(tile + gridDim.x, cur ^ 1);
			cp_async_commit();
			cp_async_wait_group<1>();  // this tile's span has landed
			__syncwarp();
		}
		if (staged_cur) {
			const Pt *sp = reinterpret_cast<const Pt *>(s_span + ((size_t) cur * (IPS_THREADS / 32) + warp) * (VEC * 32));
#pragma unroll
			for (int k = 0; k < IPS_PER_LANE; k++) {
				rec[k] = sp[32 * k + lane];
				const bool ok = rec[k].dim1 <= v && v <= rec[k].dim2;
				hit[k] = __ballot_sync(0xFFFFFFFFu, ok);
				wcount += __popc(hit[k]);
			}
			__syncwarp();  // the buffer is refilled for the tile after next
		} else {
#pragma unroll
			for (int k = 0; k < IPS_PER_LANE; k++) {
				const uint64_t i = wbase + 32 * k + lane;
				bool ok = false;
				if (i < n) {
					rec[k] = pts[i];
					ok = rec[k].dim1 <= v && v <= rec[k].dim2;
				}
				hit[k] = __ballot_sync(0xFFFFFFFFu, ok);
				wcount += __popc(hit[k]);
			}
		}
		if (lane == 0)
			s_warp[warp] = wcount;
		__syncthreads();
		if (threadIdx.x == 0) {
			uint32_t run = 0;
			for (int w = 0; w < IPS_THREADS / 32; w++) {
				const uint32_t c = s_warp[w];
				s_warp[w] = run;
				run += c;
			}
			s_base = run ? atomicAdd(counter, (unsigned long long) run) : 0ull;
		}
		__syncthreads();
		uint64_t o = s_base + s_warp[warp];
#pragma unroll
		for (int k = 0; k < IPS_PER_LANE; k++) {
			if ((hit[k] >> lane) & 1u) {
				const uint64_t pos = o + __popc(hit[k] & lanemask_lt());
				if (pos < capacity) {
					if constexpr (POINTS)
						static_cast<Pt *>(out)[pos] = rec[k];
					else
						static_cast<uint32_t *>(out)[pos] = rec[k].id;
				}
			}
			o += __popc(hit[k]);
		}
		__syncthreads();
		staged_cur = staged_next;
		cur ^= 1;
	}
	if (staging)
		cp_async_wait_all();  // nothing may still target this CTA's shared memory
}

// ---------------------------------------------------------------------------
// Metacell formation (helpers/isosurface-data-processing.tu:9-127, :181-212).
// Thread x of a CTA owns metacell column (mx = x, my) and walks a slab of metacells
// in z.  Vertex rows are read with consecutive threads on consecutive metacells;
// the shared boundary plane between consecutive metacells in z is reduced once and
// reused.

template <typename T>
__device__ __forceinline__ void plane_minmax(const T *__restrict__ vol, uint64_t px, uint64_t py, uint64_t z,
                                             uint32_t x0, uint32_t x1, uint32_t y0, uint32_t y1, T &lo, T &hi)
{
	const T *plane = vol + z * py * px;
	lo = hi = plane[(uint64_t) y0 * px + x0];
	for (uint32_t y = y0; y <= y1; y++) {
		const T *row = plane + (uint64_t) y * px;
		for (uint32_t x = x0; x <= x1; x++) {
			const T val = row[x];
			lo = val < lo ? val : lo;
			hi = val > hi ? val : hi;
		}
	}
}

// Minimum and maximum of the vertices [x0, x1] x [y0, y1] x [z0, z1] as k_metacells folds
// them, vertex after vertex, plane by plane, from those (lo, hi) of a fold in another order
// (a NaN if any vertex is one).  Without a NaN only the sign of a zero is open: it is that
// of the first zero among the vertices, which a field that is clipped or masked soon has.
// Nothing replaces a NaN at the first vertex.
template <typename T>
__device__ __noinline__ void metacell_fold(const T *__restrict__ vol, uint64_t px, uint64_t py, uint32_t x0,
                                           uint32_t x1, uint32_t y0, uint32_t y1, uint32_t z0, uint32_t z1, T &lo, T &hi)
{
	if (lo == lo && hi == hi) {
		for (uint32_t z = z0; z <= z1; z++)
			for (uint32_t y = y0; y <= y1; y++) {
				const T *row = vol + (z * py + y) * px;
				for (uint32_t x = x0; x <= x1; x += 4) {
					T v[4];
#pragma unroll
					for (uint32_t k = 0; k < 4; k++)
						v[k] = row[min(x + k, x1)];
#pragma unroll
					for (uint32_t k = 0; k < 4; k++)
						if (v[k] == T(0)) {
							lo = lo == T(0) ? v[k] : lo;
							hi = hi == T(0) ? v[k] : hi;
							return;
						}
				}
			}
		return;
	}
	lo = hi = vol[(z0 * py + y0) * px + x0];
	if (lo != lo)
		return;
	plane_minmax(vol, px, py, z0, x0, x1, y0, y1, lo, hi);
	for (uint32_t z = z0 + 1; z <= z1; z++) {
		T pl, ph;
		plane_minmax(vol, px, py, z, x0, x1, y0, y1, pl, ph);
		lo = pl < lo ? pl : lo;
		hi = ph > hi ? ph : hi;
	}
}

// Metacell layers [mz_begin, mz_end); `vol` holds the vertex planes from z_base on
// (the whole volume: z_base = 0; one z-slab of it: its first plane).
template <typename T, bool HAS_ID>
__global__ void k_metacells(const T *__restrict__ vol, uint32_t px, uint32_t py, uint32_t pz, uint32_t mcx,
                            uint32_t mcy, uint32_t mcz, uint32_t Mx, uint32_t My, uint32_t mz_begin, uint32_t mz_end,
                            uint32_t z_base, uint32_t mz_per_cta, Point<T, HAS_ID> *__restrict__ out)
{
	const uint32_t mx = blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t my = blockIdx.y;
	const uint32_t mz0 = mz_begin + blockIdx.z * mz_per_cta;
	const uint32_t mz1 = min(mz0 + mz_per_cta, mz_end);
	if (mx >= Mx)
		return;
	const uint32_t x0 = mx * mcx, x1 = min(x0 + mcx, px - 1);
	const uint32_t y0 = my * mcy, y1 = min(y0 + mcy, py - 1);
	T plo = T(0), phi = T(0);     // the last plane reduced
	uint32_t pz_done = 0xFFFFFFFFu;
	for (uint32_t mz = mz0; mz < mz1; mz++) {
		const uint32_t z0 = mz * mcz, z1 = min(z0 + mcz, pz - 1);
		T lo, hi;
		if (pz_done == z0) {
			lo = plo;
			hi = phi;
		} else {
			plane_minmax(vol, px, py, z0 - z_base, x0, x1, y0, y1, lo, hi);
		}
		for (uint32_t z = z0 + 1; z <= z1; z++) {
			plane_minmax(vol, px, py, z - z_base, x0, x1, y0, y1, plo, phi);
			lo = plo < lo ? plo : lo;
			hi = phi > hi ? phi : hi;
			pz_done = z;
		}
		const uint64_t id = (uint64_t) mx + ((uint64_t) my + (uint64_t) mz * My) * Mx;
		Point<T, HAS_ID> p;
		p.dim1 = lo;
		p.dim2 = hi;
		if constexpr (HAS_ID)
			p.id = (uint32_t) id;
		out[id] = p;
	}
}

// Metacells wider than one vertex, over rows of any length and alignment: a thread owns a
// vertex column (consecutive threads read consecutive vertices), folds it over the rows
// and planes of GROUP metacell rows, and only then are the columns of a metacell folded
// with one another, through shared memory.  Every vertex is loaded once per CTA, and
// what two CTAs share comes from L2; the rows of a plane are independent loads (sides of
// 1 to 8 rows are compiled in).  With a thread per metacell a row's lanes are mcx
// vertices apart and load them one by one: 509 x 381 x 263 f32 vertices took 130 us in
// 4^3 metacells, 130 in 2^3 and 465 in 8^3; by columns 66, 105 and 58 us (3.3, 2.7 and
// 3.5 TB/s).  A copy that loads the next plane's rows before it folds a plane was slower
// (97 us for 4^3: the second set of registers spills).
//
// Folding columns first takes a metacell's values in another order than vertex after
// vertex, which matters where two values compare equal and differ (-0.0 and +0.0) or
// do not compare (NaN).  Where a result could show that, metacell_fold settles it: the zero
// that comes first is looked up instead of every such metacell folded again.  Us for the same
// volume with zeros for all values above (below) a level, -0.0 ones: f32 in 4^3 metacells 143
// (174) -> 61 (125), in 2^3 234 (264) -> 96 (180), f64 in 4^3 414 (418) -> 133 (133); +0.0
// above it, f32 in 4^3 162 -> 119, in 2^3 244 -> 173.  (A thread per metacell: f32 131, f64
// 156.  A float's zeros noted as a double's are: all these 66 and 105, but fields without
// zeros 58 for 52.)
template <typename T, int MCY>  // MCY 0: any number of rows, eight at a time
struct ColumnShape {
	// metacell rows of a CTA, and the vertex rows it loads together
	static constexpr int GROUP = MCY == 0 ? 1 : MCY == 1 ? 4 : (sizeof(T) == 4 ? 8 : 4) / MCY > 1 ? (sizeof(T) == 4 ? 8 : 4) / MCY : 1;
	static constexpr int ROWS = MCY ? GROUP * MCY + 1 : 8;
};

// Threads of a CTA: a row of 512 vertices and the one past its last metacell fit.
constexpr int MC_COL_THREADS = 544;

// The folds of a column.  For floats in one instruction each: NaN if any value is one, and
// -0.0 below +0.0.
__device__ __forceinline__ float fold_min(float a, float b)
{
	float r;
	asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ float fold_max(float a, float b)
{
	float r;
	asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ int32_t fold_min(int32_t a, int32_t b) { return min(a, b); }
__device__ __forceinline__ int32_t fold_max(int32_t a, int32_t b) { return max(a, b); }
__device__ __forceinline__ double fold_min(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double fold_max(double a, double b) { return b > a ? b : a; }

// Whether the order of a fold could show in its result: values that hold a NaN, or zeros of
// both signs.  Doubles are asked a plane of a column at a time, in one comparison a value
// where none is a zero or a NaN; a float's folds tell by themselves, but for a few
// metacells: a minimum of +0.0 means that no -0.0 was there, and a maximum of -0.0 that no
// +0.0 was.
constexpr uint32_t HAS_NAN = 1, HAS_NEG_ZERO = 2, HAS_POS_ZERO = 4, HAS_ZEROS = HAS_NEG_ZERO | HAS_POS_ZERO;
template <int N>
__device__ __forceinline__ uint32_t marks_of(const double (&v)[N])
{
	bool any = false;
#pragma unroll
	for (int r = 0; r < N; r++)
		any |= !(fabs(v[r]) > 0.0);
	uint32_t marks = 0;
	if (any) {
#pragma unroll
		for (int r = 0; r < N; r++)
			marks |= v[r] != v[r] ? HAS_NAN : v[r] != 0.0 ? 0u : signbit(v[r]) ? HAS_NEG_ZERO : HAS_POS_ZERO;
	}
	return marks;
}
template <typename T, int N>
__device__ __forceinline__ uint32_t marks_of(const T (&)[N]) { return 0; }
// Whether metacell_fold has to look at a metacell with these folds, whose columns have these
// marks (a double's lo becomes a NaN where one of its vertices is one).
__device__ __forceinline__ bool order_shows(float lo, float hi, uint32_t)
{
	return lo != lo || hi != hi || (__float_as_uint(lo) == 0x80000000u && __float_as_uint(hi) != 0x80000000u) ||
	       (__float_as_uint(hi) == 0u && lo < 0.0f);
}
__device__ __forceinline__ bool order_shows(double &lo, double hi, uint32_t marks)
{
	if (marks & HAS_NAN)
		lo = nan("");
	return (marks & HAS_NAN) || (marks == HAS_ZEROS && (lo == 0.0 || hi == 0.0));
}
__device__ __forceinline__ bool order_shows(int32_t, int32_t, uint32_t) { return false; }

template <typename T, bool HAS_ID, int MCY>
__global__ void __launch_bounds__(MC_COL_THREADS, 2) k_metacells_cols(
    const T *__restrict__ vol, uint32_t px, uint32_t py, uint32_t pz, uint32_t mcx, uint32_t mcy, uint32_t mcz,
    uint32_t span, uint32_t Mx, uint32_t My, uint32_t mz_begin, uint32_t mz_end, uint32_t z_base,
    uint32_t mz_per_cta, Point<T, HAS_ID> *__restrict__ out)
{
	constexpr int GROUP = ColumnShape<T, MCY>::GROUP, ROWS = ColumnShape<T, MCY>::ROWS;
	__shared__ T s_lo[GROUP][MC_COL_THREADS], s_hi[GROUP][MC_COL_THREADS];
	constexpr bool MARKS = std::is_same<T, double>::value;
	__shared__ uint8_t s_mark[MARKS ? MC_COL_THREADS : 1];
	__shared__ Point<T, HAS_ID> s_out[MC_COL_THREADS];
	const uint32_t chunks = (span + 31) / 32;
	const uint32_t mx0 = blockIdx.x * span, my0 = blockIdx.y * GROUP;  // span: metacells of the CTA along x
	const uint32_t y0 = my0 * mcy;
	const uint32_t mz0 = mz_begin + blockIdx.z * mz_per_cta, mz1 = min(mz0 + mz_per_cta, mz_end);
	// the column's vertices, as offsets from the plane's row y0 (rows and columns past the
	// volume repeat its last one, as the last vertices of a cut metacell do)
	const uint32_t dx = min(mx0 * mcx + threadIdx.x, px - 1);
	const uint32_t row_last = min(GROUP * mcy, py - 1 - y0);
	uint32_t off[ROWS];
#pragma unroll
	for (int r = 0; r < ROWS; r++)
		off[r] = min((uint32_t) r, row_last) * px + dx;
	T lo[GROUP], hi[GROUP], plo[GROUP], phi[GROUP];
	uint32_t mark = 0, pmark = 0;
	// plane z's folds into plo, phi, pmark
	auto plane = [&](uint32_t z) {
		const T *p = vol + ((uint64_t) (z - z_base) * py + y0) * px;
		T v[ROWS];
#pragma unroll
		for (int r = 0; r < ROWS; r++)
			v[r] = p[off[r]];
		pmark = marks_of(v);
#pragma unroll
		for (int g = 0; g < GROUP; g++) {
			plo[g] = phi[g] = v[g * MCY];
#pragma unroll
			for (int k = 1; k < (MCY ? MCY + 1 : ROWS); k++) {
				plo[g] = fold_min(plo[g], v[g * MCY + k]);
				phi[g] = fold_max(phi[g], v[g * MCY + k]);
			}
		}
		if constexpr (MCY == 0) {
			for (uint32_t r0 = ROWS; r0 <= row_last; r0 += ROWS) {
#pragma unroll
				for (int r = 0; r < ROWS; r++)
					v[r] = p[min(r0 + r, row_last) * px + dx];
				pmark |= marks_of(v);
#pragma unroll
				for (int r = 0; r < ROWS; r++) {
					plo[0] = fold_min(plo[0], v[r]);
					phi[0] = fold_max(phi[0], v[r]);
				}
			}
		}
	};
	plane(mz0 * mcz);
	for (uint32_t mz = mz0; mz < mz1; mz++) {
		const uint32_t z0 = mz * mcz, z1 = min(z0 + mcz, pz - 1);
		mark = pmark;
#pragma unroll
		for (int g = 0; g < GROUP; g++) {
			lo[g] = plo[g];  // the plane shared with the layer below
			hi[g] = phi[g];
		}
#pragma unroll(sizeof(T) == 4 ? 2 : 1)
		for (uint32_t z = z0 + 1; z <= z1; z++) {
			plane(z);
			mark |= pmark;
#pragma unroll
			for (int g = 0; g < GROUP; g++) {
				lo[g] = fold_min(lo[g], plo[g]);
				hi[g] = fold_max(hi[g], phi[g]);
			}
		}
#pragma unroll
		for (int g = 0; g < GROUP; g++) {
			s_lo[g][threadIdx.x] = lo[g];
			s_hi[g][threadIdx.x] = hi[g];
		}
		if constexpr (MARKS)
			s_mark[threadIdx.x] = (uint8_t) mark;
		__syncthreads();
		// a warp takes 32 consecutive metacells of a row, whose records leave as consecutive
		// words
		for (uint32_t t = threadIdx.x >> 5; t < GROUP * chunks; t += blockDim.x >> 5) {
			const uint32_t g = t / chunks, m0 = (t - g * chunks) * 32, c = (m0 + lane_id()) * mcx;
			const uint32_t mx = mx0 + m0 + lane_id(), my = my0 + g;
			if (my >= My || mx0 + m0 >= Mx)
				continue;
			const uint32_t count = min(min(span - m0, Mx - (mx0 + m0)), 32u);
			const uint64_t id0 = (uint64_t) (mx0 + m0) + ((uint64_t) my + (uint64_t) mz * My) * Mx;
			if (lane_id() < count) {
				T l = s_lo[g][c], h = s_hi[g][c];
				uint32_t m = MARKS ? s_mark[c] : 0u;
				auto next = [&](uint32_t k) {
					l = fold_min(l, s_lo[g][c + k]);
					h = fold_max(h, s_hi[g][c + k]);
					if constexpr (MARKS)
						m |= s_mark[c + k];
				};
				if (MCY && mcx == (uint32_t) MCY) {
#pragma unroll
					for (uint32_t k = 1; k <= (uint32_t) MCY; k++)
						next(k);
				} else {
					for (uint32_t k = 1; k <= mcx; k++)
						next(k);
				}
				if (order_shows(l, h, m))
					metacell_fold(vol, px, py, mx * mcx, min(mx * mcx + mcx, px - 1), my * mcy,
					              min(my * mcy + mcy, py - 1), z0 - z_base, z1 - z_base, l, h);
				Point<T, HAS_ID> &p = s_out[threadIdx.x];
				p.dim1 = l;
				p.dim2 = h;
				if constexpr (HAS_ID && sizeof(T) == 8)
					*reinterpret_cast<unsigned long long *>(&p.id) = (uint32_t) id0 + lane_id();  // with its padding
				else if constexpr (HAS_ID)
					p.id = (uint32_t) id0 + lane_id();
			}
			__syncwarp();
			using W = typename std::conditional<sizeof(T) == 8, unsigned long long, uint32_t>::type;
			const W *src = reinterpret_cast<const W *>(s_out + (threadIdx.x & ~31u));
			W *dst = reinterpret_cast<W *>(out + id0);
			for (uint32_t i = lane_id(); i < count * (uint32_t) (sizeof(Point<T, HAS_ID>) / sizeof(W)); i += 32)
				dst[i] = src[i];
			__syncwarp();  // the warp's records are rewritten by its next 32
		}
		__syncthreads();  // the columns are rewritten by the next layer
	}
}

// The common layout: metacells 4 vertices wide over 4-byte values, rows a multiple of
// 4 vertices long, the volume 16-byte aligned.  A metacell's 4 low vertices of a row
// are one aligned 16-byte load; its fifth (the next metacell's first) comes from the
// next lane, or from memory for a warp's last metacell.  Same walk as k_metacells.  A
// load brings a whole metacell row, which columns (k_metacells_cols) take four for: 123
// against 137 us for 512^3 f32 vertices in 4^3 metacells.
template <typename T>
struct Quad;
template <>
struct Quad<float> {
	using V = float4;
};
template <>
struct Quad<int32_t> {
	using V = int4;
};

template <typename T, bool HAS_ID>
__global__ void k_metacells4(const T *__restrict__ vol, uint32_t px, uint32_t py, uint32_t pz, uint32_t mcy,
                             uint32_t mcz, uint32_t Mx, uint32_t My, uint32_t mz_begin, uint32_t mz_end,
                             uint32_t z_base, uint32_t mz_per_cta, Point<T, HAS_ID> *__restrict__ out)
{
	using V = typename Quad<T>::V;
	const uint32_t mx = blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t lane = lane_id();
	const bool active = mx < Mx;  // inactive lanes still take part in the shuffles
	const uint32_t my = blockIdx.y;
	const uint32_t mz0 = mz_begin + blockIdx.z * mz_per_cta;
	const uint32_t mz1 = min(mz0 + mz_per_cta, mz_end);
	const uint32_t x0 = 4 * mx;
	const bool has5 = active && x0 + 4 <= px - 1;         // the metacell has a fifth vertex column
	const bool from_next = lane < 31 && mx + 1 < Mx;     // ... and the next lane holds it
	const uint32_t y0 = my * mcy, y1 = min(y0 + mcy, py - 1);
	auto plane = [&](uint32_t z, T &lo, T &hi) {
		const T *pl = vol + (uint64_t) (z - z_base) * py * px;
		for (uint32_t y = y0; y <= y1; y++) {
			const T *row = pl + (uint64_t) y * px;
			const V a = active ? *reinterpret_cast<const V *>(row + x0) : V{};
			const T nx = __shfl_down_sync(0xFFFFFFFFu, a.x, 1);
			const T e = from_next ? nx : has5 ? row[x0 + 4] : a.x;
			// folds in row-major order that keep the first of equal values (as
			// k_metacells does), so -0.0 and +0.0 come out as they do there
			const T r[5] = {a.x, a.y, a.z, a.w, e};
			T l = r[0], h = r[0];
#pragma unroll
			for (int k = 1; k < 5; k++) {
				l = r[k] < l ? r[k] : l;
				h = r[k] > h ? r[k] : h;
			}
			if (y == y0) {
				lo = l;
				hi = h;
			} else {
				lo = l < lo ? l : lo;
				hi = h > hi ? h : hi;
			}
		}
	};
	T plo = T(0), phi = T(0);  // the last plane reduced
	uint32_t pz_done = 0xFFFFFFFFu;
	for (uint32_t mz = mz0; mz < mz1; mz++) {
		const uint32_t z0 = mz * mcz, z1 = min(z0 + mcz, pz - 1);
		T lo, hi;
		if (pz_done == z0) {
			lo = plo;
			hi = phi;
		} else {
			plane(z0, lo, hi);
		}
		for (uint32_t z = z0 + 1; z <= z1; z++) {
			plane(z, plo, phi);
			lo = plo < lo ? plo : lo;
			hi = phi > hi ? phi : hi;
			pz_done = z;
		}
		if (active) {
			const uint64_t id = (uint64_t) mx + ((uint64_t) my + (uint64_t) mz * My) * Mx;
			Point<T, HAS_ID> p;
			p.dim1 = lo;
			p.dim2 = hi;
			if constexpr (HAS_ID)
				p.id = (uint32_t) id;
			out[id] = p;
		}
	}
}

template <typename T, bool HAS_ID, bool POINTS>
void ips_launch(const void *pts, uint64_t n, T v, void *out, uint64_t cap, unsigned long long *counter,
                uint32_t blocks, cudaStream_t s)
{
	const uint64_t tiles = (n + IPS_TILE - 1) / IPS_TILE;
	uint64_t g = blocks ? blocks : std::min<uint64_t>(tiles, (uint64_t) device_info().sms * 8);
	g = std::max<uint64_t>(g, 1);
	const bool aligned16 = (reinterpret_cast<uintptr_t>(pts) & 15u) == 0;
	constexpr size_t smem = ips_smem<Point<T, HAS_ID>>();
	if (smem > 0) {
		// above the default 48 KB with the static part: opt in once per device
		static std::mutex mu;
		static bool done[64] = {};
		const int dev = device_info().device;
		std::lock_guard<std::mutex> lk(mu);
		if (dev >= 0 && dev < 64 && !done[dev]) {
			PST_CUDA(cudaFuncSetAttribute(k_ips<T, HAS_ID, POINTS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                              (int) smem));
			done[dev] = true;
		}
	}
	k_ips<T, HAS_ID, POINTS><<<(unsigned) g, IPS_THREADS, smem, s>>>(static_cast<const Point<T, HAS_ID> *>(pts), n, v,
	                                                                  out, cap, counter, aligned16);
	PST_CUDA(cudaGetLastError());
}

template <typename T>
void ips_dispatch(pst_idtype it, pst_ret ret, const void *pts, uint64_t n, T v, void *out, uint64_t cap,
                  unsigned long long *counter, uint32_t blocks, cudaStream_t s)
{
	if (ret == PST_RET_IDS) {
		if (it != PST_ID_U32)
			fail(PST_ERR_UNSUPPORTED, "id-less points can only be returned as points");
		ips_launch<T, true, false>(pts, n, v, out, cap, counter, blocks, s);
	} else if (it == PST_ID_U32) {
		ips_launch<T, true, true>(pts, n, v, out, cap, counter, blocks, s);
	} else {
		ips_launch<T, false, true>(pts, n, v, out, cap, counter, blocks, s);
	}
}

// Launch shape of k_metacells_cols: rows of up to 512 vertices a CTA, and in z as many
// layers a CTA (of at least 16 vertices in all) as leave the device two CTAs an SM.
template <typename T, bool HAS_ID, int MCY>
void metacell_cols_launch(const T *vol, const uint32_t P[3], const uint32_t mc[3], const uint32_t M[3],
                          uint32_t mz_begin, uint32_t mz_end, Point<T, HAS_ID> *out, cudaStream_t s)
{
	constexpr uint32_t GROUP = ColumnShape<T, MCY>::GROUP;
	// as few CTAs along x as hold the row, each with an equal share of it
	const uint32_t layers = mz_end - mz_begin, most = (MC_COL_THREADS - 1) / mc[0];
	const uint32_t gx = (M[0] + most - 1) / most, span = (M[0] + gx - 1) / gx;
	const uint32_t threads = (span * mc[0] + 1 + 31) / 32 * 32;
	const uint32_t gy = (M[1] + GROUP - 1) / GROUP;
	uint32_t mzp = std::max(1u, 16 / mc[2]);
	while (mzp > 1 && (uint64_t) gx * gy * ((layers + mzp - 1) / mzp) < (uint64_t) device_info().sms * 2)
		mzp /= 2;
	mzp = std::max(mzp, (layers + 65534) / 65535);
	const dim3 grid(gx, gy, (layers + mzp - 1) / mzp);
	k_metacells_cols<T, HAS_ID, MCY><<<grid, threads, 0, s>>>(vol, P[0], P[1], P[2], mc[0], mc[1], mc[2], span,
	                                                         M[0], M[1], mz_begin, mz_end, mz_begin * mc[2], mzp, out);
}

// Whether a column holds too few vertices of a metacell to pay for its way through shared
// memory and the two barriers of a layer, on a device that `threads`, one per metacell
// column of 8 layers, leave no room to hide the loads of a thread per metacell.  By
// metacells and by columns, 509 x 381 x 263 vertices: f32 in 4 x 1 x 1 119 and 262 us, in
// 4 x 4 x 1 109 and 133, in 4 x 1 x 2 108 and 142, in 4 x 2 x 2 119 and 105; f64 in 2 x 2 x 2
// 157 and 192, in 4 x 2 x 3 121 and 145, in 8 x 2 x 2 296 and 270, in 3 x 3 x 3 131 and 142
// (but 195 and 173 for 1031 x 300 x 200).  201 x 181 x 163, f32 in 2 x 4 x 1: 38 and 27.
template <typename T>
bool metacell_is_flat(const uint32_t mc[3], uint64_t threads)
{
	const uint64_t full = (uint64_t) device_info().sms * 2048;
	if (mc[2] == 1)
		return mc[1] <= 5 && threads * 5 >= full * 2;
	if (sizeof(T) == 8)
		return mc[0] <= 5 && (uint64_t) mc[1] * mc[2] <= 6 && threads * 5 >= full * 3;
	return mc[0] <= 8 && (uint64_t) mc[1] * mc[2] <= 2 && threads >= full;
}

template <typename T, bool HAS_ID>
void metacell_launch(const void *vol, const uint32_t P[3], const uint32_t mc[3], const uint32_t M[3],
                     uint32_t mz_begin, uint32_t mz_end, void *out, cudaStream_t s)
{
	if (mz_end <= mz_begin)
		return;
	const uint32_t layers = mz_end - mz_begin;
	if (M[1] > 65535 || (layers + 7) / 8 > 65535)
		fail(PST_ERR_INVALID, "metacell grid too large");
	const T *v = static_cast<const T *>(vol);
	Point<T, HAS_ID> *o = static_cast<Point<T, HAS_ID> *>(out);
	const uint32_t threads = M[0] >= 256 ? 256 : ((M[0] + 31) / 32) * 32;
	if (mc[0] == 4 && sizeof(T) == 4 && P[0] % 4 == 0 && (reinterpret_cast<uintptr_t>(vol) & 15u) == 0) {
		if constexpr (sizeof(T) == 4) {
			// fewer layers a CTA while the device has room for more threads: a layer's planes
			// are one chain of loads (128^3 vertices: 65 us with 8 layers a CTA, 16 with one;
			// 512^3: 129 us with 8, 123 with 2 or 4), but no fewer than 8 planes, as CTAs share one
			// (512 x 512 x 256 in 4 x 1 x 1: 123 us with 4 layers a CTA, 113 with 8)
			const uint32_t gx = (M[0] + threads - 1) / threads;
			uint32_t mzp = std::max(4u, 8 / mc[2]);
			while (mzp > 1 && (uint64_t) gx * threads * M[1] * ((layers + mzp - 1) / mzp) <
			                      (uint64_t) device_info().sms * 2048)
				mzp /= 2;
			mzp = std::max(mzp, (layers + 65534) / 65535);
			const dim3 grid(gx, M[1], (layers + mzp - 1) / mzp);
			k_metacells4<T, HAS_ID><<<grid, threads, 0, s>>>(v, P[0], P[1], P[2], mc[1], mc[2], M[0], M[1], mz_begin,
			                                                 mz_end, mz_begin * mc[2], mzp, o);
		}
	} else if (mc[0] == 1 || mc[0] >= (uint32_t) MC_COL_THREADS ||
	           (uint64_t) P[0] * std::min(P[1], 2 * mc[1]) >= (1ull << 30) ||
	           metacell_is_flat<T>(mc, (uint64_t) (M[0] + threads - 1) / threads * threads * M[1] * ((layers + 7) / 8))) {
		// one vertex wide (consecutive threads are consecutive vertices already: 970 us for
		// 512^3 f32 voxels, 1090 by columns), wider than a CTA of columns, rows too long
		// for its 32-bit offsets, or few vertices to a column: a thread per metacell
		const dim3 grid((M[0] + threads - 1) / threads, M[1], (layers + 7) / 8);
		k_metacells<T, HAS_ID><<<grid, threads, 0, s>>>(v, P[0], P[1], P[2], mc[0], mc[1], mc[2], M[0], M[1], mz_begin,
		                                                mz_end, mz_begin * mc[2], 8, o);
	} else {
		switch (mc[1]) {
		case 1: metacell_cols_launch<T, HAS_ID, 1>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 2: metacell_cols_launch<T, HAS_ID, 2>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 3: metacell_cols_launch<T, HAS_ID, 3>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 4: metacell_cols_launch<T, HAS_ID, 4>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 5: metacell_cols_launch<T, HAS_ID, 5>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 6: metacell_cols_launch<T, HAS_ID, 6>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 7: metacell_cols_launch<T, HAS_ID, 7>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		case 8: metacell_cols_launch<T, HAS_ID, 8>(v, P, mc, M, mz_begin, mz_end, o, s); break;
		default: metacell_cols_launch<T, HAS_ID, 0>(v, P, mc, M, mz_begin, mz_end, o, s);
		}
	}
	PST_CUDA(cudaGetLastError());
}

}  // namespace

void ips_run(pst_dtype dt, pst_idtype it, pst_ret ret, const void *pts, uint64_t n, pst_value v, void *out,
             uint64_t cap, unsigned long long *counter_d, uint32_t blocks, cudaStream_t s)
{
	switch (dt) {
	case PST_F32: ips_dispatch<float>(it, ret, pts, n, v.f32, out, cap, counter_d, blocks, s); break;
	case PST_F64: ips_dispatch<double>(it, ret, pts, n, v.f64, out, cap, counter_d, blocks, s); break;
	case PST_I32: ips_dispatch<int32_t>(it, ret, pts, n, v.i32, out, cap, counter_d, blocks, s); break;
	default: fail(PST_ERR_INVALID, "bad dtype");
	}
}

void metacells_run_layers(pst_dtype dt, pst_idtype it, const void *vol, const uint32_t P[3], const uint32_t mc[3],
                          const uint32_t M[3], uint32_t mz_begin, uint32_t mz_end, void *out, cudaStream_t s)
{
	const bool id = it == PST_ID_U32;
	const uint32_t b = mz_begin, e = mz_end;
	switch (dt) {
	case PST_F32: id ? metacell_launch<float, true>(vol, P, mc, M, b, e, out, s) : metacell_launch<float, false>(vol, P, mc, M, b, e, out, s); break;
	case PST_F64: id ? metacell_launch<double, true>(vol, P, mc, M, b, e, out, s) : metacell_launch<double, false>(vol, P, mc, M, b, e, out, s); break;
	case PST_I32: id ? metacell_launch<int32_t, true>(vol, P, mc, M, b, e, out, s) : metacell_launch<int32_t, false>(vol, P, mc, M, b, e, out, s); break;
	default: fail(PST_ERR_INVALID, "bad dtype");
	}
}

void metacells_run(pst_dtype dt, pst_idtype it, const void *vol, const uint32_t P[3], const uint32_t mc[3],
                   const uint32_t M[3], void *out, cudaStream_t s)
{
	metacells_run_layers(dt, it, vol, P, mc, M, 0, M[2], out, s);
}

}  // namespace pst
