// Searches of the static priority search tree: one query or a batch of mixed
// 3-sided / 2-sided-left / 2-sided-right queries, in one level-synchronous pass.
//
// The reference walks the tree with one thread block per query, handing subtrees
// to idle threads through shared memory and to child grids when none are idle
// (pst/static-pst-gpu-search-functions.tu:12-722, pst/static-pst-gpu.tu:819-1148).
// Here every query of a batch advances one tree level per kernel (k_bfs_level):
//   - "path" tasks follow the O(log n) boundary nodes of a query with the
//     reference's delegation rules (do3SidedSearchDelegation, doLeftSearchDelegation,
//     doRightSearchDelegation: pst/static-pst-cpu-iter.tpp:602-714);
//   - every subtree the reference would "report above" is scanned by level.  In a
//     max-heap on dim2 a node of such a subtree is reported exactly when its own
//     dim2 passes (its ancestors' dim2 are at least as large), so the work unit is a
//     block: 64 consecutive slots of one level, tested by one warp with coalesced
//     loads.  The frontier is kept as "alive records" only — (block, query, mask of
//     reported slots) — and the next level expands each record into its two child
//     blocks (spread16), masked by occupancy before anything is loaded.  Every
//     level but the last is full (a level-d node holds at least
//     floor((n + 1) / 2^d) - 1 >= 1 points for d <= D - 2), so occupancy is read
//     only for children on the last level.  A block whose whole subtree lies at
//     or above the query's min2 (TreeDev::sub_min) hands its descendants on
//     without any dim2 test (RECORD_WHOLE).
// Small batches start with one CTA that walks the upper levels with its frontier
// in shared memory (k_bfs_cta).  A count of every query falls out of the pass; an
// exclusive scan gives each query's exact output offset, and a flat emit kernel
// writes ids (or points) from the alive records.
#include <algorithm>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "scan_sort.cuh"
#include "search.cuh"

namespace pst {

namespace {

constexpr uint32_t MODE_THREE = 3, MODE_LEFT = 1, MODE_RIGHT = 2;
constexpr uint32_t FULL = 0xFFFFFFFFu;


template <typename T>
struct QDev {
	const uint32_t *kind;
	const T *min1;
	const T *max1;
	const T *min2;
};

// The same arrays, written once per pass from the caller's pst_query records.
template <typename T>
struct QOut {
	uint32_t *kind;
	T *min1;
	T *max1;
	T *min2;
};

// Alive records cover a "block" of 64 consecutive slots of one level (two
// 128-byte rows of a 4-byte field): (block base position, query, mask of reported
// slots, low and high word).  Block bases are multiples of 64; bit 0 of the first
// word (RECORD_WHOLE) marks a block below which every descendant of the reported
// slots is reported (its dim2 need no test).
constexpr uint32_t RECORD_WHOLE = 1u;

struct WorkDev {
	uint4 *rec;            // alive records of every level, level regions in order
	uint64_t rec_cap;
	uint4 *path0, *path1;  // boundary-path tasks (position, query, mode), double-buffered by level parity
	uint4 *seed0, *seed1;  // report-above seeds (chunk base, query, candidate mask), idem
	uint32_t path_cap;     // entries of each path / seed buffer (2 per query)
	uint4 *ro;             // reported boundary nodes as one-bit block records (never expanded)
	uint32_t ro_cap;
	uint64_t *counts;
	uint64_t *cursor;
	const uint64_t *offsets;
	BatchCtl *ctl;
};

// The block record of a 32-slot chunk (base pos32, a multiple of 32) and its mask.
__device__ __forceinline__ uint4 block_record(uint32_t pos32, uint32_t q, uint32_t bits32)
{
	const bool upper = (pos32 & 32u) != 0;
	return make_uint4(pos32 & ~63u, q, upper ? 0u : bits32, upper ? bits32 : 0u);
}

// What a query does at a node of its boundary path (the reference's delegation): report it
// (rep), go on to a child with a mode (pl, pr; 0 = no), report a child's subtree from above
// (rl, rr).  v1, v2, m: the node's values and median; hl, hr: whether it has the children.
template <typename T>
__device__ __forceinline__ void path_rules(uint32_t kind, uint32_t mode, T min1, T max1, T min2, T v1, T v2, T m, bool hl,
                                           bool hr, bool &rep, uint32_t &pl, uint32_t &pr, bool &rl, bool &rr)
{
	if (min2 <= v2) {
		rep = kind == PST_Q_THREE ? (min1 <= v1 && v1 <= max1) : kind == PST_Q_LEFT ? (v1 <= max1) : (v1 >= min1);
		if (mode == MODE_THREE) {
			if (min1 <= m && m <= max1) {
				pl = hl ? MODE_RIGHT : 0;
				pr = hr ? MODE_LEFT : 0;
			} else if (max1 < m && hl) {
				pl = MODE_THREE;
			} else if (m < min1 && hr) {
				pr = MODE_THREE;
			}
		} else if (mode == MODE_LEFT) {
			if (m <= max1) {
				rl = hl;
				pr = hr ? MODE_LEFT : 0;
			} else if (hl) {
				pl = MODE_LEFT;
			}
		} else {
			if (m >= min1) {
				pl = hl ? MODE_RIGHT : 0;
				rr = hr;
			} else if (hr) {
				pr = MODE_RIGHT;
			}
		}
	}
}

template <typename T>
__device__ __forceinline__ void path_step(const TreeDev<T> &t, const QDev<T> &qd, const WorkDev &w, uint32_t d,
                                          uint4 task, bool valid)
{
	const uint32_t lane = lane_id();
	const uint32_t h = task.x, q = task.y, mode = task.z;
	const uint32_t l = 2 * h, r = 2 * h + 1;
	const bool inner = d + 1 < t.levels;  // the node has a median and may have children
	bool rep = false;
	uint32_t pl = 0, pr = 0;      // continue as a path task with this mode (0 = no)
	bool rl = false, rr = false;  // report-above subtree
	if (valid) {
		// every value the step may use is loaded at once: one round trip, not a chain.
		// Every level but the last is full, so only children on the last level need
		// their occupancy read.
		const T min2 = qd.min2[q];
		const T v2 = t.dim2[h];
		const uint32_t kind = qd.kind[q];
		const T min1 = qd.min1[q], max1 = qd.max1[q];
		const T v1 = t.dim1[h];
		const uint32_t ow = !inner ? 0u : d + 2 < t.levels ? FULL : t.occ[l >> 5];
		const T m = inner ? t.med[h] : T(0);
		path_rules<T>(kind, mode, min1, max1, min2, v1, v2, m, (ow >> (l & 31)) & 1u, (ow >> (r & 31)) & 1u, rep, pl, pr,
		              rl, rr);
	}
	// The warp's reported nodes, next-level paths and seeds each take one reservation,
	// and lane 0 issues the three together.  At most two boundary paths per query and
	// level, each leaving at most one seed, so path_cap = 2 * max_q holds every list.
	const bool seed = rl || rr;
	const uint32_t repm = __ballot_sync(FULL, rep);
	const uint32_t seedm = __ballot_sync(FULL, seed);
	const uint32_t npl = (pl ? 1u : 0u) + (pr ? 1u : 0u);
	const uint32_t inc = warp_incl_scan(npl);
	const uint32_t tot = __shfl_sync(FULL, inc, 31);
	uint32_t b_rep = 0, b_path = 0, b_seed = 0;
	if (lane == 0) {
		if (repm)
			b_rep = atomicAdd(&w.ctl->rec_cnt, (uint32_t) __popc(repm));
		if (tot)
			b_path = atomicAdd(&w.ctl->path_cnt[d + 1], tot);
		if (seedm)
			b_seed = atomicAdd(&w.ctl->seed_cnt[d + 1], (uint32_t) __popc(seedm));
	}
	b_rep = __shfl_sync(FULL, b_rep, 0);
	b_path = __shfl_sync(FULL, b_path, 0);
	b_seed = __shfl_sync(FULL, b_seed, 0);
	if (rep) {
		const uint32_t i = b_rep + __popc(repm & lanemask_lt());
		if (i < w.ro_cap)
			w.ro[i] = block_record(h & ~31u, q, 1u << (h & 31));
		else
			atomicOr(&w.ctl->flags, BATCH_FLAG_INTERNAL);
		atomicAdd((unsigned long long *) &w.counts[q], 1ull);
	}
	if (npl) {
		uint32_t i = b_path + inc - npl;
		uint4 *pout = ((d + 1) & 1) ? w.path1 : w.path0;
		if (pl) {
			if (i < w.path_cap)
				pout[i] = make_uint4(l, q, pl, 0);
			else
				atomicOr(&w.ctl->flags, BATCH_FLAG_INTERNAL);
			i++;
		}
		if (pr) {
			if (i < w.path_cap)
				pout[i] = make_uint4(r, q, pr, 0);
			else
				atomicOr(&w.ctl->flags, BATCH_FLAG_INTERNAL);
		}
	}
	if (seed) {
		// l and r share a chunk
		const uint32_t bits = (rl ? 1u << (l & 31) : 0u) | (rr ? 1u << (r & 31) : 0u);
		uint4 *sout = ((d + 1) & 1) ? w.seed1 : w.seed0;
		const uint32_t i = b_seed + __popc(seedm & lanemask_lt());
		if (i < w.path_cap)
			sout[i] = make_uint4(l & ~31u, q, bits, 0u);
		else
			atomicOr(&w.ctl->flags, BATCH_FLAG_INTERNAL);
	}
}

// Appends each lane's non-empty records (at most K) to the level region (one atomic
// per warp).
template <int K>
__device__ __forceinline__ void append_blocks(const WorkDev &w, uint32_t lvl, uint64_t region_base, const uint4 (&r)[K])
{
	const uint32_t lane = lane_id();
	uint32_t nrec = 0;
#pragma unroll
	for (int k = 0; k < K; k++)
		nrec += (r[k].z | r[k].w) ? 1u : 0u;
	const uint32_t inc = warp_incl_scan(nrec);
	const uint32_t tot = __shfl_sync(FULL, inc, 31);
	if (!tot)
		return;
	uint64_t slot0 = 0;
	if (lane == 31) {
		const uint32_t off = atomicAdd(&w.ctl->lvl_cnt[lvl], tot);
		slot0 = region_base + off;
		if (slot0 + tot > w.rec_cap) {
			atomicMax((unsigned long long *) &w.ctl->need_tasks, (unsigned long long) (slot0 + tot));
			atomicOr(&w.ctl->flags, BATCH_FLAG_TASK_OVERFLOW);
			slot0 = ~0ull;
		}
	}
	slot0 = __shfl_sync(FULL, slot0, 31);
	if (slot0 == ~0ull)
		return;
	uint64_t s = slot0 + inc - nrec;
#pragma unroll
	for (int k = 0; k < K; k++)
		if (r[k].z | r[k].w)
			w.rec[s++] = r[k];
}

// Adds the lanes' point counts to their queries' counts (one atomic per run of
// equal query ids).
__device__ __forceinline__ void add_counts(const WorkDev &w, uint32_t q, uint32_t pts, bool valid)
{
	bool last;
	const uint64_t run = warp_run_sum(valid ? q : 0xFFFFFFFFu, pts, &last);
	if (valid && last && run)
		atomicAdd((unsigned long long *) &w.counts[q], (unsigned long long) run);
}

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
	using V = float4;
};
template <>
struct Vec4<int32_t> {
	using V = int4;
};

// Four consecutive values from a 16-byte aligned address (two loads for doubles).
template <typename T>
__device__ __forceinline__ void load_quad(const T *__restrict__ p, T (&v)[4])
{
	if constexpr (sizeof(T) == 4) {
		using V = typename Vec4<T>::V;
		const V x = *reinterpret_cast<const V *>(p);
		v[0] = x.x;
		v[1] = x.y;
		v[2] = x.z;
		v[3] = x.w;
	} else {
		const double2 a = reinterpret_cast<const double2 *>(p)[0];
		const double2 b = reinterpret_cast<const double2 *>(p)[1];
		v[0] = a.x;
		v[1] = a.y;
		v[2] = b.x;
		v[3] = b.y;
	}
}

// Per-warp shared staging of the 32 records a warp holds: the records, the
// candidate masks of their four child rows (parents' bits spread to their children,
// ANDed with the occupancy), their queries' min2, the child rows found, and the
// list of records that have any candidate at all.
template <typename T>
struct WarpStage {
	uint4 rec[32];
	uint4 cand[32];
	uint4 rows[32];
	T m2[32];
	uint32_t live[32];
};

// Expands the records held by the warp (lane k owns record `mine`; the valid lanes
// are a prefix) into their child records.  Each lane first stages its record's
// candidate child slots (`full`: the children's level is full, so the candidates
// are the spread parent bits with no occupancy read); records without any (all
// children absent, e.g. above a sparse last level) cost nothing more.  Then the whole warp takes the live records
// U at a time: lane l tests the child slots [2b + 4l, 2b + 4l + 4) with one 16-byte
// load (two for doubles), issued only where it has candidates; each 8-lane group
// ORs its nibbles into one 32-slot child row, and the owner reads the four rows as
// its two child records (blocks 2b and 2b + 64).
template <typename T, bool LAST>
__device__ __forceinline__ void expand_records(const TreeDev<T> &t, const T *__restrict__ min2s, const uint4 &mine,
                                               bool valid, bool full, WarpStage<T> &st, uint4 (&child)[2],
                                               uint32_t &pts)
{
	constexpr int U = sizeof(T) == 4 ? 4 : 2;  // records in flight
	const uint32_t lane = lane_id();
	const uint32_t r = lane >> 3, qd = lane & 7;
	const uint32_t base = mine.x & ~63u;  // bit 0 of a record's block: RECORD_WHOLE
	// the record's min2 stays in its owner lane's register (its load overlaps the
	// staging below) and is broadcast by a shuffle where it is compared
	const T m2_own = valid ? min2s[mine.y] : T(0);
	// A block whose every descendant has dim2 >= min2 (TreeDev::sub_min): all
	// descendants of its reported slots are reported, with no test; its child
	// records carry RECORD_WHOLE, so theirs need no look-up either.
	bool whole = (mine.x & RECORD_WHOLE) != 0;
	if (valid && !whole && t.sub_min && base >= 64)
		whole = m2_own <= t.sub_min[base >> 6];
	uint4 cand = make_uint4(0, 0, 0, 0);
	bool has_children = valid;
	if (LAST && valid) {
		// expanding into the last level: most blocks of a sparse last level have no
		// children, which one bit per parent block tells before any occupancy read
		const uint32_t j = (base - (1u << (t.levels - 2))) >> 6;
		has_children = (t.last_par[j >> 5] >> (j & 31)) & 1u;
	}
	if (has_children) {
		// children on a full level (every level but the last) need no occupancy read
		const uint4 occ = full ? make_uint4(FULL, FULL, FULL, FULL)
		                       : *reinterpret_cast<const uint4 *>(t.occ + ((2 * base) >> 5));
		cand = make_uint4(spread16(mine.z) & occ.x, spread16(mine.z >> 16) & occ.y, spread16(mine.w) & occ.z,
		                  spread16(mine.w >> 16) & occ.w);
	}
	const bool live = !whole && (cand.x | cand.y | cand.z | cand.w) != 0;
	const uint32_t lm = __ballot_sync(FULL, live);
	const int nlive = __popc(lm);
	if (live) {
		st.rec[lane] = mine;
		st.cand[lane] = cand;
		st.live[__popc(lm & lanemask_lt())] = lane;
	}
	__syncwarp();
	const uint32_t *candw = reinterpret_cast<const uint32_t *>(st.cand);
	for (int k0 = 0; k0 < nlive; k0 += U) {
		uint32_t cn[U], kk[U];
		T v[U][4];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const bool on = k0 + u < nlive;
			const uint32_t k = st.live[on ? k0 + u : 0];
			kk[u] = k;
			const uint32_t c4 = on ? (candw[4 * k + r] >> (4 * qd)) & 0xFu : 0u;
			cn[u] = c4;
			if (c4) {
				load_quad(t.dim2 + 2 * (st.rec[k].x & ~63u) + 4 * lane, v[u]);
			} else {
#pragma unroll
				for (int j = 0; j < 4; j++)
					v[u][j] = T(0);
			}
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			const T m2 = __shfl_sync(FULL, m2_own, kk[u]);
			// all four slots are compared (values of slots without a candidate are zero or
			// loaded anyway) and the candidates masked once, not tested slot by slot
			uint32_t ge = 0;
#pragma unroll
			for (int j = 0; j < 4; j++)
				ge |= (m2 <= v[u][j]) ? 1u << j : 0u;
			uint32_t row = (ge & cn[u]) << (4 * qd);
			row |= __shfl_xor_sync(FULL, row, 1);
			row |= __shfl_xor_sync(FULL, row, 2);
			row |= __shfl_xor_sync(FULL, row, 4);
			if (qd == 0 && k0 + u < nlive)
				reinterpret_cast<uint32_t *>(st.rows)[4 * kk[u] + r] = row;
		}
	}
	__syncwarp();
	// the tested rows, or for a whole block its candidates (all reported)
	const uint4 rw = live ? st.rows[lane] : whole ? cand : make_uint4(0, 0, 0, 0);
	const uint32_t cx = 2 * base + (whole ? RECORD_WHOLE : 0u);
	child[0] = make_uint4(cx, mine.y, rw.x, rw.y);
	child[1] = make_uint4(cx + 64, mine.y, rw.z, rw.w);
	pts = __popc(rw.x) + __popc(rw.y) + __popc(rw.z) + __popc(rw.w);
	__syncwarp();  // the stage is reused by the warp's next batch
}

// One tree level of the search (the body of k_bfs_level): the boundary paths, the
// seeds and the expansion of the previous level's records, spread over `gwarps`
// warps (of the grid, or of the one CTA of k_bfs_cta).
// cnt: the level's boundary-path tasks and seeds (ctl->path_cnt[d], seed_cnt[d]
// capped at path_cap) in shared memory, read by the caller with the level's other
// counters.
template <typename T, bool LAST>
__device__ __forceinline__ void level_body(const TreeDev<T> &t, const QDev<T> &qd, const WorkDev &w, uint32_t d,
                                           uint64_t gwarp, uint64_t gwarps, uint64_t base_prev, uint64_t base_cur,
                                           uint64_t n_prev, const uint32_t *cnt, WarpStage<T> &stage)
{
	const uint32_t lane = lane_id();
	const uint32_t np = cnt[0], ns = cnt[1];
	// The level's three kinds of work go to disjoint sets of warps so that their
	// dependent-load chains overlap instead of adding up: a few warps take the
	// boundary paths, a few the seeds, the rest the records.
	const uint64_t cap = gwarps / 8 + 1;
	const uint64_t wp = min((uint64_t) (np + 31) / 32, cap);
	const uint64_t ws = min((uint64_t) (ns + 31) / 32, cap);
	const uint64_t wr = gwarps - wp - ws;  // >= 1: the grid has at least 4 warps

	if (gwarp < wp) {
		// boundary paths, one task per lane
		const uint4 *pin = (d & 1) ? w.path1 : w.path0;
		for (uint64_t wb = gwarp * 32; wb < np; wb += wp * 32) {
			const bool valid = wb + lane < np;
			path_step<T>(t, qd, w, d, valid ? pin[wb + lane] : make_uint4(0, 0, 0, 0), valid);
		}
	} else if (gwarp < wp + ws) {
		// report-above seeds of this level: one or two candidate slots each, tested
		// by their own lane
		const uint4 *sin = (d & 1) ? w.seed1 : w.seed0;
		for (uint64_t wb = (gwarp - wp) * 32; wb < ns; wb += ws * 32) {
			const bool valid = wb + lane < ns;
			const uint4 sd = valid ? sin[wb + lane] : make_uint4(0, 0, 0, 0);
			uint32_t am = 0;
			if (sd.z) {
				// a seed's candidates are the two children of one node, an aligned pair of
				// slots: their dim2, the occupancy (read on the last level only, all
				// others being full) and min2 come in one round trip
				const uint32_t p = (__ffs(sd.z) - 1) & ~1u;
				const uint32_t cand = sd.z & (d + 1 < t.levels ? FULL : t.occ[sd.x >> 5]);
				const T m2 = qd.min2[sd.y];
				T v[2];
				if constexpr (sizeof(T) == 4) {
					const uint2 x = *reinterpret_cast<const uint2 *>(t.dim2 + sd.x + p);
					memcpy(&v[0], &x.x, 4);
					memcpy(&v[1], &x.y, 4);
				} else {
					const double2 x = *reinterpret_cast<const double2 *>(t.dim2 + sd.x + p);
					v[0] = x.x;
					v[1] = x.y;
				}
#pragma unroll
				for (int j = 0; j < 2; j++)
					am |= (((cand >> (p + j)) & 1u) && m2 <= v[j]) ? 1u << (p + j) : 0u;
			}
			add_counts(w, sd.y, __popc(am), valid);
			const uint4 one[1] = {am ? block_record(sd.x, sd.y, am) : make_uint4(0, 0, 0, 0)};
			append_blocks<1>(w, d, base_cur, one);
		}
	} else {
		// expansion of the previous level's alive records into their child blocks, 32
		// consecutive records per warp (their children stay together in the next
		// level's region, which keeps that level's chunks local)
		// A narrow level (records fewer than a quarter of the record warps' lanes)
		// gives each warp 8 consecutive records instead of 32: four times the warps
		// work on it, each with a quarter of the dependent load rounds, and the
		// children of 8 consecutive parents still stay together in the next level.
		const uint64_t per = n_prev * 4 < wr * 32 ? 8 : 32;
		uint64_t wb = (gwarp - wp - ws) * per;
		bool nvalid = lane < per && wb + lane < n_prev;
		uint4 nxt = nvalid ? w.rec[base_prev + wb + lane] : make_uint4(0, 0, 0, 0);
		// A round's children are reserved with one atomic per warp, but written in the
		// next round, after that round's loads: the reservation's latency overlaps them.
		// Pending: this lane's first child block (the second at pp + 64), query, the
		// four child mask words, its first slot offset in the warp's run, and the
		// warp's reservation (lane 31; ~0 = none or refused).
		uint32_t pp = 0, pq = 0, pofs = 0, pres = ~0u;
		uint4 pm = make_uint4(0, 0, 0, 0);
		auto flush = [&]() {
			const uint32_t r0 = __shfl_sync(FULL, pres, 31);
			if (r0 == ~0u)
				return;
			uint64_t sl = base_cur + r0 + pofs;
			if (pm.x | pm.y)
				w.rec[sl++] = make_uint4(pp, pq, pm.x, pm.y);
			if (pm.z | pm.w)
				w.rec[sl] = make_uint4(pp + 64, pq, pm.z, pm.w);
		};
		for (; wb < n_prev; wb += wr * per) {
			const bool valid = nvalid;
			const uint4 mine = nxt;
			// the next round's record is read now, its load overlapping this round
			const uint64_t nb = wb + wr * per;
			nvalid = lane < per && nb + lane < n_prev;
			nxt = nvalid ? w.rec[base_prev + nb + lane] : make_uint4(0, 0, 0, 0);
			uint4 child[2];
			uint32_t pts;
			expand_records<T, LAST>(t, qd.min2, mine, valid, !LAST && d + 1 < t.levels, stage,
			                        child, pts);
			// a warp whose records found no child (most of them when a sparse last
			// level is expanded) has nothing to count or append
			if (__ballot_sync(FULL, pts != 0) == 0)
				continue;
			add_counts(w, mine.y, pts, valid);
			flush();
			const uint32_t nrec = ((child[0].z | child[0].w) ? 1u : 0u) + ((child[1].z | child[1].w) ? 1u : 0u);
			const uint32_t inc = warp_incl_scan(nrec);
			pres = ~0u;
			if (lane == 31) {
				// inc = the warp's total here (pts != 0 somewhere, so it is positive)
				const uint32_t off = atomicAdd(&w.ctl->lvl_cnt[d], inc);
				if (base_cur + off + inc > w.rec_cap) {
					atomicMax((unsigned long long *) &w.ctl->need_tasks, (unsigned long long) (base_cur + off + inc));
					atomicOr(&w.ctl->flags, BATCH_FLAG_TASK_OVERFLOW);
				} else {
					pres = off;
				}
			}
			pp = child[0].x;
			pq = mine.y;
			pofs = inc - nrec;
			pm = make_uint4(child[0].z, child[0].w, child[1].z, child[1].w);
		}
		flush();
	}
}

// LAST: the expansion into the last level of a tree with TreeDev::last_par (its own
// instantiation, so the other levels keep their register budget).  THREADS: the
// CTA size (128, 256 or 512, a tuning choice); every size keeps 64 registers a
// thread, so 1024 threads of the kernel fit an SM at once.
template <typename T, bool LAST, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_bfs_level(TreeDev<T> t, QDev<T> qd, WorkDev w,
                                                                      uint32_t d)
{
	// Launched as a programmatic dependent of the previous level: its CTAs may be
	// scheduled while that level drains, and wait here until it has completed and
	// its writes are visible (a no-op for an ordinary launch).
	asm volatile("griddepcontrol.wait;" ::: "memory");
	__shared__ uint64_t s_base[2];
	__shared__ uint32_t s_cnt[3];  // paths, seeds, stop
	__shared__ WarpStage<T> s_stage[THREADS / 32];
	if (threadIdx.x == 0) {
		// the level's counters, all in one round trip: the previous region's start and
		// length, this level's paths and seeds, and the flags
		const uint64_t b = d ? w.ctl->lvl_base[d - 1] : 0;
		const uint32_t c = d ? w.ctl->lvl_cnt[d - 1] : 0u;
		const uint32_t np = w.ctl->path_cnt[d], ns = w.ctl->seed_cnt[d], fl = w.ctl->flags;
		s_base[0] = b;
		s_base[1] = b + c;
		s_cnt[0] = min(np, w.path_cap);
		s_cnt[1] = min(ns, w.path_cap);
		s_cnt[2] = fl & BATCH_FLAG_TASK_OVERFLOW;
		if (blockIdx.x == 0)
			w.ctl->lvl_base[d] = b + c;
	}
	__syncthreads();
	// Once the frontier has overflowed, the reservation that crossed the capacity
	// left some slots below it unwritten, so nothing of the previous level may be
	// read: the pass stops here and the host repeats it with a larger buffer.
	if (s_cnt[2])
		return;
	const uint64_t base_prev = s_base[0], base_cur = s_base[1];
	// after a frontier overflow the counters run past what was stored: never read beyond it
	const uint64_t end_prev = min(base_cur, w.rec_cap);
	const uint64_t n_prev = end_prev > base_prev ? end_prev - base_prev : 0;
	const uint64_t gthreads = (uint64_t) gridDim.x * blockDim.x;
	const uint64_t gtid = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
	const uint64_t gwarps = gthreads / 32, gwarp = gtid / 32;
	level_body<T, LAST>(t, qd, w, d, gwarp, gwarps, base_prev, base_cur, n_prev, s_cnt,
	                    s_stage[threadIdx.x >> 5]);
}

// Query i of the batch: its kind and bounds into the engine's per-query arrays, and
// its level-0 boundary path task (returned); a kind out of range raises
// BATCH_FLAG_BAD_QUERY in *flags (the pass still runs, and the host reports it).
template <typename T>
__device__ __forceinline__ uint4 unpack_query(const pst_query &q, uint32_t i, const QOut<T> &qo, uint32_t *flags)
{
	T a, b, c;
	if constexpr (sizeof(T) == 8) {
		a = q.min1.f64; b = q.max1.f64; c = q.min2.f64;
	} else if constexpr (std::is_same<T, float>::value) {
		a = q.min1.f32; b = q.max1.f32; c = q.min2.f32;
	} else {
		a = q.min1.i32; b = q.max1.i32; c = q.min2.i32;
	}
	const int32_t k = q.kind;
	if (k < PST_Q_THREE || k > PST_Q_RIGHT)
		atomicOr(flags, BATCH_FLAG_BAD_QUERY);
	qo.kind[i] = (uint32_t) k;
	qo.min1[i] = a;
	qo.max1[i] = b;
	qo.min2[i] = c;
	const uint32_t mode = k == PST_Q_THREE ? MODE_THREE : k == PST_Q_LEFT ? MODE_LEFT : MODE_RIGHT;
	return make_uint4(1u, i, mode, 0u);
}

// The pass's control block from the engine's pinned host copy, read through its
// mapped device address: a kernel, because inside the captured pass a
// host-to-device copy node ahead of the first kernel left the device idle for
// ≈ 25 µs per pass.
__global__ void k_load_ctl(const BatchCtl *src, BatchCtl *dst)
{
	const uint32_t *s = reinterpret_cast<const uint32_t *>(src);
	uint32_t *d = reinterpret_cast<uint32_t *>(dst);
	for (uint32_t i = threadIdx.x; i < sizeof(BatchCtl) / 4; i += blockDim.x)
		d[i] = s[i];
}

// The control block of a pass that a caller captures into a graph of theirs, from the
// kernel's own parameters: the engine's pinned copy belongs to the calls that come later.
__global__ void k_set_ctl(BatchCtl *ctl, const PassStart start)
{
	for (uint32_t i = threadIdx.x; i < sizeof(BatchCtl) / 4; i += blockDim.x)
		reinterpret_cast<uint32_t *>(ctl)[i] = 0;
	__syncthreads();
	if (threadIdx.x == 0) {
		ctl->nq = start.nq;
		ctl->raw = start.raw;
		ctl->user_offsets = start.offsets;
	}
}

// Start of a full pass (after the control block's load): the batch's queries
// unpacked and checked, their level-0 paths, and the per-query counts and output
// cursors zeroed (all max_q of them: the scan reads every count).
template <typename T>
__global__ void k_prepare_queries(BatchCtl *ctl, QOut<T> qo, uint4 *path0, uint64_t *counts, uint64_t *cursor,
                                  uint32_t max_q)
{
	const uint32_t nq = ctl->nq;
	const pst_query *raw = ctl->raw;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < max_q; i += gridDim.x * blockDim.x) {
		if (i < nq)
			path0[i] = unpack_query<T>(raw[i], i, qo, &ctl->flags);
		counts[i] = 0;
		cursor[i] = 0;
	}
	if (blockIdx.x == 0 && threadIdx.x == 0)
		ctl->path_cnt[0] = nq;
}

// Output slot of this lane's record inside its query's result: one atomic per run
// of equal query ids on the query's cursor.
__device__ __forceinline__ uint64_t claim_output(const WorkDev &w, uint32_t q, uint32_t pc, bool valid)
{
	bool last;
	const uint64_t run = warp_run_sum(valid ? q : 0xFFFFFFFFu, pc, &last);
	const uint32_t lastmask = __ballot_sync(FULL, last);
	const uint32_t run_last = (uint32_t) (__ffs(lastmask & (FULL << lane_id())) - 1);
	uint64_t rb = 0;
	if (valid && last && run)
		rb = atomicAdd((unsigned long long *) &w.cursor[q], (unsigned long long) run);
	rb = __shfl_sync(FULL, rb, run_last);
	return (valid && pc) ? w.offsets[q] + rb + run - pc : 0;
}

// Output range check of one lane's record, made once where the lane claims it: a
// record whose claimed range would end past the output's capacity is cleared (it
// writes nothing) and flagged.  Counts and claims come from the same masks, so this
// never fires; it keeps the warp-wide store loop of emit_blocks free of per-store
// checks (a 64-bit compare at every 4-byte store cost 8 % of a batched step).
__device__ __forceinline__ void guard_claim(const WorkDev &w, uint4 &rec, uint64_t out_base, uint64_t capacity)
{
	if (out_base + __popc(rec.z) + __popc(rec.w) > capacity) {
		atomicOr(&w.ctl->flags, BATCH_FLAG_INTERNAL);
		if (uint32_t *host = w.ctl->host_fault)
			*host = 1;
		rec.z = rec.w = 0;
	}
}

// Writes the results of the warp's records (lane k owns record `mine`, whose results
// start at out_base, checked by guard_claim; the valid lanes are a prefix): the
// lanes stage their records and offsets, then the warp writes U records at a time,
// each by the whole warp.
struct EmitStage {
	uint4 rec[32];
	unsigned long long ob[32];
};

// Ids: lane l takes slots 2l and 2l + 1 of the 64-slot block (one 8-byte load).  Slots
// l and l + 32, whose stores cover consecutive words, took 1468 against 1318 us for
// the 948 M ids of a 4096-query batch at 2^28 points: a second load a record costs
// more than the denser stores give, the kernel being bound by its instructions.
template <int U>
__device__ __forceinline__ void emit_ids(const uint32_t *__restrict__ id, int nrec, const EmitStage &st,
                                         uint32_t *__restrict__ out)
{
	const uint32_t lane = lane_id();
	const uint32_t psh = (2 * lane) & 31;
	// the record's slots before this lane's pair, as masks of its two 32-slot words
	const uint32_t below_z = lane < 16 ? (1u << psh) - 1u : FULL;
	const uint32_t below_w = lane < 16 ? 0u : (1u << psh) - 1u;
	for (int k0 = 0; k0 < nrec; k0 += U) {
		uint32_t b2[U];
		uint64_t o[U];
		uint2 idv[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			// every lane staged a record, and those past nrec are empty (zero masks), so
			// a batch that runs past nrec reads them and writes nothing: no bound test
			// per record (U divides 32, so k < 32)
			const int k = k0 + u;
			const uint4 rc = st.rec[k];
			b2[u] = ((lane < 16 ? rc.z : rc.w) >> psh) & 3u;
			const uint32_t before = __popc(rc.z & below_z) + __popc(rc.w & below_w);
			o[u] = st.ob[k] + before;
			const uint32_t hb = (rc.x & ~63u) + 2 * lane;  // (without RECORD_WHOLE)
			idv[u] = b2[u] ? *reinterpret_cast<const uint2 *>(id + hb) : make_uint2(0, 0);
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
#pragma unroll
			for (int j = 0; j < 2; j++) {
				if ((b2[u] >> j) & 1u) {
					const uint64_t oo = o[u] + (j & b2[u]);  // the second slot follows a reported first
					// evict-first: the output streams through L2 once and should not push
					// out tree rows that other queries' records read again
					__stcs(out + oo, j ? idv[u].y : idv[u].x);
				}
			}
		}
	}
}

// A packed point's id, with the padding of a 24-byte point (it leaves with the words).
template <typename T>
__device__ __forceinline__ void pack_id(Point<T, true> &p, uint32_t id)
{
	if constexpr (sizeof(T) == 8)
		*reinterpret_cast<unsigned long long *>(&p.id) = id;
	else
		p.id = id;
}

// Points: lane l takes slots l and l + 32 (a load reads one whole row of a field), and
// the points of a record are packed into shared memory in the order of the output and
// leave it as consecutive words.  A store a lane of a field of an 8- to 24-byte point
// touched every sector of the record's range once per field: 127 us for the 6.2 M
// 24-byte points of a 601-query batch at 12.3 M points, 69 us packed.
template <typename T, bool HAS_ID, int U>
__device__ __forceinline__ void emit_points(const TreeDev<T> &t, int nrec, const EmitStage &st,
                                            Point<T, HAS_ID> *pack, Point<T, HAS_ID> *__restrict__ out)
{
	using Pt = Point<T, HAS_ID>;
	using W = typename std::conditional<sizeof(T) == 8, unsigned long long, uint32_t>::type;
	const uint32_t lane = lane_id(), below = lanemask_lt();
	for (int k0 = 0; k0 < nrec; k0 += U) {
		uint32_t m[U][2], idv[U][2];
		T d1[U][2], d2[U][2];
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint4 rc = st.rec[k0 + u];  // (empty past nrec, as in emit_ids)
			m[u][0] = rc.z;
			m[u][1] = rc.w;
#pragma unroll
			for (int j = 0; j < 2; j++) {
				const uint32_t h = (rc.x & ~63u) + 32 * j + lane;
				const bool on = (m[u][j] >> lane) & 1u;
				d1[u][j] = on ? t.dim1[h] : T(0);
				d2[u][j] = on ? t.dim2[h] : T(0);
				if constexpr (HAS_ID)
					idv[u][j] = on ? t.id[h] : 0u;
			}
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			const uint32_t nz = __popc(m[u][0]);
#pragma unroll
			for (int j = 0; j < 2; j++) {
				if ((m[u][j] >> lane) & 1u) {
					Pt &p = pack[(j ? nz : 0u) + __popc(m[u][j] & below)];
					p.dim1 = d1[u][j];
					p.dim2 = d2[u][j];
					if constexpr (HAS_ID)
						pack_id(p, idv[u][j]);
				}
			}
			__syncwarp();
			const uint32_t words = (nz + __popc(m[u][1])) * (uint32_t) (sizeof(Pt) / sizeof(W));
			const W *src = reinterpret_cast<const W *>(pack);
			W *dst = reinterpret_cast<W *>(out + st.ob[k0 + u]);
			for (uint32_t i = lane; i < words; i += 32)
				__stcs(dst + i, src[i]);  // evict-first, as the ids
			__syncwarp();  // the pack is refilled by the next record
		}
	}
}

// Shared memory of one emitting warp.
template <typename Pt, bool POINTS>
struct EmitWarp {
	EmitStage st;
	Pt pack[POINTS ? 64 : 1];
};

template <typename T, bool HAS_ID, bool POINTS, int U>
__device__ __forceinline__ void emit_blocks(const TreeDev<T> &t, const uint4 &mine, uint64_t out_base, bool valid,
                                            EmitWarp<Point<T, HAS_ID>, POINTS> &sm, void *__restrict__ out)
{
	static_assert(32 % U == 0, "a batch of records ends inside the 32 staged ones");
	const uint32_t lane = lane_id();
	sm.st.rec[lane] = mine;
	sm.st.ob[lane] = out_base;
	__syncwarp();
	const int nrec = __popc(__ballot_sync(FULL, valid));
	if constexpr (POINTS)
		emit_points<T, HAS_ID, U>(t, nrec, sm.st, sm.pack, static_cast<Point<T, HAS_ID> *>(out));
	else
		emit_ids<U>(t.id, nrec, sm.st, static_cast<uint32_t *>(out));
	__syncwarp();  // the stage is reused by the warp's next batch
}

// Small batches (a single query, or a few): one CTA takes the tree from the top,
// level by level with a CTA barrier in place of a kernel boundary, while the
// records to expand stay few enough for it (at most CTA_REC_CAP); it leaves
// ctl->cta_levels = the levels done and the host launches the per-level kernels
// for the rest only.  When it reaches the bottom it also scans the queries' counts
// into their offsets, and writes the results itself when they are few
// (CTA_EMIT_CAP), so that the call is this one kernel.
//
// The pass is a chain of levels, each a few dependent steps, so everything a level
// touches but the tree is in shared memory: the control block, the paths and seeds (pcap
// of each of the four lists), the counts (qcap) and the records of every level it takes
// (rcap).  A record's children are read at once with the subtree minimum that may make
// the reading needless (level_body asks for that first, to spare the loads: two round
// trips a level); reservations are single shared-memory atomics, counts are sums of
// one; and every thread keeps the level's bounds itself, so that one barrier ends a level.
// One query on 64.5 k points (16 levels, 6.5 k ids): 30 us with the per-level kernels' body
// between two barriers a level and 7 for the emit, 21 us with its results written; the
// call 88 -> 41 us.  A few host queries and the arguments come as the kernel's
// parameters (reading them from mapped host memory takes 3.7 us), and the control block goes
// back to mapped host memory: a copy each way took 16 us of a call.
// Where the pass stops, it writes the records, the counts and the next level's paths
// and seeds to their global buffers, in the layout the per-level kernels and the emit
// read.  It stops early when the next level might not fit in rcap.
// With 256 records instead of 160, 16 isovalues over 2^21 metacells took 108 us, and with
// 96 one query for 1 % of 2^24 points took 87; with 160 they take 106 and 83.
constexpr uint32_t CTA_REC_CAP = 160;
// A single query's 6.5 k ids from a kernel of their own: 69 us a call instead of 45.
constexpr uint32_t CTA_EMIT_CAP = 16384;
constexpr int TOP_THREADS = 512, TOP_WARPS = TOP_THREADS / 32;

// Dynamic shared memory of k_bfs_cta: the control block (built at the end), a cell of
// counters per level, the queries' offsets, counts and cursors, the four path and seed
// lists, then the records.
constexpr uint32_t TOP_CELLS = 41;
__host__ __device__ constexpr size_t cta_smem_bytes(uint32_t qcap, uint32_t pcap, uint32_t rcap)
{
	return sizeof(BatchCtl) + (size_t) (TOP_CELLS + qcap + 4 * pcap + rcap) * sizeof(uint4);
}
static_assert(sizeof(BatchCtl) % 16 == 0, "the lists after the control block stay 16-byte aligned");

// Shared memory by its own 32-bit addresses: accesses through pointers that reach a level's
// code in a struct were compiled as generic ones (130 cycles for a load, 30 as such).
__device__ __forceinline__ uint4 sh_ld4(uint32_t a)
{
	uint4 v;
	asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
	return v;
}
__device__ __forceinline__ void sh_st4(uint32_t a, const uint4 &v)
{
	asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sh_st(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t sh_add(uint32_t a, uint32_t n)
{
	uint32_t v;
	asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(v) : "r"(a), "r"(n) : "memory");
	return v;
}
__device__ __forceinline__ void sh_or(uint32_t a, uint32_t m) { asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(a), "r"(m) : "memory"); }

// The top pass's shared memory (addresses in it) and where its query bounds are.
template <typename T>
struct TopPass {
	QDev<T> qd;
	// cell d: records of level d - 1, paths and seeds of level d, start of level d's records
	uint32_t cells;
	uint32_t flags, rec_cnt;
	uint32_t cnt, cur;  // a word per query, from query q0 on
	uint32_t q0;
	uint32_t lists, rec;
	uint4 *ro;          // reported boundary nodes
	uint32_t pcap, ro_cap;

	__device__ __forceinline__ uint32_t cell(uint32_t d) const { return cells + 16 * d; }
	// entry i of the paths and of the seeds of level d
	__device__ __forceinline__ uint32_t path(uint32_t d, uint32_t i) const { return lists + 16 * ((d & 1) * pcap + i); }
	__device__ __forceinline__ uint32_t seed(uint32_t d, uint32_t i) const { return lists + 16 * ((2 + (d & 1)) * pcap + i); }
};

// 32 boundary-path tasks of level d (path_step's rules).  Every lane reserves for itself:
// the lanes at work are few.
template <typename T>
__device__ __forceinline__ void top_paths(const TreeDev<T> &t, const TopPass<T> &p, uint32_t d, uint32_t at, uint32_t np)
{
	const uint32_t i = at + lane_id();
	if (i >= np)
		return;
	const uint4 task = sh_ld4(p.path(d, i));
	const uint32_t h = task.x, q = task.y, mode = task.z, l = 2 * h, r = l + 1;
	bool rep = false, rl = false, rr = false;
	uint32_t pl = 0, pr = 0;
	const bool inner = d + 1 < t.levels;
	const T v2 = t.dim2[h], v1 = t.dim1[h];
	const T m = inner ? t.med[h] : T(0);
	const uint32_t ow = !inner ? 0u : d + 2 < t.levels ? FULL : t.occ[l >> 5];
	const T min2 = p.qd.min2[q], min1 = p.qd.min1[q], max1 = p.qd.max1[q];
	const uint32_t kind = p.qd.kind[q];
	path_rules<T>(kind, mode, min1, max1, min2, v1, v2, m, (ow >> (l & 31)) & 1u, (ow >> (r & 31)) & 1u, rep, pl, pr, rl,
	              rr);
	const uint32_t next = p.cell(d + 1), npl = (pl ? 1u : 0u) + (pr ? 1u : 0u);
	const bool seed = rl || rr;
	// the three reservations are on their way together
	const uint32_t b_path = npl ? sh_add(next + 4, npl) : 0u, b_seed = seed ? sh_add(next + 8, 1) : 0u,
	               b_rep = rep ? sh_add(p.rec_cnt, 1) : 0u;
	// (the lists hold all there can be: two paths a query and level)
	bool lost = b_path + npl > p.pcap;
	if (!lost) {
		if (pl)
			sh_st4(p.path(d + 1, b_path), make_uint4(l, q, pl, 0));
		if (pr)
			sh_st4(p.path(d + 1, b_path + npl - 1), make_uint4(r, q, pr, 0));
	}
	if (seed) {
		if (b_seed < p.pcap)
			sh_st4(p.seed(d + 1, b_seed), make_uint4(l & ~31u, q, (rl ? 1u << (l & 31) : 0u) | (rr ? 1u << (r & 31) : 0u), 0u));
		else
			lost = true;
	}
	if (rep) {
		if (b_rep < p.ro_cap)
			p.ro[b_rep] = block_record(h & ~31u, q, 1u << (h & 31));
		else
			lost = true;
		sh_add(p.cnt + 4 * (q - p.q0), 1);
	}
	if (lost)
		sh_or(p.flags, BATCH_FLAG_INTERNAL);
}

// 32 report-above seeds of level d: each the aligned pair of one node's children.
template <typename T>
__device__ __forceinline__ void top_seeds(const TreeDev<T> &t, const TopPass<T> &p, uint32_t d, uint32_t at, uint32_t ns,
                                          uint32_t base_cur)
{
	const uint32_t i = at + lane_id();
	if (i >= ns)
		return;
	const uint4 sd = sh_ld4(p.seed(d, i));
	const uint32_t b = (__ffs(sd.z) - 1) & ~1u;
	const T v0 = t.dim2[sd.x + b], v1 = t.dim2[sd.x + b + 1];
	const uint32_t cand = sd.z & (d + 1 < t.levels ? FULL : t.occ[sd.x >> 5]);
	const T m2 = p.qd.min2[sd.y];
	const uint32_t am =
	    (((cand >> b) & 1u) && m2 <= v0 ? 1u << b : 0u) | (((cand >> (b + 1)) & 1u) && m2 <= v1 ? 2u << b : 0u);
	if (am) {
		sh_st4(p.rec + 16 * (base_cur + sh_add(p.cell(d + 1), 1)), block_record(sd.x, sd.y, am));
		sh_add(p.cnt + 4 * (sd.y - p.q0), (uint32_t) __popc(am));
	}
}

// The children of the records [at, end) of the level above (at most TOP_U): the warp takes
// each record whole, lane l its child slots [2b + 4l, 2b + 4l + 4).
constexpr int TOP_U = 4;

template <typename T>
__device__ __forceinline__ void top_records(const TreeDev<T> &t, const TopPass<T> &p, uint32_t d, uint32_t at,
                                            uint32_t end, uint32_t base_cur)
{
	const uint32_t lane = lane_id();
	const bool last = d + 1 == t.levels;
	uint4 rc[TOP_U];
	uint32_t nib[TOP_U];
	T v[TOP_U][4], m2[TOP_U], sm[TOP_U];
#pragma unroll
	for (int u = 0; u < TOP_U; u++)
		rc[u] = at + u < end ? sh_ld4(p.rec + 16 * (at + u)) : make_uint4(0, 0, 0, 0);
#pragma unroll
	for (int u = 0; u < TOP_U; u++) {
		const uint32_t base = rc[u].x & ~63u;
		const uint32_t two = ((lane < 16 ? rc[u].z : rc[u].w) >> ((2 * lane) & 31)) & 3u;  // the lane's parents
		nib[u] = (two & 1u ? 3u : 0u) | (two & 2u ? 12u : 0u);
		const bool look = (rc[u].x & RECORD_WHOLE) == 0 && (rc[u].z | rc[u].w) != 0;
		m2[u] = look ? p.qd.min2[rc[u].y] : T(0);
		sm[u] = look && t.sub_min && base >= 64 ? t.sub_min[base >> 6] : T(0);
		const uint32_t c = 2 * base + 4 * lane;
		const uint32_t ow = last && nib[u] ? t.occ[c >> 5] >> (c & 31) : FULL;
		if (look && nib[u]) {
			load_quad(t.dim2 + c, v[u]);
		} else {
#pragma unroll
			for (int j = 0; j < 4; j++)
				v[u][j] = T(0);
		}
		nib[u] &= ow;
	}
	// the lane's child record of the warp: half (lane & 1) of record lane >> 1
	uint4 mine = make_uint4(0, 0, 0, 0);
	uint32_t pts = 0, ptsq = 0;  // lane u: the points of record u, and its query
#pragma unroll
	for (int u = 0; u < TOP_U; u++) {
		const uint32_t base = rc[u].x & ~63u;
		const bool whole = (rc[u].x & RECORD_WHOLE) != 0 || (t.sub_min && base >= 64 && m2[u] <= sm[u]);
		uint32_t ge = 0;
#pragma unroll
		for (int j = 0; j < 4; j++)
			ge |= m2[u] <= v[u][j] ? 1u << j : 0u;
		nib[u] &= whole ? 0xFu : ge;
		const uint32_t n = __reduce_add_sync(FULL, __popc(nib[u]));
		if (lane == (uint32_t) u) {
			pts = n;
			ptsq = rc[u].y;
		}
		// 8 lanes make a 32-slot row, two rows a child block
		uint32_t row = nib[u] << (4 * (lane & 7));
		row |= __shfl_xor_sync(FULL, row, 1);
		row |= __shfl_xor_sync(FULL, row, 2);
		row |= __shfl_xor_sync(FULL, row, 4);
		const uint32_t lo = __shfl_sync(FULL, row, 16 * (lane & 1)), hi = __shfl_sync(FULL, row, 16 * (lane & 1) + 8);
		if (lane >> 1 == (uint32_t) u)
			mine = make_uint4(2 * base + 64 * (lane & 1) + (whole ? RECORD_WHOLE : 0u), rc[u].y, lo, hi);
	}
	if (mine.z | mine.w)
		sh_st4(p.rec + 16 * (base_cur + sh_add(p.cell(d + 1), 1)), mine);
	if (pts)
		sh_add(p.cnt + 4 * (ptsq - p.q0), pts);
}

// Level d of the pass, shared out over the CTA's warps: np paths, ns seeds, and the records
// [base_prev, base_cur) of the level above.
template <typename T>
__device__ __forceinline__ void top_level(const TreeDev<T> &t, const TopPass<T> &p, uint32_t d, uint32_t np, uint32_t ns,
                                          uint32_t base_prev, uint32_t base_cur)
{
	const uint32_t wp = (np + 31) / 32, ws = (ns + 31) / 32, wr = (base_cur - base_prev + TOP_U - 1) / TOP_U;
	for (uint32_t i = threadIdx.x >> 5; i < wp + ws + wr; i += TOP_WARPS) {
		if (i < wp)
			top_paths<T>(t, p, d, 32 * i, np);
		else if (i < wp + ws)
			top_seeds<T>(t, p, d, 32 * (i - wp), ns, base_cur);
		else
			top_records<T>(t, p, d, base_prev + TOP_U * (i - wp - ws), base_cur, base_cur);
	}
}

// Writes the slots of the blocks at[0 .. n) that their masks name, each from output place
// rec.y on (the place the record has claimed), TOP_U blocks in flight.
template <typename T>
__device__ __forceinline__ void top_write(const TreeDev<T> &t, const uint4 *at, uint32_t n, uint32_t ret, void *out)
{
	const uint32_t lane = lane_id(), below = lanemask_lt();
	uint4 rc[TOP_U];
#pragma unroll
	for (int u = 0; u < TOP_U; u++)
		rc[u] = (uint32_t) u < n ? at[u] : make_uint4(0, 0, 0, 0);
	if (ret == PST_RET_IDS) {
		uint32_t id[TOP_U][2];
#pragma unroll
		for (int u = 0; u < TOP_U; u++)
#pragma unroll
			for (int j = 0; j < 2; j++)
				id[u][j] = ((j ? rc[u].w : rc[u].z) >> lane) & 1u ? t.id[(rc[u].x & ~63u) + 32 * j + lane] : 0u;
#pragma unroll
		for (int u = 0; u < TOP_U; u++)
#pragma unroll
			for (int j = 0; j < 2; j++) {
				const uint32_t m = j ? rc[u].w : rc[u].z;
				if ((m >> lane) & 1u)
					static_cast<uint32_t *>(out)[rc[u].y + (j ? __popc(rc[u].z) : 0) + __popc(m & below)] = id[u][j];
			}
		return;
	}
#pragma unroll
	for (int u = 0; u < TOP_U; u++)
#pragma unroll
		for (int j = 0; j < 2; j++) {
			const uint32_t m = j ? rc[u].w : rc[u].z;
			if (!((m >> lane) & 1u))
				continue;
			const uint32_t h = (rc[u].x & ~63u) + 32 * j + lane;
			const uint32_t k = rc[u].y + (j ? __popc(rc[u].z) : 0) + __popc(m & below);
			if (t.id) {
				Point<T, true> &pt = static_cast<Point<T, true> *>(out)[k];
				pt.dim1 = t.dim1[h];
				pt.dim2 = t.dim2[h];
				pack_id(pt, t.id[h]);
			} else {
				Point<T, false> &pt = static_cast<Point<T, false> *>(out)[k];
				pt.dim1 = t.dim1[h];
				pt.dim2 = t.dim2[h];
			}
		}
}

template <typename T>
__global__ void __launch_bounds__(TOP_THREADS, 1) k_bfs_cta(TreeDev<T> t, QDev<T> qd, WorkDev wg, uint32_t max_q,
                                                            uint32_t qcap, uint32_t pcap, uint32_t rcap, QOut<T> qo,
                                                            const __grid_constant__ TopIn in, BatchCtl *back)
{
	extern __shared__ __align__(16) unsigned char s_dyn[];
	__shared__ uint64_t s_total;
	__shared__ uint32_t s_word[2];  // flags, reported boundary nodes
	BatchCtl *sc = reinterpret_cast<BatchCtl *>(s_dyn);
	uint4 *s_cell = reinterpret_cast<uint4 *>(s_dyn + sizeof(BatchCtl));
	uint64_t *s_offs = reinterpret_cast<uint64_t *>(s_cell + TOP_CELLS);
	uint32_t *s_cnt = reinterpret_cast<uint32_t *>(s_offs + qcap), *s_cur = s_cnt + qcap;
	uint4 *s_list = reinterpret_cast<uint4 *>(s_cur + qcap), *s_rec = s_list + 4 * pcap;
	TopPass<T> p;
	p.qd = qd;
	auto addr = [](const void *x) { return static_cast<uint32_t>(__cvta_generic_to_shared(x)); };
	p.cells = addr(s_cell);
	p.flags = addr(&s_word[0]);
	p.rec_cnt = addr(&s_word[1]);
	p.cnt = addr(s_cnt);
	p.cur = addr(s_cur);
	p.q0 = 0;
	p.lists = addr(s_list);
	p.rec = addr(s_rec);
	p.pcap = pcap;
	p.ro = wg.ro;
	p.ro_cap = wg.ro_cap;
	// the start of the pass (k_prepare_queries of a full pass): the counters zeroed, the
	// queries unpacked and checked, their level-0 paths (at most qcap queries: the host runs
	// this pass for small batches only)
	const uint32_t nq = min(in.args.nq, qcap);
	if (threadIdx.x < 2)
		s_word[threadIdx.x] = 0;
	for (uint32_t i = threadIdx.x; i < TOP_CELLS; i += TOP_THREADS)
		s_cell[i] = make_uint4(0, i ? 0u : nq, 0, 0);
	for (uint32_t i = threadIdx.x; i < sizeof(BatchCtl) / 4; i += TOP_THREADS)
		reinterpret_cast<uint32_t *>(sc)[i] = 0;
	__syncthreads();
	for (uint32_t i = threadIdx.x; i < qcap; i += TOP_THREADS) {
		if (i < nq)
			s_list[i] = unpack_query<T>(in.args.raw ? in.args.raw[i] : in.q[i], i, qo, &s_word[0]);
		s_cnt[i] = 0;
		s_cur[i] = 0;
	}
	__syncthreads();
	const uint32_t warp = threadIdx.x >> 5;
	uint32_t base_prev = 0, base_cur = 0, d = 0;
	for (; d < t.levels; d++) {
		const uint4 c = sh_ld4(p.cell(d));
		const uint32_t prev = c.x, np = min(c.y, pcap), ns = min(c.z, pcap);
		base_prev = base_cur;
		base_cur += prev;
		// the level appends at most two children per record and one record per seed
		if (prev > CTA_REC_CAP || base_cur + 2 * prev + ns > rcap)
			break;
		if (prev + np + ns == 0) {
			d = t.levels;  // nothing is left on any level below
			break;
		}
		if (threadIdx.x == 0)
			sh_st(p.cell(d) + 12, base_cur);
		top_level<T>(t, p, d, np, ns, base_prev, base_cur);
		__syncthreads();  // the level's records, paths, seeds and counts are visible to the CTA
	}
	// records written: at the bottom the last level's follow base_cur (none, where the pass
	// ended above it because nothing was left); where the pass stopped at level d, base_cur
	// is already past level d - 1
	const bool done = d == t.levels;
	const uint32_t nrec = min(base_cur + (done ? s_cell[t.levels].x : 0u), rcap);
	if (done && warp == 0) {
		uint64_t run = 0;
		for (uint32_t q0 = 0; q0 < nq; q0 += 32) {
			const uint32_t q = q0 + lane_id();
			const uint64_t c = q < nq ? s_cnt[q] : 0u;
			const uint64_t inc = warp_incl_scan(c);
			if (q < nq)
				s_offs[q] = run + inc - c;
			run += __shfl_sync(FULL, inc, 31);
		}
		if (lane_id() == 0)
			s_total = run;
	}
	__syncthreads();
	const uint64_t total = done ? s_total : 0;
	const uint32_t flags = s_word[0], nro = min(s_word[1], p.ro_cap);
	const bool emit = done && in.args.out && total <= in.args.out_cap && total <= CTA_EMIT_CAP &&
	                  !(flags & (BATCH_FLAG_BAD_QUERY | BATCH_FLAG_INTERNAL));
	const bool over = !emit && nrec > wg.rec_cap;
	// the control block: every counter the host and the next kernels read
	if (threadIdx.x < 40) {
		const uint4 c = s_cell[threadIdx.x];
		sc->lvl_cnt[threadIdx.x] = s_cell[threadIdx.x + 1].x;
		sc->path_cnt[threadIdx.x] = c.y;
		sc->seed_cnt[threadIdx.x] = c.z;
		sc->lvl_base[threadIdx.x] = c.w;
	} else if (threadIdx.x == 64) {
		sc->rec_cnt = s_word[1];
		sc->nq = nq;
		sc->flags = flags | (over ? (uint32_t) BATCH_FLAG_TASK_OVERFLOW : 0u);
		sc->cta_levels = d;
		sc->need_tasks = over ? nrec : 0;
		sc->total = total;
		sc->emitted = emit;
		sc->waits = 1;
		sc->user_offsets = in.args.offsets;  // for a scan that follows
		sc->host_fault = back ? &back->fault : nullptr;
		sc->emit_follows = in.args.out != nullptr;
	}
	uint64_t *offsets = const_cast<uint64_t *>(wg.offsets);
	if (done) {
		for (uint32_t q = threadIdx.x; q <= max_q; q += TOP_THREADS)
			offsets[q] = q < nq ? s_offs[q] : total;
		if (in.args.offsets && !(flags & BATCH_FLAGS_FAILED))
			for (uint32_t q = threadIdx.x; q <= nq; q += TOP_THREADS)
				in.args.offsets[q] = q < nq ? s_offs[q] : total;
	}
	for (uint32_t q = threadIdx.x; q < max_q; q += TOP_THREADS) {
		wg.counts[q] = q < nq ? s_cnt[q] : 0u;
		wg.cursor[q] = 0;
	}
	if (emit) {
		// every record claims its place (kept where its query was); the reported boundary
		// nodes follow them as records of one slot
		for (uint32_t i = threadIdx.x; i < nrec; i += TOP_THREADS) {
			const uint4 x = s_rec[i];
			s_rec[i].y = (uint32_t) s_offs[x.y] + sh_add(p.cur + 4 * x.y, (uint32_t) (__popc(x.z) + __popc(x.w)));
		}
		for (uint32_t i = threadIdx.x; i < nro; i += TOP_THREADS) {
			const uint32_t q = p.ro[i].y;
			p.ro[i].y = (uint32_t) s_offs[q] + sh_add(p.cur + 4 * q, 1);
		}
		__syncthreads();
		for (uint32_t i = warp * TOP_U; i < nrec; i += TOP_WARPS * TOP_U)
			top_write<T>(t, s_rec + i, min(nrec - i, (uint32_t) TOP_U), in.args.ret, in.args.out);
		for (uint32_t i = warp * TOP_U; i < nro; i += TOP_WARPS * TOP_U)
			top_write<T>(t, p.ro + i, min(nro - i, (uint32_t) TOP_U), in.args.ret, in.args.out);
	} else {
		for (uint32_t i = threadIdx.x; i < nrec && nrec <= wg.rec_cap; i += TOP_THREADS)
			wg.rec[i] = s_rec[i];
		if (!done) {
			const uint32_t np = min(s_cell[d].y, pcap), ns = min(s_cell[d].z, pcap);
			uint4 *pd = (d & 1) ? wg.path1 : wg.path0, *sd = (d & 1) ? wg.seed1 : wg.seed0;
			for (uint32_t i = threadIdx.x; i < np; i += TOP_THREADS)
				pd[i] = s_list[(d & 1) * pcap + i];
			for (uint32_t i = threadIdx.x; i < ns; i += TOP_THREADS)
				sd[i] = s_list[(2 + (d & 1)) * pcap + i];
		}
	}
	__syncthreads();
	if (threadIdx.x < sizeof(BatchCtl) / 4) {
		const uint32_t x = reinterpret_cast<const uint32_t *>(sc)[threadIdx.x];
		reinterpret_cast<uint32_t *>(wg.ctl)[threadIdx.x] = x;
		if (back)
			reinterpret_cast<uint32_t *>(back)[threadIdx.x] = x;
	}
}

// The first `stop` levels of a whole pass, in place of as many level kernels: a CTA per
// group of g queries, which walks them as k_bfs_cta does and waits for no other CTA.  What
// it leaves: the records of the last level it took, in that level's region, and the paths
// and seeds of the next, for the level kernels; the records above, which nobody expands
// again, with the reported boundary nodes.  (After the control block's load; it unpacks
// the queries and zeroes the counts and cursors too.)
//
// A narrow level is a launch and one warp's chain of loads, 5 to 6 us whatever its size; in
// here it takes 1.1 to 1.5 us.  How far that reaches is a bound on the records (top_levels
// below), not a look at the queries: the pass is queued without waiting.
template <typename T>
__global__ void __launch_bounds__(TOP_THREADS, 1) k_bfs_groups(TreeDev<T> t, QDev<T> qd, WorkDev wg, QOut<T> qo,
                                                               uint32_t max_q, uint32_t g, uint32_t rocap,
                                                               uint32_t rcap, uint32_t stop)
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	extern __shared__ __align__(16) unsigned char s_dyn[];
	__shared__ uint32_t s_word[2];  // flags, reported boundary nodes
	__shared__ uint32_t s_at[4];    // places taken in the global lists
	uint4 *s_cell = reinterpret_cast<uint4 *>(s_dyn);
	uint4 *s_list = s_cell + TOP_CELLS, *s_ro = s_list + 8 * g, *s_rec = s_ro + rocap;
	uint32_t *s_cnt = reinterpret_cast<uint32_t *>(s_rec + rcap);
	const uint32_t q0 = blockIdx.x * g, nq = wg.ctl->nq;
	const pst_query *raw = wg.ctl->raw;
	const uint32_t mine = nq > q0 ? min(nq - q0, g) : 0u;
	TopPass<T> p;
	p.qd = qd;
	auto addr = [](const void *x) { return static_cast<uint32_t>(__cvta_generic_to_shared(x)); };
	p.cells = addr(s_cell);
	p.flags = addr(&s_word[0]);
	p.rec_cnt = addr(&s_word[1]);
	p.cnt = addr(s_cnt);
	p.cur = 0;
	p.q0 = q0;
	p.lists = addr(s_list);
	p.rec = addr(s_rec);
	p.pcap = 2 * g;
	p.ro = s_ro;
	p.ro_cap = rocap;
	if (threadIdx.x < 2)
		s_word[threadIdx.x] = 0;
	for (uint32_t i = threadIdx.x; i < TOP_CELLS; i += TOP_THREADS)
		s_cell[i] = make_uint4(0, i ? 0u : mine, 0, 0);
	for (uint32_t i = threadIdx.x; i < g; i += TOP_THREADS)
		s_cnt[i] = 0;
	__syncthreads();
	for (uint32_t i = threadIdx.x; i < mine; i += TOP_THREADS)
		s_list[i] = unpack_query<T>(raw[q0 + i], q0 + i, qo, &s_word[0]);
	__syncthreads();
	uint32_t base_prev = 0, base_cur = 0;
	for (uint32_t d = 0; d < stop; d++) {
		const uint4 c = sh_ld4(p.cell(d));
		const uint32_t np = min(c.y, p.pcap), ns = min(c.z, p.pcap);
		base_prev = base_cur;
		base_cur += c.x;
		// (the records of the levels taken fit, by the bound that chose `stop`)
		if (base_cur + 2 * c.x + ns > rcap) {
			if (threadIdx.x == 0)
				sh_or(p.flags, BATCH_FLAG_INTERNAL);
			break;
		}
		if (c.x + np + ns == 0)
			continue;
		top_level<T>(t, p, d, np, ns, base_prev, base_cur);
		__syncthreads();
	}
	__syncthreads();
	const uint32_t flags = s_word[0];
	const uint32_t open = flags & BATCH_FLAG_INTERNAL ? 0u : s_cell[stop].x, nro = min(s_word[1], rocap);
	const uint32_t np = min(s_cell[stop].y, p.pcap), ns = min(s_cell[stop].z, p.pcap);
	if (threadIdx.x < 4) {
		const uint32_t n = threadIdx.x == 0 ? open : threadIdx.x == 1 ? base_cur + nro : threadIdx.x == 2 ? np : ns;
		uint32_t *c = threadIdx.x == 0   ? &wg.ctl->lvl_cnt[stop - 1]
		              : threadIdx.x == 1 ? &wg.ctl->rec_cnt
		              : threadIdx.x == 2 ? &wg.ctl->path_cnt[stop]
		                                 : &wg.ctl->seed_cnt[stop];
		s_at[threadIdx.x] = n ? atomicAdd(c, n) : 0u;
	}
	if (threadIdx.x >= 64 && threadIdx.x < 64 + stop) {
		// what the level kernels would have counted
		const uint32_t d = threadIdx.x - 64;
		if (d + 1 < stop && s_cell[d + 1].x)
			atomicAdd(&wg.ctl->top_cnt[d], s_cell[d + 1].x);
		if (s_cell[d].z)
			atomicAdd(&wg.ctl->seed_cnt[d], s_cell[d].z);
	}
	if (threadIdx.x == 32 && flags)
		atomicOr(&wg.ctl->flags, flags);
	for (uint32_t i = threadIdx.x; i < g && q0 + i < max_q; i += TOP_THREADS) {
		wg.counts[q0 + i] = s_cnt[i];
		wg.cursor[q0 + i] = 0;
	}
	__syncthreads();
	// (the region of the last level taken starts the frontier: lvl_base is 0 there)
	const uint64_t b_open = s_at[0];
	if (b_open + open > wg.rec_cap) {
		if (threadIdx.x == 0) {
			atomicMax((unsigned long long *) &wg.ctl->need_tasks, (unsigned long long) (b_open + open));
			atomicOr(&wg.ctl->flags, BATCH_FLAG_TASK_OVERFLOW);
		}
	} else {
		for (uint32_t i = threadIdx.x; i < open; i += TOP_THREADS)
			wg.rec[b_open + i] = s_rec[base_cur + i];
	}
	const uint32_t b_ro = s_at[1];
	if (b_ro + base_cur + nro > wg.ro_cap) {
		if (threadIdx.x == 0)
			atomicOr(&wg.ctl->flags, BATCH_FLAG_INTERNAL);
	} else {
		for (uint32_t i = threadIdx.x; i < base_cur + nro; i += TOP_THREADS)
			wg.ro[b_ro + i] = i < base_cur ? s_rec[i] : s_ro[i - base_cur];
	}
	uint4 *pd = (stop & 1) ? wg.path1 : wg.path0, *sd = (stop & 1) ? wg.seed1 : wg.seed0;
	for (uint32_t i = threadIdx.x; i < np && s_at[2] + i < wg.path_cap; i += TOP_THREADS)
		pd[s_at[2] + i] = s_list[(stop & 1) * p.pcap + i];
	for (uint32_t i = threadIdx.x; i < ns && s_at[3] + i < wg.path_cap; i += TOP_THREADS)
		sd[s_at[3] + i] = s_list[(2 + (stop & 1)) * p.pcap + i];
}

// Shared memory a top-pass kernel may take beyond its static arrays on the current device,
// after allowing it for the kernel there (once per device; done before any launch is
// captured into a graph).
template <typename T>
size_t cta_pass_budget(bool groups = false)
{
	static std::mutex mu;
	static size_t budget[64][2];
	static bool done[64] = {};
	const DeviceInfo &di = device_info();
	std::lock_guard<std::mutex> lk(mu);
	if (!done[di.device]) {
		auto allow = [&](auto *kernel) {
			cudaFuncAttributes a{};
			PST_CUDA(cudaFuncGetAttributes(&a, kernel));
			const size_t b = di.smem_optin > a.sharedSizeBytes + 1024 ? di.smem_optin - a.sharedSizeBytes - 1024 : 0;
			PST_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) b));
			return b;
		};
		budget[di.device][0] = allow(k_bfs_cta<T>);
		budget[di.device][1] = allow(k_bfs_groups<T>);
		done[di.device] = true;
	}
	return budget[di.device][groups];
}

// How far k_bfs_groups goes with groups of g queries: the levels on which a CTA's records
// stay below GROUP_REC_CAP whatever the queries, and within its shared memory.  A query has
// at most a record per 64-slot block of a level and 14 more (the bound of
// NOALLOC_MAX_LEVELS).  1024 records are 16 rounds of the CTA's warps, which a level kernel
// would beat, but only queries for most of the tree come near: 64 queries for 30 % of 2^22
// points each take 260 us without the groups and 213, 210 and 210 with limits of 512, 1024
// and 2048; 601 mixed ones on 12.3 M doubles 248, and 214, 213 and 210; 4096 on 2^28 points
// 2091, and 2069, 2057 and 2070.
constexpr uint32_t GROUP_REC_CAP = 1024, GROUP_MIN_LEVELS = 6;
constexpr size_t GROUP_SMEM = size_t(200) << 10;
// Records of the first s levels of one query, and its boundary nodes.
constexpr uint32_t group_records(uint32_t s) { return (1u << s) / 32 + 14 * s + 64; }
constexpr size_t group_smem_bytes(uint32_t g, uint32_t s)
{
	return (size_t) (TOP_CELLS + g * (8 + 2 * s + group_records(s))) * sizeof(uint4) + (size_t) g * 4;
}
inline uint32_t group_levels(uint32_t levels, uint32_t g)
{
	uint32_t s = 0;
	while (s < levels && s < 20 && (uint64_t) g * ((1u << s) / 64 + 14) <= GROUP_REC_CAP &&
	       group_smem_bytes(g, s + 1) <= GROUP_SMEM)
		s++;
	return s;
}

// Launches the one-CTA top pass of at most qcap queries: two paths and two seeds for each
// in the lists, and as many records as the rest of the CTA's shared memory holds.
template <typename T>
void launch_cta_pass(const TreeDev<T> &tv, const QDev<T> &qd, const WorkDev &w, uint32_t max_q, uint32_t qcap,
                     const QOut<T> &qo, const TopIn &in, BatchCtl *back, cudaStream_t s)
{
	const size_t budget = cta_pass_budget<T>();
	const uint32_t pcap = 2 * qcap;
	const size_t fixed = cta_smem_bytes((qcap + 1) & ~1u, pcap, 0);
	// room for at least one level's records beyond the lists
	if (budget < fixed + (size_t) (2 * CTA_REC_CAP + pcap) * sizeof(uint4))
		fail(PST_ERR_INTERNAL, "shared memory too small for the top pass of " + std::to_string(max_q) + " queries");
	const uint32_t rcap = (uint32_t) ((budget - fixed) / sizeof(uint4));
	k_bfs_cta<T><<<1, TOP_THREADS, cta_smem_bytes((qcap + 1) & ~1u, pcap, rcap), s>>>(
	    tv, qd, w, max_q, (qcap + 1) & ~1u, pcap, rcap, qo, in, back);
}

// The host's copy of a pass's control block (by the whole CTA; `back` may be null).
__device__ __forceinline__ void ctl_to_host(const BatchCtl *ctl, BatchCtl *back, bool emitting = false)
{
	if (back)
		copy_ctl(ctl, back, threadIdx.x, blockDim.x, emitting);
}

// THREADS: the CTA size and U the records each warp has in flight (both tuning
// choices; point records keep U = 4).
template <typename T, bool HAS_ID, bool POINTS, int THREADS, int U>
__global__ void __launch_bounds__(THREADS) k_emit(TreeDev<T> t, WorkDev w, void *out, uint64_t capacity,
                                                 BatchCtl *back)
{
	// a programmatic dependent of the scan (a no-op after any other predecessor)
	asm volatile("griddepcontrol.wait;" ::: "memory");
	__shared__ uint64_t s_total;
	__shared__ EmitWarp<Point<T, HAS_ID>, POINTS> s_warp[THREADS / 32];
	if (blockIdx.x == 0)
		ctl_to_host(w.ctl, back, true);
	if (threadIdx.x == 0) {
		uint64_t b = 0;
		for (uint32_t e = 0; e < t.levels; e++)
			b += w.ctl->lvl_cnt[e];
		s_total = b;
	}
	__syncthreads();
	if (w.ctl->total > capacity || (w.ctl->flags & (w.ctl->waits ? BATCH_FLAGS_FAILED : BATCH_FLAG_TASK_OVERFLOW))) {
		if (blockIdx.x == 0 && threadIdx.x == 0 && w.ctl->total > capacity)
			atomicOr(&w.ctl->flags, BATCH_FLAG_OUT_OVERFLOW);
		return;
	}
	const uint64_t total = s_total < w.rec_cap ? s_total : w.rec_cap;
	const uint32_t nro = min(w.ctl->rec_cnt, w.ro_cap);
	const uint32_t lane = lane_id();
	const uint64_t gtid = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x;
	const uint64_t gwarps = (uint64_t) gridDim.x * blockDim.x / 32, gwarp = gtid / 32;
	// Two batches in flight: the next batch's records are read and its output claimed
	// (an atomic whose result is needed only one batch later) before this batch's
	// results are written.
	const uint64_t stride = gwarps * 32;
	uint64_t wb = gwarp * 32;
	bool v0 = wb + lane < total;
	uint4 m0 = v0 ? w.rec[wb + lane] : make_uint4(0, 0, 0, 0);
	uint64_t ob0 = wb < total ? claim_output(w, m0.y, __popc(m0.z) + __popc(m0.w), v0) : 0;
	guard_claim(w, m0, ob0, capacity);
	while (wb < total) {
		const uint64_t nb = wb + stride;
		const bool v1 = nb + lane < total;
		uint4 m1 = v1 ? w.rec[nb + lane] : make_uint4(0, 0, 0, 0);
		const uint64_t ob1 = nb < total ? claim_output(w, m1.y, __popc(m1.z) + __popc(m1.w), v1) : 0;
		guard_claim(w, m1, ob1, capacity);
		emit_blocks<T, HAS_ID, POINTS, U>(t, m0, ob0, v0, s_warp[threadIdx.x >> 5], out);
		wb = nb;
		v0 = v1;
		m0 = m1;
		ob0 = ob1;
	}
	for (uint64_t wb = gwarp * 32; wb < nro; wb += gwarps * 32) {
		const bool valid = wb + lane < nro;
		uint4 mine = valid ? w.ro[wb + lane] : make_uint4(0, 0, 0, 0);
		const uint64_t ob = claim_output(w, mine.y, __popc(mine.z) + __popc(mine.w), valid);
		guard_claim(w, mine, ob, capacity);
		emit_blocks<T, HAS_ID, POINTS, U>(t, mine, ob, valid, s_warp[threadIdx.x >> 5], out);
	}
}

// Result offsets of a batch in one launch: offsets[q] = the counts of the queries
// before q, offsets[max_q] = ctl->total = all of them.  One CTA walks the counts a
// tile at a time (batches of up to OFFSETS_ONE_CTA queries; larger ones take the
// three-kernel scan and k_pass_end).  Launched as a programmatic dependent of the last
// level.  It also writes the caller's offsets and the host's copy of the control block,
// which spares a copy of each (2 to 3 us on the device).
constexpr uint32_t OFFSETS_ONE_CTA = 4 * SCAN_TILE;

__global__ void __launch_bounds__(SCAN_THREADS) k_offsets(const uint64_t *counts, uint64_t *offsets, uint32_t n,
                                                          BatchCtl *ctl, BatchCtl *back)
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	__shared__ uint64_t ws[33];
	const uint32_t nq = ctl->nq;
	uint64_t *user = ctl->waits && (ctl->flags & BATCH_FLAGS_FAILED) ? nullptr : ctl->user_offsets;
	uint64_t carry = 0;
	for (uint32_t c0 = 0; c0 < n; c0 += SCAN_TILE) {
		const uint32_t base = c0 + threadIdx.x * SCAN_ITEMS;
		uint64_t v[SCAN_ITEMS];
		uint64_t sum = 0;
#pragma unroll
		for (int i = 0; i < SCAN_ITEMS; i++) {
			v[i] = base + i < n ? counts[base + i] : 0;
			sum += v[i];
		}
		uint64_t tot;
		uint64_t ex = block_excl_scan(sum, &tot, ws) + carry;
#pragma unroll
		for (int i = 0; i < SCAN_ITEMS; i++) {
			if (base + i < n)
				offsets[base + i] = ex;
			if (user && base + i < n && base + i <= nq)
				user[base + i] = ex;
			ex += v[i];
		}
		carry += tot;
	}
	if (threadIdx.x == 0) {
		offsets[n] = carry;
		if (user && nq == n)
			user[n] = carry;
		ctl->total = carry;
	}
	__syncthreads();
	if (!ctl->emit_follows)
		ctl_to_host(ctl, back);
}

// The end of a pass of more queries, after its scan.
__global__ void __launch_bounds__(SCAN_THREADS) k_pass_end(const uint64_t *offsets, const BatchCtl *ctl, BatchCtl *back)
{
	if (ctl->user_offsets && !(ctl->waits && (ctl->flags & BATCH_FLAGS_FAILED)))
		for (uint64_t q = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; q <= ctl->nq; q += (uint64_t) gridDim.x * blockDim.x)
			ctl->user_offsets[q] = offsets[q];
	if (blockIdx.x == 0 && !ctl->emit_follows)
		ctl_to_host(ctl, back);
}

// Launch configuration of a programmatic dependent of the kernel before it on `s`:
// its CTAs may be scheduled while that kernel drains, and wait (griddepcontrol.wait)
// until it has completed and its writes are visible.
struct DependentLaunch {
	cudaLaunchConfig_t cfg{};
	cudaLaunchAttribute attr[1];
	DependentLaunch(unsigned grid, unsigned threads, cudaStream_t s)
	{
		cfg.gridDim = dim3(grid);
		cfg.blockDim = dim3(threads);
		cfg.dynamicSmemBytes = 0;
		cfg.stream = s;
		attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[0].val.programmaticStreamSerializationAllowed = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
	}
};

// The batch's result offsets and total (exclusive scan of its counts).
inline void scan_offsets(uint64_t *counts, uint64_t *offsets, uint32_t max_q, uint64_t *scan_tmp, BatchCtl *ctl,
                         BatchCtl *back, cudaStream_t s)
{
	if (max_q <= OFFSETS_ONE_CTA) {
		DependentLaunch l(1, SCAN_THREADS, s);
		PST_CUDA(cudaLaunchKernelEx(&l.cfg, k_offsets, (const uint64_t *) counts, offsets, max_q, ctl, back));
		return;
	}
	exclusive_scan<uint64_t>(counts, offsets, max_q, scan_tmp, &ctl->total, s);
	PST_CUDA(cudaMemcpyAsync(offsets + max_q, &ctl->total, 8, cudaMemcpyDeviceToDevice, s));
	k_pass_end<<<32, SCAN_THREADS, 0, s>>>(offsets, ctl, back);
	PST_CUDA(cudaGetLastError());
}

// Grid of k_emit: as many CTAs as fit on the device at once (its own occupancy,
// which can differ from the level kernel's), so the grid-stride loop has no tail wave.
template <typename T, bool HAS_ID, bool POINTS, int THREADS, int U>
unsigned emit_grid()
{
	static const int occ = [] {
		int o = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_emit<T, HAS_ID, POINTS, THREADS, U>, THREADS, 0) !=
		    cudaSuccess) {
			cudaGetLastError();
			o = 1;
		}
		return o > 0 ? o : 1;
	}();
	return (unsigned) (device_info().sms * occ);
}

template <typename T>
void launch_level(const TreeDev<T> &tv, const QDev<T> &qd, const WorkDev &w, uint32_t d, unsigned grid,
                  unsigned threads, cudaStream_t s)
{
	// a programmatic dependent launch: the level's CTAs start as the previous kernel
	// drains (the kernel waits for it before reading anything)
	DependentLaunch l(grid, threads, s);
	cudaLaunchConfig_t &cfg = l.cfg;
	const bool last = d + 1 == tv.levels && tv.last_par;
	switch (threads) {
	case 128:
		PST_CUDA(last ? cudaLaunchKernelEx(&cfg, k_bfs_level<T, true, 128>, tv, qd, w, d)
		              : cudaLaunchKernelEx(&cfg, k_bfs_level<T, false, 128>, tv, qd, w, d));
		break;
	case 512:
		PST_CUDA(last ? cudaLaunchKernelEx(&cfg, k_bfs_level<T, true, 512>, tv, qd, w, d)
		              : cudaLaunchKernelEx(&cfg, k_bfs_level<T, false, 512>, tv, qd, w, d));
		break;
	default:
		PST_CUDA(last ? cudaLaunchKernelEx(&cfg, k_bfs_level<T, true, BFS_THREADS>, tv, qd, w, d)
		              : cudaLaunchKernelEx(&cfg, k_bfs_level<T, false, BFS_THREADS>, tv, qd, w, d));
	}
}

template <typename T>
const void *bfs_kernel_ptr(unsigned threads)
{
	switch (threads) {
	case 128: return reinterpret_cast<const void *>(&k_bfs_level<T, false, 128>);
	case 512: return reinterpret_cast<const void *>(&k_bfs_level<T, false, 512>);
	default: return reinterpret_cast<const void *>(&k_bfs_level<T, false, BFS_THREADS>);
	}
}

// Launches the emit with the batch's CTA size and records in flight.
template <typename T, bool HAS_ID, bool POINTS, int THREADS, int U>
void launch_emit_tu(const TreeDev<T> &tv, const WorkDev &w, void *out, uint64_t capacity, BatchCtl *back, cudaStream_t s)
{
	DependentLaunch l(emit_grid<T, HAS_ID, POINTS, THREADS, U>(), THREADS, s);
	PST_CUDA(cudaLaunchKernelEx(&l.cfg, k_emit<T, HAS_ID, POINTS, THREADS, U>, tv, w, out, capacity, back));
}

template <typename T, bool HAS_ID, bool POINTS, int THREADS>
void launch_emit_t(const TreeDev<T> &tv, const WorkDev &w, void *out, uint64_t capacity, uint32_t u, BatchCtl *back,
                   cudaStream_t s)
{
	if constexpr (POINTS) {
		(void) u;
		launch_emit_tu<T, HAS_ID, POINTS, THREADS, 4>(tv, w, out, capacity, back, s);
	} else if (u == 4) {
		launch_emit_tu<T, HAS_ID, POINTS, THREADS, 4>(tv, w, out, capacity, back, s);
	} else if (u == 16) {
		launch_emit_tu<T, HAS_ID, POINTS, THREADS, 16>(tv, w, out, capacity, back, s);
	} else {
		launch_emit_tu<T, HAS_ID, POINTS, THREADS, 8>(tv, w, out, capacity, back, s);
	}
}

template <typename T, bool HAS_ID, bool POINTS>
void launch_emit(const TreeDev<T> &tv, const WorkDev &w, void *out, uint64_t capacity, uint32_t threads, uint32_t u,
                 BatchCtl *back, cudaStream_t s)
{
	switch (threads) {
	case 128: launch_emit_t<T, HAS_ID, POINTS, 128>(tv, w, out, capacity, u, back, s); break;
	case 512: launch_emit_t<T, HAS_ID, POINTS, 512>(tv, w, out, capacity, u, back, s); break;
	default: launch_emit_t<T, HAS_ID, POINTS, BFS_THREADS>(tv, w, out, capacity, u, back, s);
	}
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side.

Batch::~Batch() { release(); }

void Batch::Graph::drop()
{
	if (exec)
		cudaGraphExecDestroy(exec);
	exec = nullptr;
}

void Batch::release()
{
	full_graph.drop();
	if (open)
		wait_for_device(device);  // a call that failed with some of its kernels queued, or a server's
	if (passes)
		passes->wait(this);  // an asynchronous pass may still use the buffers
	pool_release(work, device);
	pool_release(rec, device);
	for (void *p : captured_recs)
		pool_release(p, device);
	captured_recs.clear();
	work = nullptr;
	pinned_release(ctl_host, device);  // the staged queries lie behind the control block
	ctl_host = nullptr;
	ctl_host_d = nullptr;
	q_stage = nullptr;
	rec = nullptr;
}

void Batch::init(TreeStorage *t, const pst_batch_opts &o)
{
	tree = t;
	passes = t->passes;
	device = device_info().device;
	max_q = std::max<uint32_t>(o.max_queries, 1);
	use_graph = o.use_graph != 0;
	threads = o.block_threads ? o.block_threads : BFS_THREADS;
	if (threads != 128 && threads != 256 && threads != 512)
		fail(PST_ERR_INVALID, "block_threads must be 0, 128, 256 or 512");
	emit_u = o.emit_records ? o.emit_records : 8;
	if (emit_u != 4 && emit_u != 8 && emit_u != 16)
		fail(PST_ERR_INVALID, "emit_records must be 0, 4, 8 or 16");
	top_q = o.top_pass_queries ? o.top_pass_queries : SMALL_BATCH_Q;
	if (top_q > MAX_TOP_PASS_Q)
		fail(PST_ERR_INVALID, "top_pass_queries must be at most " + std::to_string(MAX_TOP_PASS_Q));
	int occ = 0;
	const void *kfn = nullptr;
	switch (t->dtype) {
	case PST_F32: kfn = bfs_kernel_ptr<float>(threads); cta_pass_budget<float>(); break;
	case PST_F64: kfn = bfs_kernel_ptr<double>(threads); cta_pass_budget<double>(); break;
	case PST_I32: kfn = bfs_kernel_ptr<int32_t>(threads); cta_pass_budget<int32_t>(); break;
	}
	PST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kfn, threads, 0));
	blocks_per_sm = o.blocks_per_sm ? std::min<uint32_t>(o.blocks_per_sm, (uint32_t) std::max(occ, 1))
	                                : (uint32_t) std::max(occ, 1);
	grid = (uint32_t) device_info().sms * blocks_per_sm;
	const size_t vs = value_size(t->dtype);
	path_cap = 2 * max_q;
	// groups of queries for the first levels of a whole pass, a CTA each; for a batch of any
	// size, also where waiting ones start with the one-CTA pass (1, 4, 16 and 32 isovalues,
	// asynchronously: 124, 124, 130 and 134 us on 2^21 points by levels alone, 86, 91, 89
	// and 88 this way; on 2^26 145, 155, 230 and 292, and 110, 122, 189 and 245)
	group = (max_q + (uint32_t) device_info().sms - 1) / (uint32_t) device_info().sms;
	group_stop = group_levels(t->levels, group);
	if (group_stop < GROUP_MIN_LEVELS)
		group_stop = 0;
	ro_cap = max_q * (2 * 32 + (group_stop ? group_records(group_stop) : 0));
	{
		// laid out twice: once for the size, once for the addresses
		size_t off = 0;
		auto take = [&](auto **p, size_t bytes) {
			if (work)
				*p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(static_cast<char *>(work) + off);
			off += (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
		};
		auto layout = [&] {
			off = 0;
			take(&q_copy, (size_t) max_q * sizeof(pst_query));
			take(&kind, (size_t) max_q * 4);
			take(&min1, (size_t) max_q * vs);
			take(&max1, (size_t) max_q * vs);
			take(&min2, (size_t) max_q * vs);
			take(&path0, (size_t) path_cap * sizeof(uint4));
			take(&path1, (size_t) path_cap * sizeof(uint4));
			take(&seed0, (size_t) path_cap * sizeof(uint4));
			take(&seed1, (size_t) path_cap * sizeof(uint4));
			take(&ro, (size_t) ro_cap * sizeof(uint4));
			take(&counts, (size_t) max_q * 8);
			take(&cursor, (size_t) max_q * 8);
			take(&offsets, ((size_t) max_q + 1) * 8);
			take(&scan_tmp, scan_tmp_elems(max_q) * 8);
			take(&ctl, sizeof(BatchCtl));
		};
		layout();
		work = pool_alloc(off, "batch workspace");
		layout();
	}
	const size_t head = 2 * sizeof(BatchCtl);
	ctl_host = static_cast<BatchCtl *>(pinned_alloc(head + (size_t) max_q * sizeof(pst_query), "query staging"));
	back = ctl_host + 1;
	q_stage = reinterpret_cast<pst_query *>(back + 1);
	memset(ctl_host, 0, head);
	void *mapped = nullptr;
	PST_CUDA(cudaHostGetDevicePointer(&mapped, ctl_host, 0));
	BatchCtl *ctl_d = static_cast<BatchCtl *>(mapped);
	ctl_host_d = ctl_d;
	back_d = ctl_d + 1;
	q_stage_d = reinterpret_cast<const pst_query *>(back_d + 1);
	idle = true;
	const uint64_t want = o.task_capacity ? o.task_capacity : std::max<uint64_t>(1ull << 16, (uint64_t) max_q * 64);
	rec = static_cast<uint4 *>(pool_alloc(want * sizeof(uint4), "frontier"));
	task_cap = want;
}

void Batch::grow_tasks(uint64_t cap, cudaStream_t s)
{
	if (captured) {
		// a graph of the caller's holds the old frontier's address
		captured_recs.push_back(rec);
	} else {
		// Only the passes that used the old frontier are waited for (those on `s`, and an
		// asynchronous one), not work on the device's other streams.
		PST_CUDA(cudaStreamSynchronize(s));
		passes->wait(this);
		pool_release(rec, device);
	}
	rec = nullptr;
	task_cap = 0;
	rec = static_cast<uint4 *>(pool_alloc(cap * sizeof(uint4), "frontier"));
	task_cap = cap;
	// the captured passes hold the old frontier's address
	full_graph.drop();
}

#define PST_WORKDEV                                                                                                   \
	WorkDev w{rec, task_cap, path0, path1, seed0, seed1, path_cap, ro, ro_cap, counts, cursor, offsets, ctl}

template <typename T>
void Batch::enqueue_count(cudaStream_t s, const PassStart *own)
{
	TreeDev<T> tv = tree->view<T>();
	QDev<T> qd{kind, static_cast<const T *>(min1), static_cast<const T *>(max1), static_cast<const T *>(min2)};
	PST_WORKDEV;
	if (own)
		k_set_ctl<<<1, 256, 0, s>>>(ctl, *own);
	else
		k_load_ctl<<<1, 256, 0, s>>>(ctl_host_d, ctl);
	const QOut<T> qo{kind, static_cast<T *>(min1), static_cast<T *>(max1), static_cast<T *>(min2)};
	if (group_stop) {
		const uint32_t rocap = 2 * group_stop * group, rcap = group * group_records(group_stop);
		DependentLaunch l((max_q + group - 1) / group, TOP_THREADS, s);
		l.cfg.dynamicSmemBytes = group_smem_bytes(group, group_stop);
		if (l.cfg.dynamicSmemBytes > cta_pass_budget<T>(true))
			fail(PST_ERR_INTERNAL, "shared memory too small for groups of " + std::to_string(group) + " queries");
		PST_CUDA(cudaLaunchKernelEx(&l.cfg, k_bfs_groups<T>, tv, qd, w, qo, max_q, group, rocap, rcap, group_stop));
	} else {
		const unsigned ug = (unsigned) std::min<uint64_t>((max_q + 255) / 256, (uint64_t) device_info().sms * 4);
		k_prepare_queries<T><<<ug, 256, 0, s>>>(ctl, qo, path0, counts, cursor, max_q);
	}
	for (uint32_t d = group_stop; d < tv.levels; d++)
		launch_level<T>(tv, qd, w, d, grid, threads, s);
	scan_offsets(counts, offsets, max_q, scan_tmp, ctl, own ? nullptr : back_d, s);
	PST_CUDA(cudaGetLastError());
}

template <typename T>
void Batch::enqueue_count_top(cudaStream_t s)
{
	TreeDev<T> tv = tree->view<T>();
	QDev<T> qd{kind, static_cast<const T *>(min1), static_cast<const T *>(max1), static_cast<const T *>(min2)};
	PST_WORKDEV;
	// one kernel: the queries unpacked and the whole top pass
	const QOut<T> qo{kind, static_cast<T *>(min1), static_cast<T *>(max1), static_cast<T *>(min2)};
	launch_cta_pass<T>(tv, qd, w, max_q, std::min(top_q, max_q), qo, top_in, back_d, s);
	PST_CUDA(cudaGetLastError());
}

template <typename T>
void Batch::enqueue_count_rest(uint32_t from, cudaStream_t s)
{
	TreeDev<T> tv = tree->view<T>();
	QDev<T> qd{kind, static_cast<const T *>(min1), static_cast<const T *>(max1), static_cast<const T *>(min2)};
	PST_WORKDEV;
	for (uint32_t d = from; d < tv.levels; d++)
		launch_level<T>(tv, qd, w, d, grid, threads, s);
	scan_offsets(counts, offsets, max_q, scan_tmp, ctl, back_d, s);
	PST_CUDA(cudaGetLastError());
}

template <typename T, bool HAS_ID, bool POINTS>
void Batch::enqueue_emit_t(void *out, uint64_t capacity, cudaStream_t s, bool to_host)
{
	TreeDev<T> tv = tree->view<T>();
	PST_WORKDEV;
	launch_emit<T, HAS_ID, POINTS>(tv, w, out, capacity, threads, emit_u, to_host ? back_d : nullptr, s);
	PST_CUDA(cudaGetLastError());
}

template <typename T>
void Batch::enqueue_emit_v(pst_ret ret, void *out, uint64_t capacity, cudaStream_t s, bool to_host)
{
	const bool has_id = tree->idtype == PST_ID_U32;
	if (ret == PST_RET_IDS) {
		if (!has_id)
			fail(PST_ERR_UNSUPPORTED, "an id-less tree can only return points");
		enqueue_emit_t<T, true, false>(out, capacity, s, to_host);
	} else if (has_id) {
		enqueue_emit_t<T, true, true>(out, capacity, s, to_host);
	} else {
		enqueue_emit_t<T, false, true>(out, capacity, s, to_host);
	}
}

void Batch::enqueue_counting(cudaStream_t s, const PassStart *own)
{
	switch (tree->dtype) {
	case PST_F32: enqueue_count<float>(s, own); break;
	case PST_F64: enqueue_count<double>(s, own); break;
	case PST_I32: enqueue_count<int32_t>(s, own); break;
	}
}

void Batch::enqueue_counting_top(cudaStream_t s)
{
	switch (tree->dtype) {
	case PST_F32: enqueue_count_top<float>(s); break;
	case PST_F64: enqueue_count_top<double>(s); break;
	case PST_I32: enqueue_count_top<int32_t>(s); break;
	}
}

void Batch::enqueue_emit(pst_ret ret, void *out, uint64_t capacity, cudaStream_t s, bool to_host)
{
	open = true;
	switch (tree->dtype) {
	case PST_F32: enqueue_emit_v<float>(ret, out, capacity, s, to_host); break;
	case PST_F64: enqueue_emit_v<double>(ret, out, capacity, s, to_host); break;
	case PST_I32: enqueue_emit_v<int32_t>(ret, out, capacity, s, to_host); break;
	}
}

void Batch::capture_next(cudaStream_t s)
{
	full_graph.drop();
	full_graph.stream = s;
	full_graph.direct = DIRECT_PASSES;
}

void Batch::launch_count(cudaStream_t s)
{
	Graph &g = full_graph;
	open = true;
	// an engine's first passes on a stream are launched as they are: capturing one and
	// destroying it again takes 310 us, many engines live for a query or two, and a replay
	// saves 60 us of host time
	if (!use_graph || g.stream != s || g.direct < DIRECT_PASSES) {
		if (g.stream != s)
			g.direct = 0;
		g.drop();
		g.direct++;
		g.stream = s;
		enqueue_counting(s);
		return;
	}
	if (!g.exec) {
		cudaStream_t cs;
		PST_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
		cudaGraph_t gr;
		PST_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
		try {
			enqueue_counting(cs);
		} catch (...) {
			cudaStreamEndCapture(cs, &gr);
			cudaStreamDestroy(cs);
			throw;
		}
		PST_CUDA(cudaStreamEndCapture(cs, &gr));
		PST_CUDA(cudaGraphInstantiate(&g.exec, gr, 0));
		cudaGraphDestroy(gr);
		cudaStreamDestroy(cs);
	}
	PST_CUDA(cudaGraphLaunch(g.exec, s));
}

bool Batch::run_captured(const pst_query *q, uint32_t nq, bool on_device, pst_ret ret, void *out, uint64_t capacity,
                         uint64_t *to_offsets, cudaStream_t s)
{
	cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
	PST_CUDA(cudaStreamIsCapturing(s, &st));
	if (st == cudaStreamCaptureStatusNone)
		return false;
	check_queries(q, nq);
	if (!on_device && nq)
		fail(PST_ERR_UNSUPPORTED, "the queries of a pass that is captured into a graph must be a device array");
	// Nothing of the pass is the engine's to change later: its queries' and offsets' places
	// are kernel parameters, the kernels are the caller's graph's own, and the frontier stays
	// (grow_tasks).  The block that the host waits with is left alone: a pass before this one
	// may still use it.
	captured = true;
	passes->mark(this, s);
	const PassStart own = place(q, nq, on_device, to_offsets, s);
	enqueue_counting(s, &own);
	enqueue_emit(ret, out, capacity, s);
	copy_offsets(nq, s);
	return true;
}

void Batch::launch_count_top(cudaStream_t s)
{
	if (ctl_host->nq > top_q)
		fail(PST_ERR_INTERNAL, "top pass on a batch of more than " + std::to_string(top_q) + " queries");
	open = true;
	enqueue_counting_top(s);
}

void Batch::launch_count_rest(uint32_t from, cudaStream_t s)
{
	open = true;
	switch (tree->dtype) {
	case PST_F32: enqueue_count_rest<float>(from, s); break;
	case PST_F64: enqueue_count_rest<double>(from, s); break;
	case PST_I32: enqueue_count_rest<int32_t>(from, s); break;
	}
}

void Batch::check_queries(const pst_query *q, uint32_t nq) const
{
	if (nq > max_q)
		fail(PST_ERR_INVALID, "batch of " + std::to_string(nq) + " queries exceeds max_queries " +
		                          std::to_string(max_q));
	if (nq && !q)
		fail(PST_ERR_INVALID, "null query array");
}

// Whether kernels of the engine's device can use the caller's array of 8-byte words where
// it is: an array of another device may be out of their reach, and an address that is not
// a multiple of 8 would end the context.
static bool usable_in_place(const void *p, int device)
{
	if (reinterpret_cast<uintptr_t>(p) & 7u)
		return false;
	cudaPointerAttributes a{};
	if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	return a.type == cudaMemoryTypeDevice ? a.device == device : a.type != cudaMemoryTypeUnregistered && a.devicePointer == p;
}

// Where the pass finds its queries and leaves the caller's offsets: the caller's arrays
// themselves where kernels can use them (a copy of each costs 2 to 3 us), the staged
// queries through their mapping, or else copies.
PassStart Batch::place(const pst_query *q, uint32_t nq, bool on_device, uint64_t *to_offsets, cudaStream_t s)
{
	PassStart at{nq, q, to_offsets};
	copy_offsets_to = nullptr;
	if (!on_device) {
		if (nq)
			memcpy(q_stage, q, (size_t) nq * sizeof(pst_query));
		at.raw = q_stage_d;
	} else if (nq && !usable_in_place(q, device)) {
		PST_CUDA(cudaMemcpyAsync(q_copy, q, (size_t) nq * sizeof(pst_query), cudaMemcpyDeviceToDevice, s));
		at.raw = q_copy;
	}
	if (to_offsets && !usable_in_place(to_offsets, device)) {
		copy_offsets_to = to_offsets;
		at.offsets = nullptr;
	}
	return at;
}

bool Batch::copy_offsets(uint32_t nq, cudaStream_t s)
{
	if (!copy_offsets_to)
		return false;
	PST_CUDA(cudaMemcpyAsync(copy_offsets_to, offsets, ((size_t) nq + 1) * 8, cudaMemcpyDeviceToDevice, s));
	return true;
}

void Batch::stage_queries(const pst_query *q, uint32_t nq, bool on_device, cudaStream_t s, uint64_t *to_offsets)
{
	check_queries(q, nq);
	// the pinned control block and query staging may still feed an earlier pass
	if (!idle)
		PST_CUDA(cudaStreamSynchronize(s));
	idle = false;
	const PassStart at = place(q, nq, on_device, to_offsets, s);
	ctl_host->nq = nq;
	ctl_host->raw = at.raw;
	ctl_host->user_offsets = at.offsets;
	ctl_host->host_fault = &back_d->fault;
	ctl_host->emit_follows = 0;
	ctl_host->waits = 0;
	back->fault = 0;
	top_in.args = TopArgs{};
	top_in.args.nq = nq;
	top_in.args.offsets = at.offsets;
	if (!on_device && nq <= TOP_IN_QUERIES)
		std::copy(q, q + nq, top_in.q);
	else
		top_in.args.raw = ctl_host->raw;
}

pst_status Batch::last_status() const
{
	if (last.flags & BATCH_FLAG_BAD_QUERY)
		return PST_ERR_INVALID;
	if (last.flags & (BATCH_FLAG_TASK_OVERFLOW | BATCH_FLAG_INTERNAL))
		return PST_ERR_INTERNAL;
	if (last.flags & BATCH_FLAG_OUT_OVERFLOW)
		return PST_ERR_CAPACITY;
	return PST_OK;
}

pst_status Batch::read_ctl(cudaStream_t s, uint64_t *total)
{
	PST_CUDA(cudaMemcpyAsync(&last, ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (total)
		*total = last.total;
	return last_status();
}

pst_status Batch::finish(cudaStream_t s)
{
	PST_CUDA(cudaStreamSynchronize(s));
	last = *back;
	if (last.fault)
		last.flags |= BATCH_FLAG_INTERNAL;
	idle = true;
	open = false;
	return last_status();
}

// Count pass with the host waiting for it.
void Batch::count_sync(cudaStream_t s, uint64_t *total, const EmitTo *to)
{
	if (ctl_host->nq <= top_q)
		count_small_sync(s, total, to);
	else
		count_full_sync(s, total, to);
}

// Looks at a finished pass (b.last); true when it is complete, false when the frontier
// overflowed (and has been grown for another attempt).
static bool settle(Batch &b, int attempt, cudaStream_t s, uint64_t *total)
{
	const BatchCtl &h = b.last;
	if (h.flags & BATCH_FLAG_BAD_QUERY)
		fail(PST_ERR_INVALID, "query kind must be PST_Q_THREE, PST_Q_LEFT or PST_Q_RIGHT");
	if (h.flags & BATCH_FLAG_INTERNAL)
		fail(PST_ERR_INTERNAL, "search consistency check failed");
	if (!(h.flags & BATCH_FLAG_TASK_OVERFLOW)) {
		*total = h.total;
		return true;
	}
	if (attempt > 8)
		fail(PST_ERR_INTERNAL, "frontier did not fit after growth");
	b.grow_tasks(std::max<uint64_t>(h.need_tasks + h.need_tasks / 4, b.task_cap * 2), s);
	return false;
}

// The whole pass, with automatic growth of the frontier buffer.  An emit queued behind a
// count pass writes nothing when the pass failed, did not fit the frontier or its results
// the buffer.
void Batch::count_full_sync(cudaStream_t s, uint64_t *total, const EmitTo *to)
{
	const bool emits = to && to->out && to->capacity;
	ctl_host->emit_follows = emits;
	ctl_host->waits = 1;
	for (int attempt = 0;; attempt++) {
		launch_count(s);
		if (emits)
			enqueue_emit(to->ret, to->out, to->capacity, s, true);
		finish(s);
		if (settle(*this, attempt, s, total))
			return;
	}
}

// A small batch: the one-CTA top pass, then, if it stopped above the bottom, the
// per-level kernels for the rest and the scan; with automatic growth of the
// frontier buffer as in count_full_sync.
void Batch::count_small_sync(cudaStream_t s, uint64_t *total, const EmitTo *to)
{
	const bool emits = to && to->out && to->capacity;
	if (emits) {
		top_in.args.out = to->out;
		top_in.args.out_cap = to->capacity;
		top_in.args.ret = to->ret;
	}
	for (int attempt = 0;; attempt++) {
		launch_count_top(s);
		finish(s);
		if (!(last.flags & (BATCH_FLAG_BAD_QUERY | BATCH_FLAG_INTERNAL | BATCH_FLAG_TASK_OVERFLOW))) {
			const bool rest = last.cta_levels < tree->levels;
			if (rest)
				launch_count_rest(last.cta_levels, s);
			const bool emit = emits && (rest || (!last.emitted && last.total && last.total <= to->capacity));
			if (emit)
				enqueue_emit(to->ret, to->out, to->capacity, s, true);
			if (rest || emit)
				finish(s);
		}
		if (settle(*this, attempt, s, total))
			return;
	}
}

uint64_t Batch::record_size(pst_ret ret) const
{
	return ret == PST_RET_IDS ? 4 : point_size(tree->dtype, tree->idtype);
}

// ---------------------------------------------------------------------------
// Single query with no allocation at all (pst_search_noalloc).
//
// For callers that cannot allocate device memory during a search: code whose
// device memory is all owned by its own allocator (so a cudaMalloc here would fail
// or compete with it), and latency-critical loops that cannot take the implicit
// device-wide synchronisation of cudaMalloc/cudaFree.  The search's working memory
// (control block, the query, its boundary paths and its frontier) lives in the
// file-scope array below, which every GPU that loads this library holds until the
// process exits.

namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = size_t(8) << 20;  // 8 MiB per device
constexpr uint32_t NOALLOC_MAX_LEVELS = 22;                  // trees of up to 2^22 - 1 points

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

// Sub-buffers of the scratch array, 256-byte aligned, in bytes.
constexpr size_t NA_CTL = 0;
constexpr size_t NA_KIND = 1280;
constexpr size_t NA_MIN1 = NA_KIND + 256;
constexpr size_t NA_MAX1 = NA_MIN1 + 256;
constexpr size_t NA_MIN2 = NA_MAX1 + 256;
constexpr size_t NA_PATH0 = NA_MIN2 + 256;
constexpr size_t NA_PATH1 = NA_PATH0 + 256;
constexpr size_t NA_SEED0 = NA_PATH1 + 256;
constexpr size_t NA_SEED1 = NA_SEED0 + 256;
constexpr uint32_t NA_RO_CAP = 2 * 32;  // two boundary results per level
constexpr size_t NA_RO = NA_SEED1 + 256;
constexpr size_t NA_COUNTS = NA_RO + NA_RO_CAP * sizeof(uint4);
constexpr size_t NA_CURSOR = NA_COUNTS + 256;
constexpr size_t NA_OFFSETS = NA_CURSOR + 256;
constexpr size_t NA_SCAN = NA_OFFSETS + 256;
constexpr size_t NA_RECS = NA_SCAN + 256;
// alive records (16 B each) take the rest
constexpr uint64_t NA_REC_CAP = (NOALLOC_SCRATCH_BYTES - NA_RECS) / sizeof(uint4) / 64 * 64;
static_assert(sizeof(BatchCtl) <= NA_KIND, "control block");
static_assert(NA_RECS + NA_REC_CAP * sizeof(uint4) <= NOALLOC_SCRATCH_BYTES, "scratch layout");
// One query has at most one alive record per 64-slot block of every level, plus the
// records of report-above subtrees that still share a block with another subtree:
// a seed's subtree shares blocks for its first six levels and a query leaves at
// most two seeds per level, so at most 12 more per level: fewer than
// 2^L/32 + 14L + 64 records for a tree of L levels.
static_assert((1ull << NOALLOC_MAX_LEVELS) / 32 + 14 * NOALLOC_MAX_LEVELS + 64 <= NA_REC_CAP, "frontier bound");

std::mutex g_noalloc_mu;

// The scratch array's device address per device, with the id of the context it was
// looked up in.  cudaDeviceReset ends that context (and the array with it); the next
// call on the device, in the new context, looks the address up again.
struct NoallocSlot {
	unsigned long long ctx = 0;
	unsigned char *ptr = nullptr;
};
NoallocSlot g_noalloc_slot[64];

// Device address of the scratch array for device `dev`, which must be current
// (the host-side name of a __device__ array is only a stand-in for it): looked up
// once per device and context.
unsigned char *noalloc_scratch(int dev)
{
	if (dev < 0 || dev >= 64)
		fail(PST_ERR_CUDA, "device index out of range");
	const unsigned long long ctx = current_context_id(dev);
	NoallocSlot &slot = g_noalloc_slot[dev];
	if (!slot.ptr || slot.ctx != ctx) {
		void *p = nullptr;
		check_cuda(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(no-alloc scratch)");
		slot.ptr = static_cast<unsigned char *>(p);
		slot.ctx = ctx;
	}
	return slot.ptr;
}

template <typename T>
uint64_t noalloc_run(TreeStorage &t, const pst_query &q, pst_ret ret, void *out, uint64_t capacity, cudaStream_t s,
                     unsigned char *base)
{
	BatchCtl *ctl = reinterpret_cast<BatchCtl *>(base + NA_CTL);
	uint32_t *kind = reinterpret_cast<uint32_t *>(base + NA_KIND);
	T *min1 = reinterpret_cast<T *>(base + NA_MIN1);
	T *max1 = reinterpret_cast<T *>(base + NA_MAX1);
	T *min2 = reinterpret_cast<T *>(base + NA_MIN2);
	uint4 *path0 = reinterpret_cast<uint4 *>(base + NA_PATH0);
	uint4 *path1 = reinterpret_cast<uint4 *>(base + NA_PATH1);
	uint4 *seed0 = reinterpret_cast<uint4 *>(base + NA_SEED0);
	uint4 *seed1 = reinterpret_cast<uint4 *>(base + NA_SEED1);
	uint4 *ro = reinterpret_cast<uint4 *>(base + NA_RO);
	uint64_t *counts = reinterpret_cast<uint64_t *>(base + NA_COUNTS);
	uint64_t *cursor = reinterpret_cast<uint64_t *>(base + NA_CURSOR);
	uint64_t *offsets = reinterpret_cast<uint64_t *>(base + NA_OFFSETS);
	uint64_t *scan = reinterpret_cast<uint64_t *>(base + NA_SCAN);
	uint4 *rec = reinterpret_cast<uint4 *>(base + NA_RECS);

	// The array keeps the previous call's contents: the top pass starts the control block,
	// the query's count and its output cursor over.
	BatchCtl h{};
	TopIn in{};
	in.q[0] = q;
	in.args.nq = 1;
	in.args.out = out;
	in.args.out_cap = capacity;
	in.args.ret = ret;

	int occ = 0;
	PST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, bfs_kernel_ptr<T>(BFS_THREADS), BFS_THREADS, 0));
	const unsigned grid = (unsigned) device_info().sms * (unsigned) std::max(occ, 1);
	TreeDev<T> tv = t.view<T>();
	QDev<T> qd{kind, min1, max1, min2};
	WorkDev w{rec, NA_REC_CAP, path0, path1, seed0, seed1, 2u, ro, NA_RO_CAP, counts, cursor, offsets, ctl};
	// the one-CTA top pass (which unpacks the query and zeroes its count and output
	// cursor), then the per-level kernels for whatever it left
	launch_cta_pass<T>(tv, qd, w, 1u, 1u, QOut<T>{kind, min1, max1, min2}, in, nullptr, s);
	PST_CUDA(cudaMemcpyAsync(&h, ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (!(h.flags & (BATCH_FLAG_BAD_QUERY | BATCH_FLAG_INTERNAL | BATCH_FLAG_TASK_OVERFLOW)) &&
	    h.cta_levels < tv.levels) {
		for (uint32_t d = h.cta_levels; d < tv.levels; d++)
			launch_level<T>(tv, qd, w, d, grid, BFS_THREADS, s);
		scan_offsets(counts, offsets, 1, scan, ctl, nullptr, s);
		PST_CUDA(cudaMemcpyAsync(&h, ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, s));
		PST_CUDA(cudaStreamSynchronize(s));
	}
	if (h.flags & BATCH_FLAG_BAD_QUERY)
		fail(PST_ERR_INVALID, "query kind must be PST_Q_THREE, PST_Q_LEFT or PST_Q_RIGHT");
	if (h.flags & (BATCH_FLAG_TASK_OVERFLOW | BATCH_FLAG_INTERNAL))
		fail(PST_ERR_INTERNAL, "no-alloc search: frontier consistency check failed");
	if (h.total == 0 || h.total > capacity || h.emitted)
		return h.total;
	const bool has_id = t.idtype == PST_ID_U32;
	if (ret == PST_RET_IDS)
		launch_emit<T, true, false>(tv, w, out, capacity, BFS_THREADS, 8, nullptr, s);
	else if (has_id)
		launch_emit<T, true, true>(tv, w, out, capacity, BFS_THREADS, 4, nullptr, s);
	else
		launch_emit<T, false, true>(tv, w, out, capacity, BFS_THREADS, 4, nullptr, s);
	PST_CUDA(cudaGetLastError());
	PST_CUDA(cudaMemcpyAsync(&h, ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (h.flags & (BATCH_FLAG_OUT_OVERFLOW | BATCH_FLAG_INTERNAL))
		fail(PST_ERR_INTERNAL, "no-alloc search: emit consistency check failed");
	return h.total;
}

}  // namespace

uint64_t search_noalloc(TreeStorage &t, const pst_query &q, pst_ret ret, void *out, uint64_t capacity, cudaStream_t s)
{
	if (t.levels > NOALLOC_MAX_LEVELS)
		fail(PST_ERR_CAPACITY, "pst_search_noalloc handles trees of at most " +
		                           std::to_string((1ull << NOALLOC_MAX_LEVELS) - 1) + " points (" +
		                           std::to_string(NOALLOC_SCRATCH_BYTES >> 20) + " MiB static scratch); this tree has " +
		                           std::to_string(t.n));
	int dev = 0;
	PST_CUDA(cudaGetDevice(&dev));
	if (t.device != dev)
		fail(PST_ERR_INVALID, "the tree lives on device " + std::to_string(t.device) + " but device " +
		                          std::to_string(dev) + " is current");
	// Every call on a device shares the one array, so two calls whose GPU work
	// overlapped would race on it; within this process the lock, held until the
	// call's work has completed, keeps calls from overlapping.
	std::lock_guard<std::mutex> lk(g_noalloc_mu);
	unsigned char *base = noalloc_scratch(dev);
	try {
		switch (t.dtype) {
		case PST_F32: return noalloc_run<float>(t, q, ret, out, capacity, s, base);
		case PST_F64: return noalloc_run<double>(t, q, ret, out, capacity, s, base);
		case PST_I32: return noalloc_run<int32_t>(t, q, ret, out, capacity, s, base);
		}
	} catch (...) {
		// kernels enqueued before the failure may still be using the array: let them
		// finish before the lock is released and another call rewrites it
		cudaStreamSynchronize(s);
		cudaGetLastError();
		throw;
	}
	fail(PST_ERR_INVALID, "bad dtype");
}

}  // namespace pst
