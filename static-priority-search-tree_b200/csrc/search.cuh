// Batched / single-query search engine (host side).
#pragma once

#include <cstddef>
#include <vector>

#include "tree.cuh"

namespace pst {

constexpr int BFS_THREADS = 256;
// Batches of at most this many queries (by default; pst_batch_opts.top_pass_queries
// sets it per engine, up to MAX_TOP_PASS_Q) start with the one-CTA top pass, which
// walks the upper levels without a kernel boundary between them.
constexpr uint32_t SMALL_BATCH_Q = 32;
constexpr uint32_t MAX_TOP_PASS_Q = 1024;
// Passes of an engine on a stream that are launched kernel by kernel before one is captured.
constexpr uint32_t DIRECT_PASSES = 4;

enum : uint32_t {
	BATCH_FLAG_TASK_OVERFLOW = 1u,  // frontier buffer too small (results incomplete)
	BATCH_FLAG_OUT_OVERFLOW = 2u,   // output buffer too small (nothing written)
	BATCH_FLAG_BAD_QUERY = 4u,      // a query kind out of range
	BATCH_FLAG_INTERNAL = 8u,       // a device-side consistency check failed
	BATCH_FLAGS_FAILED = BATCH_FLAG_TASK_OVERFLOW | BATCH_FLAG_BAD_QUERY | BATCH_FLAG_INTERNAL,
};

// Device control block of one pass; the host uploads a zeroed copy (with nq set)
// at the start of every pass.
struct BatchCtl {
	uint32_t lvl_cnt[40];   // alive records appended per level region
	uint32_t path_cnt[40];  // boundary-path tasks per level
	uint32_t seed_cnt[40];  // report-above seeds per level
	uint32_t rec_cnt;       // reported boundary nodes
	uint32_t nq;
	uint32_t flags;
	uint32_t cta_levels;    // levels already done by the one-CTA top pass (small batches)
	uint64_t need_tasks;
	uint64_t total;
	// start of each level region (the sum of the counts before it), written by the
	// kernel that fills the region, so the next kernel reads its bounds in one load
	// each instead of summing every count before them
	uint64_t lvl_base[40];
	uint32_t emitted;       // the top pass wrote the results itself
	uint32_t waits;         // the host waits for the pass: one that fails leaves the caller's buffers alone
	uint32_t unused[2];
	uint32_t top_cnt[40];   // records per level that k_bfs_groups put with the boundary nodes
	const pst_query *raw;   // the queries: mapped pinned memory or the caller's device array
	uint64_t *user_offsets; // the caller's nq + 1 offsets, or null
	uint32_t *host_fault;   // `fault` of the host's copy, or null
	uint32_t emit_follows;  // the emit hands the host its copy, while it runs, not the scan
	uint32_t fault;         // (host copy; the last word) the emit's consistency check failed
};

// Copies words first, first + step, .. of a pass's control block to the host's copy.  An emit
// does so while its other CTAs may be storing `fault` there (its own words hold none): it
// leaves that one word alone.
__host__ __device__ inline void copy_ctl(const BatchCtl *ctl, BatchCtl *to, uint32_t first, uint32_t step, bool emitting)
{
	const uint32_t end = sizeof(BatchCtl) / 4 - (emitting ? 1 : 0);
	for (uint32_t i = first; i < end; i += step)
		reinterpret_cast<uint32_t *>(to)[i] = reinterpret_cast<const uint32_t *>(ctl)[i];
}
static_assert(offsetof(BatchCtl, fault) + 4 == sizeof(BatchCtl), "the fault is the last word");

// What the top pass of a small batch works on (kernel parameters).
struct TopArgs {
	const pst_query *raw;   // the queries: null (they come along), mapped pinned memory or the
	                        // caller's device array
	void *out;              // where a pass that fits may write its results (null: count only)
	uint64_t out_cap;       // records `out` holds
	uint64_t *offsets;      // the caller's nq + 1 offsets, or null
	uint32_t ret;           // pst_ret
	uint32_t nq;
};

constexpr uint32_t TOP_IN_QUERIES = 32;  // host queries that come along
struct TopIn {
	TopArgs args;
	pst_query q[TOP_IN_QUERIES];
};

// What a whole pass starts from, apart from the control block's zeros.
struct PassStart {
	uint32_t nq;
	const pst_query *raw;
	uint64_t *offsets;
};

// Where a waiting call wants its results.
struct EmitTo {
	pst_ret ret;
	void *out;
	uint64_t capacity;
};

struct Batch {
	TreeStorage *tree = nullptr;
	std::shared_ptr<InFlight> passes;  // the tree's, kept for an engine that outlives it
	int device = 0;
	void *work = nullptr;              // one allocation of every buffer below but the frontier
	uint32_t max_q = 0;
	bool use_graph = true;
	uint32_t threads = BFS_THREADS;  // CTA size of the level and emit kernels
	uint32_t emit_u = 8;             // records in flight per warp in the emit (ids)
	uint32_t top_q = SMALL_BATCH_Q;  // largest batch that starts with the one-CTA top pass
	uint32_t blocks_per_sm = 0;
	uint32_t grid = 0;
	// queries
	pst_query *q_copy = nullptr;   // of a device array that kernels cannot read where it is
	uint64_t *copy_offsets_to = nullptr;  // the caller's offsets where kernels cannot write them
	pst_query *q_stage = nullptr;  // pinned staging for host query arrays
	uint32_t *kind = nullptr;
	void *min1 = nullptr, *max1 = nullptr, *min2 = nullptr;
	// frontier and results
	uint4 *rec = nullptr;       // alive records: (64-slot block base, query, reported-slot mask lo, hi)
	uint64_t task_cap = 0;      // alive-record capacity
	uint4 *path0 = nullptr, *path1 = nullptr;
	uint4 *seed0 = nullptr, *seed1 = nullptr;
	uint32_t path_cap = 0;
	uint4 *ro = nullptr;        // reported boundary nodes, as one-bit records
	uint32_t ro_cap = 0;
	uint32_t group = 0, group_stop = 0;  // queries a CTA of k_bfs_groups takes, and its levels (0: not used)
	uint64_t *counts = nullptr, *cursor = nullptr, *offsets = nullptr, *scan_tmp = nullptr;
	BatchCtl *ctl = nullptr;
	// One mapped pinned block: the control block a whole pass starts from (zeroed except
	// nq), the control block a pass ended with, the staged queries.  The _d pointers are
	// device addresses.
	BatchCtl *ctl_host = nullptr;
	const BatchCtl *ctl_host_d = nullptr;
	BatchCtl *back = nullptr;
	BatchCtl *back_d = nullptr;
	const pst_query *q_stage_d = nullptr;
	TopIn top_in{};
	bool idle = false;             // no pass that uses the block can be in flight
	bool open = false;             // kernels may be queued that nobody has waited for or marked
	BatchCtl last{};
	// the captured whole count pass, for the stream it was captured for
	struct Graph {
		cudaGraphExec_t exec = nullptr;
		cudaStream_t stream = nullptr;
		uint32_t direct = 0;  // passes launched on `stream` without it
		void drop();
	};
	Graph full_graph;
	bool captured = false;              // a graph of the caller's holds a pass of this engine
	std::vector<void *> captured_recs;  // outgrown frontiers such a graph may use

	~Batch();
	void init(TreeStorage *t, const pst_batch_opts &o);
	void release();
	void grow_tasks(uint64_t cap, cudaStream_t s);
	// offsets: where the pass also writes the result offsets (nq + 1 on the device, or null).
	void stage_queries(const pst_query *q, uint32_t nq, bool on_device, cudaStream_t s, uint64_t *offsets = nullptr);
	// Has the next whole pass on `s` captured at once: for an engine that will serve many.
	void capture_next(cudaStream_t s);
	// Whole count pass (every level kernel and the scan), asynchronous.
	void launch_count(cudaStream_t s);
	// Where `s` is capturing: adds the asynchronous pass to the caller's graph and returns
	// true.  Replays answer the same queries into the same buffers whatever the engine is
	// called with in between.
	bool run_captured(const pst_query *q, uint32_t nq, bool on_device, pst_ret ret, void *out, uint64_t capacity,
	                  uint64_t *offsets, cudaStream_t s);
	// Queues the copy of the pass's offsets to an array that its kernels could not write;
	// false where they have.
	bool copy_offsets(uint32_t nq, cudaStream_t s);
	// Notes that work queued on `s` may still run when the call returns.
	void mark_async(cudaStream_t s)
	{
		idle = false;
		passes->mark(this, s);
		open = false;
	}
	// Top pass of a small batch (nq <= top_q), asynchronous: when it stops
	// above the bottom (ctl->cta_levels < tree levels), launch_count_rest finishes it.
	void launch_count_top(cudaStream_t s);
	void launch_count_rest(uint32_t from, cudaStream_t s);
	// Count pass with the host waiting for it: the top pass for small batches, the
	// whole pass otherwise; grows the frontier buffer until the pass fits.  With `to` the
	// results (when they fit) are written too, before the one wait that the pass ends with;
	// last_status tells how that went.
	void count_sync(cudaStream_t s, uint64_t *total, const EmitTo *to = nullptr);
	void count_full_sync(cudaStream_t s, uint64_t *total, const EmitTo *to);
	void count_small_sync(cudaStream_t s, uint64_t *total, const EmitTo *to);
	// own: the pass's start by value instead of the engine's control block.
	void enqueue_counting(cudaStream_t s, const PassStart *own = nullptr);
	void enqueue_counting_top(cudaStream_t s);
	// to_host: the emit also writes the host's copy of the control block.
	void enqueue_emit(pst_ret ret, void *out, uint64_t capacity, cudaStream_t s, bool to_host = false);
	pst_status read_ctl(cudaStream_t s, uint64_t *total);  // of the device, after whatever ran
	pst_status finish(cudaStream_t s);  // waits for a waiting call's last kernels
	pst_status last_status() const;     // of the pass waited for last
	uint64_t record_size(pst_ret ret) const;

  private:
	template <typename T>
	void enqueue_count(cudaStream_t s, const PassStart *own);
	template <typename T>
	void enqueue_count_top(cudaStream_t s);
	template <typename T>
	void enqueue_count_rest(uint32_t from, cudaStream_t s);
	void check_queries(const pst_query *q, uint32_t nq) const;
	PassStart place(const pst_query *q, uint32_t nq, bool on_device, uint64_t *to_offsets, cudaStream_t s);
	template <typename T>
	void enqueue_emit_v(pst_ret ret, void *out, uint64_t capacity, cudaStream_t s, bool to_host);
	template <typename T, bool HAS_ID, bool POINTS>
	void enqueue_emit_t(void *out, uint64_t capacity, cudaStream_t s, bool to_host);
};

// One query into a caller buffer using only the library's static device scratch
// (no allocation); see pst_search_noalloc in include/pst_c.h.
uint64_t search_noalloc(TreeStorage &t, const pst_query &q, pst_ret ret, void *out, uint64_t capacity, cudaStream_t s);

}  // namespace pst
