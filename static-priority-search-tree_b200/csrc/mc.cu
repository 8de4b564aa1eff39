// Marching cubes over active metacells: the isosurface stage after the PST query.
// The query gives the metacells whose [min, max] contains the isovalue; every cell
// (voxel cube) of those metacells is classified by its 8 corner values and turned
// into triangles.  Headless: triangles go to a device buffer (9 float32 each, three
// vertices in vertex-index units).
//
// The triangle table is derived here from first principles (no third-party table):
//   * corner c of a cell sits at (c & 1, c >> 1 & 1, c >> 2 & 1); edge 4a + u + 2v runs
//     along axis a at the other two coordinates (u, v); a corner is inside when its
//     value is >= iso;
//   * on each cell face the edges whose ends differ are joined in pairs: two such
//     edges by one segment; four (diagonal corners inside) by two segments that each
//     cut off one inside corner.  A face decides alone, so the two cells sharing it
//     agree and the surface is closed;
//   * every crossed edge then has two segment ends, so the segments form loops; a
//     loop is oriented so that its (Newell) normal points from the inside ends of its
//     edges to the outside ends, rotated to start at its smallest edge, and fanned
//     from the first vertex whose diagonals all leave the cube faces (a diagonal on a
//     face would overlap the neighbouring cell).  At most 5 triangles per cell.
// Vertices: on the edge from global vertex a (the lower end) to b,
// t = (iso - f_a) / (f_b - f_a) and the coordinate along the edge's axis is a + t,
// rounded IEEE operations with nothing fused, so a vertex shared by neighbouring
// cells has the same bits in both.
//
// Kernels: k_mc_count sums each metacell's triangles and scans them into offsets in one
// pass, k_mc_emit writes them (cubic metacells of 2, 4 or 8 cells a side, whose vertices
// a warp holds in shared memory); k_mc_cells does either for any other sides, one warp
// per metacell, 32 cells at a time.  The output is ordered by metacell (as given), then
// cell (x fastest), then table order.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "scan_sort.cuh"
#include "tree.cuh"

namespace pst {

namespace {

constexpr int MC_MAX_TRI = 5;

struct McTables {
	uint8_t ntri[256];
	uint8_t edges[256][3 * MC_MAX_TRI];
};

// ---------------------------------------------------------------------------
// Table generation (host).

struct Geometry {
	int corner[8][3];
	int edge[12][2];
	int axis[12];
	int face[6][4];  // corners in ring order

	Geometry()
	{
		for (int c = 0; c < 8; c++) {
			corner[c][0] = c & 1;
			corner[c][1] = (c >> 1) & 1;
			corner[c][2] = (c >> 2) & 1;
		}
		int e = 0;
		for (int a = 0; a < 3; a++) {
			const int o0 = a == 0 ? 1 : 0, o1 = a == 2 ? 1 : 2;
			for (int v = 0; v < 2; v++)
				for (int u = 0; u < 2; u++) {
					int lo[3] = {0, 0, 0};
					lo[o0] = u;
					lo[o1] = v;
					int hi[3] = {lo[0], lo[1], lo[2]};
					hi[a] = 1;
					edge[e][0] = lo[0] | (lo[1] << 1) | (lo[2] << 2);
					edge[e][1] = hi[0] | (hi[1] << 1) | (hi[2] << 2);
					axis[e] = a;
					e++;
				}
		}
		int f = 0;
		const int ring[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
		for (int a = 0; a < 3; a++) {
			const int o0 = a == 0 ? 1 : 0, o1 = a == 2 ? 1 : 2;
			for (int s = 0; s < 2; s++) {
				for (int r = 0; r < 4; r++) {
					int p[3];
					p[a] = s;
					p[o0] = ring[r][0];
					p[o1] = ring[r][1];
					face[f][r] = p[0] | (p[1] << 1) | (p[2] << 2);
				}
				f++;
			}
		}
	}
	int edge_between(int c0, int c1) const
	{
		for (int e = 0; e < 12; e++)
			if ((edge[e][0] == c0 && edge[e][1] == c1) || (edge[e][0] == c1 && edge[e][1] == c0))
				return e;
		return -1;
	}
	unsigned faces_of_edge(int e) const
	{
		unsigned m = 0;
		for (int f = 0; f < 6; f++) {
			bool a = false, b = false;
			for (int r = 0; r < 4; r++) {
				a |= face[f][r] == edge[e][0];
				b |= face[f][r] == edge[e][1];
			}
			if (a && b)
				m |= 1u << f;
		}
		return m;
	}
};

void build_tables(McTables &T)
{
	const Geometry G;
	memset(&T, 0, sizeof(T));
	memset(T.edges, 255, sizeof(T.edges));
	for (int cfg = 0; cfg < 256; cfg++) {
		int inside[8];
		for (int c = 0; c < 8; c++)
			inside[c] = (cfg >> c) & 1;
		std::vector<int> adj[12];
		for (int f = 0; f < 6; f++) {
			int cut[4], xs[4], nx = 0;
			for (int i = 0; i < 4; i++) {
				cut[i] = G.edge_between(G.face[f][i], G.face[f][(i + 1) % 4]);
				if (inside[G.face[f][i]] != inside[G.face[f][(i + 1) % 4]])
					xs[nx++] = i;
			}
			auto join = [&](int a, int b) {
				adj[a].push_back(b);
				adj[b].push_back(a);
			};
			if (nx == 2)
				join(cut[xs[0]], cut[xs[1]]);
			else if (nx == 4)
				for (int i = 0; i < 4; i++)
					if (inside[G.face[f][i]])
						join(cut[(i + 3) % 4], cut[i]);
		}
		bool seen[12] = {};
		int ntri = 0;
		for (int e0 = 0; e0 < 12; e0++) {
			if (adj[e0].empty() || seen[e0])
				continue;
			std::vector<int> loop{e0};
			seen[e0] = true;
			int prev = -1, cur = e0, nxt = std::min(adj[e0][0], adj[e0][1]);
			while (nxt != e0) {
				loop.push_back(nxt);
				seen[nxt] = true;
				prev = cur;
				cur = nxt;
				nxt = adj[cur][0] != prev ? adj[cur][0] : adj[cur][1];
			}
			// orientation: Newell normal of the loop (twice the edge midpoints, integer)
			// against the inside-to-outside directions of its edges
			const int k = (int) loop.size();
			long nrm[3] = {0, 0, 0}, g[3] = {0, 0, 0};
			for (int i = 0; i < k; i++) {
				const int e = loop[i], e2 = loop[(i + 1) % k];
				long p[3], q[3];
				for (int d = 0; d < 3; d++) {
					p[d] = G.corner[G.edge[e][0]][d] + G.corner[G.edge[e][1]][d];
					q[d] = G.corner[G.edge[e2][0]][d] + G.corner[G.edge[e2][1]][d];
				}
				nrm[0] += p[1] * q[2] - p[2] * q[1];
				nrm[1] += p[2] * q[0] - p[0] * q[2];
				nrm[2] += p[0] * q[1] - p[1] * q[0];
				const int a = G.edge[e][0], b = G.edge[e][1];
				const int in = inside[a] ? a : b, out = inside[a] ? b : a;
				for (int d = 0; d < 3; d++)
					g[d] += G.corner[out][d] - G.corner[in][d];
			}
			const long dot = nrm[0] * g[0] + nrm[1] * g[1] + nrm[2] * g[2];
			if (dot == 0)
				fail(PST_ERR_INTERNAL, "marching-cubes table: degenerate loop");
			if (dot < 0)
				std::reverse(loop.begin(), loop.end());
			std::rotate(loop.begin(), std::min_element(loop.begin(), loop.end()), loop.end());
			// fan from the first vertex whose diagonals all leave the cube faces
			int apex = -1;
			for (int j = 0; j < k && apex < 0; j++) {
				bool ok = true;
				for (int i = 2; i < k - 1 && ok; i++)
					ok = (G.faces_of_edge(loop[j]) & G.faces_of_edge(loop[(j + i) % k])) == 0;
				if (ok)
					apex = j;
			}
			if (apex < 0)
				fail(PST_ERR_INTERNAL, "marching-cubes table: no valid fan");
			for (int i = 1; i < k - 1; i++) {
				if (ntri >= MC_MAX_TRI)
					fail(PST_ERR_INTERNAL, "marching-cubes table: too many triangles");
				T.edges[cfg][3 * ntri + 0] = (uint8_t) loop[apex];
				T.edges[cfg][3 * ntri + 1] = (uint8_t) loop[(apex + i) % k];
				T.edges[cfg][3 * ntri + 2] = (uint8_t) loop[(apex + i + 1) % k];
				ntri++;
			}
		}
		T.ntri[cfg] = (uint8_t) ntri;
	}
}

const McTables &host_tables()
{
	static McTables T;
	static std::once_flag once;
	std::call_once(once, [] { build_tables(T); });
	return T;
}

// ---------------------------------------------------------------------------
// Device side.

__constant__ McTables c_mc;
// corner offsets and edge ends, in the numbering above
__constant__ uint8_t c_edge_lo[12] = {0, 2, 4, 6, 0, 1, 4, 5, 0, 1, 2, 3};
__constant__ uint8_t c_edge_axis[12] = {0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 2, 2};

std::mutex g_mc_mu;
bool g_mc_uploaded[64] = {};

void upload_tables()
{
	int dev = 0;
	PST_CUDA(cudaGetDevice(&dev));
	if (dev < 0 || dev >= 64)
		fail(PST_ERR_CUDA, "device index out of range");
	std::lock_guard<std::mutex> lk(g_mc_mu);
	if (g_mc_uploaded[dev])
		return;
	PST_CUDA(cudaMemcpyToSymbol(c_mc, &host_tables(), sizeof(McTables)));
	g_mc_uploaded[dev] = true;
}

struct McGrid {
	uint32_t px, py, pz, mcx, mcy, mcz, Mx, My;
};

constexpr int MC_THREADS = 128;
// Triangles a warp stages per 32 cells (at most MC_MAX_TRI each), 9 floats each.
constexpr int MC_STAGE_FLOATS = 32 * MC_MAX_TRI * 9;

template <bool EMIT>
__global__ void __launch_bounds__(MC_THREADS) k_mc_cells(const float *__restrict__ vol, McGrid g,
                                                  const uint32_t *__restrict__ ids, uint64_t n, float iso,
                                                  uint64_t *__restrict__ counts, const uint64_t *__restrict__ offsets,
                                                  float *__restrict__ tri, uint64_t capacity)
{
	__shared__ McTables s_t;
	// the warp's triangles of 32 cells, in output order, written out together
	__shared__ float s_tri[EMIT ? MC_THREADS / 32 : 1][EMIT ? MC_STAGE_FLOATS : 1];
	for (int i = threadIdx.x; i < (int) sizeof(McTables) / 4; i += blockDim.x)
		reinterpret_cast<uint32_t *>(&s_t)[i] = reinterpret_cast<const uint32_t *>(&c_mc)[i];
	__syncthreads();
	const uint32_t lane = threadIdx.x & 31;
	const uint64_t gw = ((uint64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const uint64_t nw = ((uint64_t) gridDim.x * blockDim.x) >> 5;
	const uint64_t plane = (uint64_t) g.px * g.py;
	for (uint64_t i = gw; i < n; i += nw) {
		const uint32_t id = ids[i];
		const uint32_t mx = id % g.Mx, my = (id / g.Mx) % g.My, mz = id / (g.Mx * g.My);
		const uint32_t x0 = mx * g.mcx, y0 = my * g.mcy, z0 = mz * g.mcz;
		const uint32_t nx = min(x0 + g.mcx, g.px - 1) - min(x0, g.px - 1);
		const uint32_t ny = min(y0 + g.mcy, g.py - 1) - min(y0, g.py - 1);
		const uint32_t nz = min(z0 + g.mcz, g.pz - 1) - min(z0, g.pz - 1);
		const uint32_t ncell = nx * ny * nz;
		uint64_t base = EMIT ? offsets[i] : 0;
		uint32_t total = 0;
		for (uint32_t c0 = 0; c0 < ncell; c0 += 32) {
			const uint32_t c = c0 + lane;
			float f[8];
			uint32_t cfg = 0, x = 0, y = 0, z = 0;
			if (c < ncell) {
				x = x0 + c % nx;
				y = y0 + (c / nx) % ny;
				z = z0 + c / (nx * ny);
				const float *p = vol + (uint64_t) z * plane + (uint64_t) y * g.px + x;
#pragma unroll
				for (int k = 0; k < 8; k++) {
					f[k] = p[(uint64_t) ((k >> 2) & 1) * plane + (uint64_t) ((k >> 1) & 1) * g.px + (k & 1)];
					cfg |= f[k] >= iso ? 1u << k : 0u;
				}
			}
			const uint32_t nt = c < ncell ? s_t.ntri[cfg] : 0u;
			if constexpr (!EMIT) {
				total += nt;
			} else {
				const uint32_t inc = warp_incl_scan(nt);
				const uint32_t tot = __shfl_sync(0xFFFFFFFFu, inc, 31);
				float *stage = s_tri[threadIdx.x >> 5];
				for (uint32_t k = 0; k < nt; k++) {
					float *dst = stage + (inc - nt + k) * 9;
#pragma unroll
					for (int v = 0; v < 3; v++) {
						const uint32_t e = s_t.edges[cfg][3 * k + v];
						const uint32_t a = c_edge_lo[e], ax = c_edge_axis[e];
						const uint32_t b = a | (1u << ax);
						const float t = __fdiv_rn(__fsub_rn(iso, f[a]), __fsub_rn(f[b], f[a]));
						float pos[3] = {(float) (x + (a & 1)), (float) (y + ((a >> 1) & 1)),
						                (float) (z + ((a >> 2) & 1))};
						pos[ax] = __fadd_rn(pos[ax], t);
						dst[3 * v + 0] = pos[0];
						dst[3 * v + 1] = pos[1];
						dst[3 * v + 2] = pos[2];
					}
				}
				__syncwarp();
				// the 32 cells' triangles are one contiguous range: consecutive lanes
				// write consecutive floats
				const uint64_t nf = (uint64_t) tot * 9;
				const uint64_t room = base < capacity ? (capacity - base) * 9 : 0;
				float *out = tri + base * 9;
				for (uint32_t j = lane; j < nf && j < room; j += 32)
					out[j] = stage[j];
				__syncwarp();  // the stage is refilled by the next 32 cells
				base += tot;
			}
		}
		if constexpr (!EMIT) {
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
			if (lane == 0)
				counts[i] = total;
		}
	}
}

// ---------------------------------------------------------------------------
// Cubic metacells of MC = 2, 4 or 8 cells a side.
//
// A warp takes a group of consecutive metacells, reads each of their vertices once (a
// cell on its own reads eight) and keeps one bit of each, inside or not, from which a
// cell's pattern is cut out by a shift; the vertices of the next group are on their way
// meanwhile.  In the emit 64 cells list their triangles, and a lane makes a triangle: a
// lane per cell would walk 0 to 5 triangles of its own, the warp as long as its fullest
// cell, each vertex through indexed registers (local memory).  Bound by instructions and by
// what they wait for in shared memory (57 % of the cycles issue):
// 76 k active metacells of a 512^3 volume (3.9 M triangles, 142 MB) took 2 x 48 us to
// count, 22 to scan and 241 to emit with a lane per cell, and take 2 x 29 and 102 (the
// vertices as floats in shared memory, a lane per triangle corner: 2 x 46 and 128).  More
// CTAs an SM through launch bounds were slower (8: 104 us, 10: 120 with spills).
template <int MC>
struct McShape {
	static constexpr int V = MC + 1, NV = V * V * V, NC = MC * MC * MC;
	static constexpr int G = MC == 2 ? 8 : 1;                       // metacells of a group: 64 cells or more
	static constexpr int CELLS = G * NC;
	static constexpr int LOADS = (G * NV + 31) / 32;                // vertices of a group a lane reads
	static constexpr int WORDS = LOADS + 1;                         // inside bits of a group, and a word to shift in
	// groups of a warp's batch when it counts, and when it emits (fewer: its warps are
	// resident ones, which share the batches out evenly)
	static constexpr int R = MC == 4 ? 8 : 2, RE = MC == 4 ? 4 : 1;
	static constexpr int BATCH = R * G, EMIT_BATCH = RE * G;        // metacells (at most 32: a lane each)
	static constexpr int TILE = (MC_THREADS / 32) * BATCH;          // metacells of a counting CTA
};

// Head of the scratch of a call, zeroed before it.
struct McHead {
	unsigned long long total;
	uint32_t ticket, err;
};

// A warp's batch of metacells: lane b holds the lowest vertex of metacell b, its place in
// the volume, and whether no side of the metacell is cut by the volume's end.
template <int MC>
struct McBatch {
	uint32_t x, y, z;
	uint64_t at;
	bool whole;

	// Metacells ids[i0 .. i0 + size) as far as there are that many.
	__device__ __forceinline__ McBatch(const McGrid &g, const uint32_t *__restrict__ ids, uint64_t i0, uint64_t n,
	                                   int size)
	{
		const uint32_t lane = lane_id();
		const bool on = lane < (uint32_t) size && i0 + lane < n;
		const uint32_t id = on ? ids[i0 + lane] : 0u;
		x = id % g.Mx * MC;
		y = id / g.Mx % g.My * MC;
		z = id / (g.Mx * g.My) * MC;
		at = ((uint64_t) z * g.py + y) * g.px + x;
		whole = (uint64_t) x + MC < g.px && (uint64_t) y + MC < g.py && (uint64_t) z + MC < g.pz;
	}
};

// The lane's vertices of group r (m metacells of it exist): vertex lane + 32 j of the
// group, vertices past the volume repeating its last ones.
template <int MC>
__device__ __forceinline__ void mc_read(const float *__restrict__ vol, const McGrid &g, const McBatch<MC> &b, int r,
                                        int m, const uint32_t (&rel)[McShape<MC>::LOADS], float (&v)[McShape<MC>::LOADS])
{
	using S = McShape<MC>;
	const int lane = (int) lane_id();
	if (S::G == 1 && __shfl_sync(0xFFFFFFFFu, b.whole, r)) {
		const float *p = vol + __shfl_sync(0xFFFFFFFFu, b.at, r);
#pragma unroll
		for (int j = 0; j < S::LOADS; j++)
			v[j] = lane + 32 * j < S::NV ? p[rel[j]] : 0.0f;
	} else {
#pragma unroll
		for (int j = 0; j < S::LOADS; j++) {
			const int i = lane + 32 * j, k = S::G == 1 ? 0 : min(i / S::NV, S::G - 1), q = i - k * S::NV;
			const uint32_t x = __shfl_sync(0xFFFFFFFFu, b.x, r * S::G + k), y = __shfl_sync(0xFFFFFFFFu, b.y, r * S::G + k),
			               z = __shfl_sync(0xFFFFFFFFu, b.z, r * S::G + k);
			v[j] = i < m * S::NV ? vol[((uint64_t) min(z + q / (S::V * S::V), g.pz - 1) * g.py +
			                            min(y + q / S::V % S::V, g.py - 1)) * g.px + min(x + q % S::V, g.px - 1)]
			                     : 0.0f;
		}
	}
}

// Offsets of the lane's vertices from a metacell's lowest one (32 bits: mc_run sends
// volumes of larger planes to k_mc_cells).
template <int MC>
__device__ __forceinline__ void mc_rel(const McGrid &g, uint32_t (&rel)[McShape<MC>::LOADS])
{
	using S = McShape<MC>;
#pragma unroll
	for (int j = 0; j < S::LOADS; j++) {
		const uint32_t q = lane_id() + 32 * j;
		rel[j] = (q / (S::V * S::V) * g.py + q / S::V % S::V) * g.px + q % S::V;
	}
}

// The group's inside bits, vertex i at bit i, into `words` (the caller synchronises).
template <int MC>
__device__ __forceinline__ void mc_bits(const float (&v)[McShape<MC>::LOADS], float iso, uint32_t *words)
{
	using S = McShape<MC>;
	uint32_t mine = 0;
#pragma unroll
	for (int j = 0; j < S::LOADS; j++) {
		const uint32_t bits = __ballot_sync(0xFFFFFFFFu, v[j] >= iso);
		mine = lane_id() == (uint32_t) j ? bits : mine;
	}
	if (lane_id() < (uint32_t) S::WORDS)
		words[lane_id()] = mine;
}

__device__ __forceinline__ uint32_t mc_window(const uint32_t *words, uint32_t bit)
{
	return __funnelshift_r(words[bit >> 5], words[(bit >> 5) + 1], bit & 31);
}

// Inside pattern of the cell whose lowest vertex is vertex i of the group.
template <int MC>
__device__ __forceinline__ uint32_t mc_pattern(const uint32_t *words, uint32_t i)
{
	constexpr int V = McShape<MC>::V, Z = V * V;
	const uint32_t lo = mc_window(words, i);
	if constexpr (Z + V + 1 < 32) {
		return (lo & 3u) | ((lo >> V & 3u) << 2) | ((lo >> Z & 3u) << 4) | ((lo >> (Z + V) & 3u) << 6);
	} else {
		const uint32_t hi = mc_window(words, i + Z);
		return (lo & 3u) | ((lo >> V & 3u) << 2) | ((hi & 3u) << 4) | ((hi >> V & 3u) << 6);
	}
}

// Triangles of cell c of group r (0 past the group's m metacells and where the volume cuts
// the metacell); `cfg`: its pattern.  Called by the whole warp.
template <int MC>
__device__ __forceinline__ uint32_t mc_cell(const McGrid &g, const McBatch<MC> &b, int r, int m, int c,
                                            const uint32_t *words, const uint8_t *ntri, uint32_t &cfg)
{
	using S = McShape<MC>;
	const int k = S::G == 1 ? 0 : c / S::NC, q = c % S::NC, src = r * S::G + k;
	const uint32_t x = q % MC, y = q / MC % MC, z = q / (MC * MC);
	cfg = mc_pattern<MC>(words, k * S::NV + x + S::V * (y + S::V * z));
	bool on = __shfl_sync(0xFFFFFFFFu, b.whole, src);
	if (S::G > 1 || !on) {
		const uint32_t ox = __shfl_sync(0xFFFFFFFFu, b.x, src), oy = __shfl_sync(0xFFFFFFFFu, b.y, src),
		               oz = __shfl_sync(0xFFFFFFFFu, b.z, src);
		on = k < m && ox < g.px - 1 && ox + x < g.px - 1 && oy < g.py - 1 && oy + y < g.py - 1 && oz < g.pz - 1 &&
		     oz + z < g.pz - 1;
	}
	return on ? ntri[cfg] : 0u;
}

// Status word of a counting tile: flag (2 bits) | triangles of the tile, or of all tiles
// up to it.
constexpr unsigned long long MC_AGG = 1ull << 62, MC_PREFIX = 2ull << 62, MC_VALUE = MC_AGG - 1;
constexpr uint32_t MC_SPIN_LIMIT = 1u << 22;

// Triangles of the tiles before `tile`, whose own `total` is published (the whole of warp
// 0; a wait that runs out raises head->err).  Tiles are numbered in the order they start,
// so one only waits for tiles that are already running.
__device__ __forceinline__ unsigned long long mc_look_back(volatile unsigned long long *status, uint32_t tile,
                                                           unsigned long long total, McHead *head)
{
	const uint32_t lane = lane_id();
	if (lane == 0)
		status[tile] = (tile ? MC_AGG : MC_PREFIX) | total;
	unsigned long long before = 0;
	for (int64_t at = (int64_t) tile - 1 - lane; tile != 0; at -= 32) {
		unsigned long long x = MC_PREFIX;  // (before tile 0)
		uint32_t spins = 0;
		while (at >= 0 && (x = status[at]) < MC_AGG) {
			if (++spins > MC_SPIN_LIMIT) {
				atomicOr(&head->err, 1u);
				x = MC_PREFIX;
				break;
			}
			__nanosleep(32);
		}
		const uint32_t ends = __ballot_sync(0xFFFFFFFFu, x >= MC_PREFIX);
		const uint32_t end = ends ? __ffs(ends) - 1 : 31;
		unsigned long long v = lane <= end ? x & MC_VALUE : 0ull;
#pragma unroll
		for (int o = 16; o > 0; o >>= 1)
			v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
		before += v;
		if (ends)
			break;
	}
	if (lane == 0 && tile)
		status[tile] = MC_PREFIX | (before + total);
	return before;
}

// Triangles per metacell: their sum to head->total, and (offsets non-null) the exclusive
// scan of the metacells' counts.
template <int MC>
__global__ void __launch_bounds__(MC_THREADS) k_mc_count(const float *__restrict__ vol, McGrid g,
                                                         const uint32_t *__restrict__ ids, uint64_t n, float iso,
                                                         McHead *head, unsigned long long *status,
                                                         uint64_t *__restrict__ offsets)
{
	using S = McShape<MC>;
	__shared__ uint32_t s_words[MC_THREADS / 32][2][S::WORDS];
	__shared__ uint32_t s_cnt[S::TILE];
	__shared__ uint8_t s_ntri[256];
	__shared__ uint32_t s_tile;
	for (int i = threadIdx.x; i < 256; i += MC_THREADS)
		s_ntri[i] = c_mc.ntri[i];
	if (threadIdx.x == 0)
		s_tile = offsets ? atomicAdd(&head->ticket, 1u) : blockIdx.x;
	__syncthreads();
	const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
	const uint64_t t0 = (uint64_t) s_tile * S::TILE;
	const uint64_t w0 = t0 + warp * S::BATCH;
	const McBatch<MC> b(g, ids, w0, n, S::BATCH);
	const int have = w0 < n ? (int) min((uint64_t) S::BATCH, n - w0) : 0;  // the batch's metacells
	uint32_t rel[S::LOADS];
	mc_rel<MC>(g, rel);
	float v[S::LOADS];
	if (have)
		mc_read<MC>(vol, g, b, 0, min(have, S::G), rel, v);
	for (int r = 0; r < S::R; r++) {
		const int m = min(have - r * S::G, S::G);
		uint32_t *words = s_words[warp][r & 1];
		if (m > 0) {
			mc_bits<MC>(v, iso, words);
			if (have > (r + 1) * S::G)
				mc_read<MC>(vol, g, b, r + 1, min(have - (r + 1) * S::G, S::G), rel, v);
			__syncwarp();
		}
		constexpr int LANES = S::NC < 32 ? S::NC : 32;  // of a metacell
		uint32_t sum = 0;
#pragma unroll
		for (int c = 0; c < S::CELLS; c += 32) {
			uint32_t cfg;
			const uint32_t nt = m > 0 ? mc_cell<MC>(g, b, r, m, c + lane, words, s_ntri, cfg) : 0u;
			sum = LANES == 32 ? sum + nt : nt;
			if (LANES < 32) {
#pragma unroll
				for (int o = LANES / 2; o > 0; o >>= 1)
					sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
				if (lane % LANES == 0)
					s_cnt[warp * S::BATCH + r * S::G + (c + lane) / LANES] = sum;
			}
		}
		if (LANES == 32) {
			sum = __reduce_add_sync(0xFFFFFFFFu, sum);
			if (lane == 0)
				s_cnt[warp * S::BATCH + r] = sum;
		}
	}
	__syncthreads();
	if (warp != 0)
		return;
	uint32_t run = 0;  // (a tile's triangles fit 32 bits)
	for (int i = 0; i < S::TILE; i += 32) {
		const uint32_t v = i + lane < S::TILE ? s_cnt[i + lane] : 0u;
		const uint32_t inc = warp_incl_scan(v);
		if (i + lane < S::TILE)
			s_cnt[i + lane] = run + inc - v;
		run += __shfl_sync(0xFFFFFFFFu, inc, 31);
	}
	if (!offsets) {
		if (lane == 0 && run)
			atomicAdd(&head->total, (unsigned long long) run);
		return;
	}
	const unsigned long long before = mc_look_back(status, s_tile, run, head);
	__syncwarp();
	for (int i = lane; i < S::TILE && t0 + i < n; i += 32)
		offsets[t0 + i] = before + s_cnt[i];
	if (lane == 0 && t0 + S::TILE >= n)
		head->total = before + run;
}

template <int MC>
struct McEmitWarp {
	float v[McShape<MC>::G * McShape<MC>::NV];
	uint32_t words[McShape<MC>::WORDS];
	uint32_t task[64 * MC_MAX_TRI];  // cell | triangle of the cell << 6 | pattern << 9, in output order
	float out[32 * 9];
};

// A triangle corner in the table of the emit: offset of the edge's lower end from the
// cell's lowest vertex (7 bits), axis (2 bits), lower end's corner (bits x, y, z).
template <int MC>
__device__ __forceinline__ uint16_t mc_corner(uint32_t e)
{
	const uint32_t a = (uint32_t) (0x321054106420ull >> (4 * (e & 15u))) & 7u;
	const uint32_t off = (a & 1u) + McShape<MC>::V * ((a >> 1) & 1u) + McShape<MC>::V * McShape<MC>::V * (a >> 2);
	return (uint16_t) (off | ((e >> 2) & 3u) << 7 | a << 9);
}

// Writes every metacell's triangles at its offset, when all of them fit `capacity`.
template <int MC>
__global__ void __launch_bounds__(MC_THREADS) k_mc_emit(const float *__restrict__ vol, McGrid g,
                                                        const uint32_t *__restrict__ ids, uint64_t n, float iso,
                                                        const McHead *head, const uint64_t *__restrict__ offsets,
                                                        float *__restrict__ tri, uint64_t capacity)
{
	using S = McShape<MC>;
	__shared__ uint8_t s_ntri[256];
	__shared__ uint16_t s_corner[256 * 3 * MC_MAX_TRI];
	__shared__ McEmitWarp<MC> s_warp[MC_THREADS / 32];
	if (head->total > capacity || head->err)
		return;
	for (int i = threadIdx.x; i < 256; i += MC_THREADS)
		s_ntri[i] = c_mc.ntri[i];
	for (int i = threadIdx.x; i < 256 * 3 * MC_MAX_TRI; i += MC_THREADS)
		s_corner[i] = mc_corner<MC>((&c_mc.edges[0][0])[i]);
	__syncthreads();
	const uint32_t lane = lane_id();
	McEmitWarp<MC> &s = s_warp[threadIdx.x >> 5];
	const uint64_t nw = (uint64_t) gridDim.x * (MC_THREADS / 32), batches = (n + S::EMIT_BATCH - 1) / S::EMIT_BATCH;
	uint32_t rel[S::LOADS];
	mc_rel<MC>(g, rel);
	for (uint64_t w = (uint64_t) blockIdx.x * (MC_THREADS / 32) + (threadIdx.x >> 5); w < batches; w += nw) {
		const uint64_t w0 = w * S::EMIT_BATCH;
		const int have = (int) min((uint64_t) S::EMIT_BATCH, n - w0);
		const McBatch<MC> b(g, ids, w0, n, S::EMIT_BATCH);
		float *out = tri + offsets[w0] * 9;
		float v[S::LOADS];
		mc_read<MC>(vol, g, b, 0, min(have, S::G), rel, v);
		for (int r = 0; r * S::G < have; r++) {
			const int m = min(have - r * S::G, S::G);
			__syncwarp();  // the group before this one has been read
			mc_bits<MC>(v, iso, s.words);
#pragma unroll
			for (int j = 0; j < S::LOADS; j++)
				if (lane + 32 * j < S::G * S::NV)
					s.v[lane + 32 * j] = v[j];
			if (have > (r + 1) * S::G)
				mc_read<MC>(vol, g, b, r + 1, min(have - (r + 1) * S::G, S::G), rel, v);
			__syncwarp();
			for (int c0 = 0; c0 < S::CELLS; c0 += 64) {
				uint32_t cfg0, cfg1;
				const uint32_t n0 = mc_cell<MC>(g, b, r, m, c0 + lane, s.words, s_ntri, cfg0);
				const uint32_t n1 = mc_cell<MC>(g, b, r, m, c0 + 32 + lane, s.words, s_ntri, cfg1);
				// both halves in one scan (at most 160 triangles each)
				const uint32_t inc = warp_incl_scan(n0 | n1 << 16);
				const uint32_t all = __shfl_sync(0xFFFFFFFFu, inc, 31);
				const uint32_t first = all & 0xFFFFu, total = first + (all >> 16);
				if (!total)
					continue;
				for (uint32_t k = 0; k < n0; k++)
					s.task[(inc & 0xFFFFu) - n0 + k] = lane | k << 6 | cfg0 << 9;
				for (uint32_t k = 0; k < n1; k++)
					s.task[first + (inc >> 16) - n1 + k] = (lane + 32) | k << 6 | cfg1 << 9;
				__syncwarp();
				for (uint32_t t0 = 0; t0 < total; t0 += 32) {
					const bool on = t0 + lane < total;
					const uint32_t task = on ? s.task[t0 + lane] : 0u;
					const uint32_t c = c0 + (task & 63u), k = S::G == 1 ? 0u : c / S::NC, q = c % S::NC;
					const uint32_t x = q % MC, y = q / MC % MC, z = q / (MC * MC);
					const uint32_t src = r * S::G + k;
					const uint32_t ox = __shfl_sync(0xFFFFFFFFu, b.x, src) + x, oy = __shfl_sync(0xFFFFFFFFu, b.y, src) + y,
					               oz = __shfl_sync(0xFFFFFFFFu, b.z, src) + z;
					if (on) {
						const float x0 = (float) ox, x1 = (float) (ox + 1), y0 = (float) oy, y1 = (float) (oy + 1),
						            z0 = (float) oz, z1 = (float) (oz + 1);
						const float *cell = s.v + k * S::NV + x + S::V * (y + S::V * z);
						const uint16_t *corner = s_corner + (task >> 9) * (3 * MC_MAX_TRI) + 3 * ((task >> 6) & 7u);
#pragma unroll
						for (int e = 0; e < 3; e++) {
							const uint32_t w = corner[e], ax = (w >> 7) & 3u;
							const float *p = cell + (w & 127u);
							const float fa = p[0], fb = p[ax == 0 ? 1 : ax == 1 ? S::V : S::V * S::V];
							const float d = __fdiv_rn(__fsub_rn(iso, fa), __fsub_rn(fb, fa));
							const float fx = w & 0x200u ? x1 : x0, fy = w & 0x400u ? y1 : y0, fz = w & 0x800u ? z1 : z0;
							s.out[9 * lane + 3 * e + 0] = ax == 0 ? __fadd_rn(fx, d) : fx;
							s.out[9 * lane + 3 * e + 1] = ax == 1 ? __fadd_rn(fy, d) : fy;
							s.out[9 * lane + 3 * e + 2] = ax == 2 ? __fadd_rn(fz, d) : fz;
						}
					}
					__syncwarp();
					const uint32_t words = min(288u, 9 * (total - t0));
					for (uint32_t i = lane; i < words; i += 32)
						__stcs(out + i, s.out[i]);
					out += words;
					__syncwarp();  // the triangles are rewritten by the next 32
				}
			}
		}
	}
}

McGrid make_grid(const uint32_t P[3], const uint32_t mc[3])
{
	McGrid g;
	g.px = P[0];
	g.py = P[1];
	g.pz = P[2];
	g.mcx = mc[0];
	g.mcy = mc[1];
	g.mcz = mc[2];
	g.Mx = (P[0] - 1 + mc[0] - 1) / mc[0];
	g.My = (P[1] - 1 + mc[1] - 1) / mc[1];
	return g;
}

unsigned mc_grid_blocks(uint64_t n)
{
	const uint64_t want = (n + MC_THREADS / 32 - 1) / (MC_THREADS / 32);  // one metacell per warp
	return (unsigned) std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t) device_info().sms * 16));
}

}  // namespace

void mc_tables(uint8_t *ntri, uint8_t *edges)
{
	const McTables &T = host_tables();
	memcpy(ntri, T.ntri, 256);
	memcpy(edges, T.edges, sizeof(T.edges));
}

namespace {

// Device scratch of a call, given back when the stream's work is done.
struct McScratch {
	cudaStream_t s;
	char *p;
	McScratch(size_t bytes, cudaStream_t stream)
	    : s(stream), p(static_cast<char *>(pool_alloc(bytes, "marching-cubes scratch")))
	{
	}
	~McScratch()
	{
		cudaStreamSynchronize(s);
		pool_release(p, device_info().device);
	}
	McScratch(const McScratch &) = delete;
	McScratch &operator=(const McScratch &) = delete;
};

template <int MC>
uint64_t mc_run_cubic(const float *vol, const McGrid &g, const uint32_t *ids, uint64_t n, float iso, float *tri,
                      uint64_t capacity, bool emit, cudaStream_t s)
{
	using S = McShape<MC>;
	const uint64_t tiles = (n + S::TILE - 1) / S::TILE;
	const size_t head_bytes = sizeof(McHead) + (emit ? tiles * 8 : 0);
	McScratch buf(head_bytes + (emit ? n * 8 : 0), s);
	McHead *head = reinterpret_cast<McHead *>(buf.p);
	unsigned long long *status = reinterpret_cast<unsigned long long *>(head + 1);
	uint64_t *offsets = emit ? reinterpret_cast<uint64_t *>(buf.p + head_bytes) : nullptr;
	PST_CUDA(cudaMemsetAsync(head, 0, head_bytes, s));
	k_mc_count<MC><<<(unsigned) tiles, MC_THREADS, 0, s>>>(vol, g, ids, n, iso, head, status, offsets);
	PST_CUDA(cudaGetLastError());
	if (emit && tri && capacity) {
		// no more CTAs than fit at once: each makes a copy of the table
		int fit = 0;
		PST_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_mc_emit<MC>, MC_THREADS, 0));
		const uint64_t want = (n + S::EMIT_BATCH * (MC_THREADS / 32) - 1) / (S::EMIT_BATCH * (MC_THREADS / 32));
		const unsigned blocks = (unsigned) std::min<uint64_t>(want, (uint64_t) device_info().sms * std::max(fit, 1));
		k_mc_emit<MC><<<blocks, MC_THREADS, 0, s>>>(vol, g, ids, n, iso, head, offsets, tri, capacity);
		PST_CUDA(cudaGetLastError());
	}
	struct Pinned {
		McHead *h = static_cast<McHead *>(pinned_alloc(sizeof(McHead), "marching-cubes total"));
		~Pinned() { pinned_release(h, device_info().device); }
	} host;
	PST_CUDA(cudaMemcpyAsync(host.h, head, sizeof(McHead), cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (host.h->err)
		fail(PST_ERR_INTERNAL, "marching cubes: a wait on an earlier tile ran out");
	const uint64_t total = host.h->total;
	if (emit && !tri && total && total <= capacity)
		fail(PST_ERR_INVALID, "null triangle buffer");
	return total;
}

}  // namespace

uint64_t mc_run(const float *vol, const uint32_t P[3], const uint32_t mc[3], const uint32_t *ids, uint64_t n, float iso,
                float *tri, uint64_t capacity, bool emit, cudaStream_t s)
{
	upload_tables();
	if (n == 0)
		return 0;
	const McGrid g = make_grid(P, mc);
	if (mc[0] == mc[1] && mc[1] == mc[2] && (uint64_t) P[0] * P[1] < (1ull << 28)) {
		switch (mc[0]) {
		case 2: return mc_run_cubic<2>(vol, g, ids, n, iso, tri, capacity, emit, s);
		case 4: return mc_run_cubic<4>(vol, g, ids, n, iso, tri, capacity, emit, s);
		case 8: return mc_run_cubic<8>(vol, g, ids, n, iso, tri, capacity, emit, s);
		}
	}
	uint64_t *counts = nullptr, *offsets = nullptr, *scan = nullptr, *total_d = nullptr;
	const size_t tmp = scan_tmp_elems(n) * 8;
	const size_t bytes = n * 8 + (n + 1) * 8 + tmp + 64;
	McScratch scratch(bytes, s);
	char *buf = scratch.p;
	offsets = reinterpret_cast<uint64_t *>(buf);
	scan = reinterpret_cast<uint64_t *>(buf + (n + 1) * 8);
	total_d = reinterpret_cast<uint64_t *>(buf + (n + 1) * 8 + tmp);
	counts = reinterpret_cast<uint64_t *>(buf + (n + 1) * 8 + tmp + 64);
	const unsigned blocks = mc_grid_blocks(n);
	k_mc_cells<false><<<blocks, MC_THREADS, 0, s>>>(vol, g, ids, n, iso, counts, nullptr, nullptr, 0);
	PST_CUDA(cudaGetLastError());
	exclusive_scan<uint64_t>(counts, offsets, n, scan, total_d, s);
	uint64_t total = 0;
	PST_CUDA(cudaMemcpyAsync(&total, total_d, 8, cudaMemcpyDeviceToHost, s));
	PST_CUDA(cudaStreamSynchronize(s));
	if (!emit || total == 0 || total > capacity)
		return total;
	if (!tri)
		fail(PST_ERR_INVALID, "null triangle buffer");
	k_mc_cells<true><<<blocks, MC_THREADS, 0, s>>>(vol, g, ids, n, iso, nullptr, offsets, tri, capacity);
	PST_CUDA(cudaGetLastError());
	PST_CUDA(cudaStreamSynchronize(s));
	return total;
}

}  // namespace pst
