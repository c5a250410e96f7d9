// Four-clique support and the direct variant's clique list on bit matrices.
//
// Reference: count_support (nucleus/cuNucleus34_ondemand.cu:176-194);
// cu_cliques_quds (nucleus/utils.cuh:550-619) and the triangle -> clique
// incidence (cuNucleus34.cu:627-669).
//
// How the rows and in-rows of a triangle (u, v, w) give its cliques is told in
// bitpeel.cu. A clique is listed once, by its lowest triangle, in ascending
// order of its fourth vertex, so the direct variant needs to know of a
// candidate whether the other three triangles have higher ids. Ids ascend with
// the source, then the head's position, then the tail's, so words of masks tell
// it for 32 candidates at once:
//   (u, v, x), (u, w, x)  the head's position, then the tail's, against p and j
//   (v, w, x)             its source, v or x, against u
//   of an in-row's y      all three have source y: y against u
// and the number of cliques that a triangle owns is a sum of popcounts. The
// list form intersected the three lists of every triangle and searched the
// longest one for each common entry. R-MAT scale 14 (2.8 million triangles, 35
// million cliques), ms: in-rows 0.31, counts 0.10, list 1.36, against 0.62 for
// the incidence lists, 3.3, and 5.8 with the clique lists that the peel then
// needed; random geometric graph of 50,021 vertices (7.8 million cliques): 0.07
// + 0.69 against 0.61 + 1.03, both with clique lists.
// Bound by: the writes of the list, 16 bytes per clique from one thread per
// triangle, and the ids' scattered cells (35 million cliques in 1.4 ms are
// 0.4 TB/s of list).
#include "pipeline.cuh"

namespace n34 {

namespace {

constexpr int CL_THREADS = 256;
constexpr uint32_t NO_VERTEX = 0xffffffffu; // (a graph has fewer vertices)

// bits of word q that stand for positions >= i
__device__ __forceinline__ uint32_t from_mask(uint32_t i, uint32_t q)
{
	return q > (i >> 5) ? FULL : (q == (i >> 5) ? FULL << (i & 31) : 0u);
}

// A triangle's rows and the bounds of its own cliques.
struct TriRows
{
	uint4 ra, rb;          // records of its head edge (w) and tail edge (v)
	uint32_t p, j;         // positions of w and v in N+(u)
	uint32_t first_out;    // position in N+(u) of the first vertex above u
	uint32_t first_in;     // column of the first in-edge of u from above u
};

// Which of the common bits of word q of rows v and w t owns.
__device__ __forceinline__ uint32_t own_row(const TriRows &r, const uint4 cv, const uint4 cw, uint32_t q)
{
	const uint32_t above_p = from_mask(r.p + 1, q), above_j = from_mask(r.j + 1, q);
	return ((cv.x & (r.j > r.p ? FULL : 0u)) | (~cv.x & above_p)) & // (u, v, x): head v or x
		   ((cw.x & above_j) | (~cw.x & above_p)) &                 // (u, w, x): head w or x
		   ((cv.x & from_mask(r.first_out, q)) | (~cv.x & (r.j >= r.first_out ? FULL : 0u))); // source x or v
}

__device__ __forceinline__ TriRows tri_rows(const uint32_t *__restrict__ tris, uint64_t t,
											const uint4 *__restrict__ erec, const uint32_t *__restrict__ src,
											const uint2 *__restrict__ above)
{
	TriRows r;
	const uint32_t b = __ldg(tris + 3 * t + 1);
	r.ra = __ldg(erec + __ldg(tris + 3 * t));
	r.rb = __ldg(erec + b);
	r.p = r.ra.y & 0xffffu;
	r.j = r.rb.y & 0xffffu;
	const uint2 f = above ? __ldg(above + __ldg(src + b)) : make_uint2(0, 0);
	r.first_out = f.x;
	r.first_in = f.y;
	return r;
}

// above[u] = {position in N+(u), column among u's in-edges} of the first vertex
// above u
__global__ void k_above(const uint32_t *__restrict__ O, const uint32_t *__restrict__ E, uint64_t n,
						const uint64_t *__restrict__ in_off, const unsigned long long *__restrict__ in_edges,
						uint2 *__restrict__ above)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t u = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; u < n; u += stride)
	{
		const uint32_t out = lower_bound32(E, O[u], O[u + 1], uint32_t(u)) - O[u];
		uint64_t lo = in_off[u], k = in_off[u + 1] - lo;
		while (k > 0)
		{
			const uint64_t half = k >> 1;
			const bool less = (in_edges[lo + half] >> 32) < u;
			lo = less ? lo + half + 1 : lo;
			k = less ? k - half - 1 : half;
		}
		above[u] = make_uint2(out, uint32_t(lo - in_off[u]));
	}
}

// support[t] = cliques on t: the common bits of its two rows and of its two
// in-rows, one thread per triangle (neighbours share their source, so the rows
// come from L1). With OWN also the cliques whose lowest triangle is t. total:
// cliques found over all triangles, and those of them found in the rows. A clique
// is in the rows of three of its triangles and in the in-rows of the fourth; three
// vertices above a source that form a directed cycle are in the rows alone. (The
// second sum in 64 bits per thread: 40 registers instead of 32, support of 2.5e7
// triangles 0.33 ms instead of 0.26.)
template <bool OWN>
__global__ void __launch_bounds__(CL_THREADS) k_support_bits(
	const uint32_t *__restrict__ tris, uint64_t T, const uint4 *__restrict__ erec, const uint4 *__restrict__ rows,
	const uint4 *__restrict__ in_rows, const uint2 *__restrict__ in_live, const uint32_t *__restrict__ src,
	const uint2 *__restrict__ above, int32_t *__restrict__ support, uint32_t *__restrict__ own,
	unsigned long long *__restrict__ total)
{
	unsigned long long acc = 0;
	uint32_t rowcnt = 0; // below 1e8: a thread takes 1200 triangles at most, of fewer than 2^16 bits each
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
	{
		const TriRows r = tri_rows(tris, t, erec, src, above);
		const uint2 la = __ldg(in_live + __ldg(tris + 3 * t)), lb = __ldg(in_live + __ldg(tris + 3 * t + 1));
		uint32_t cnt = 0, mine = 0;
		for (uint32_t q = 0; q < (r.ra.y >> 16); ++q)
		{
			if (OWN)
			{
				const uint4 cw = __ldg(rows + r.ra.x + q), cv = __ldg(rows + r.rb.x + q);
				cnt += __popc(cw.z & cv.z);
				mine += __popc(cw.z & cv.z & own_row(r, cv, cw, q));
			}
			else
				cnt += __popc(__ldg(&rows[r.ra.x + q].z) & __ldg(&rows[r.rb.x + q].z));
		}
		rowcnt += cnt;
		if (la.x && lb.x)
			for (uint32_t q = 0; q < la.y; ++q)
			{
				const uint32_t z = __ldg(&in_rows[r.ra.z + q].x) & __ldg(&in_rows[r.rb.z + q].x);
				cnt += __popc(z);
				if (OWN)
					mine += __popc(z & from_mask(r.first_in, q));
			}
		support[t] = int32_t(cnt);
		if (OWN)
			own[t] = mine;
		acc += cnt;
	}
	unsigned long long sums[2] = {acc, rowcnt};
	block_sums(sums, total);
}

__device__ __forceinline__ void sort2(uint32_t &a, uint32_t &b)
{
	const uint32_t lo = min(a, b), hi = max(a, b);
	a = lo;
	b = hi;
}

// Id of the triangle with head edge record h and tail edge record l (edges of
// one source).
__device__ __forceinline__ uint32_t tri_id(const uint4 *__restrict__ rows, uint2 h, uint2 l)
{
	const uint32_t it = l.y & 0xffffu;
	if ((it >> 5) >= (h.y >> 16))
		return 0u; // not edges of one source: no clique of a degree-ordered graph
	const uint2 c = __ldg(reinterpret_cast<const uint2 *>(rows + h.x + (it >> 5)));
	return c.y + __popc(c.x & ((1u << (it & 31)) - 1u));
}

// The own cliques of every triangle at qoff[t], by their fourth vertex: one
// thread walks the own bits of its rows (x ascending) and of its in-rows (y
// ascending) side by side.
__global__ void __launch_bounds__(CL_THREADS) k_cliques_bits(
	const uint32_t *__restrict__ tris, uint64_t T, const uint32_t *__restrict__ O, const uint32_t *__restrict__ E,
	const uint32_t *__restrict__ src, const uint4 *__restrict__ erec, const uint4 *__restrict__ rows,
	const uint4 *__restrict__ in_rows, const uint2 *__restrict__ in_live, const uint32_t *__restrict__ in_tri,
	const uint64_t *__restrict__ in_off, const unsigned long long *__restrict__ in_edges,
	const uint2 *__restrict__ above, const uint64_t *__restrict__ qoff, uint4 *__restrict__ quds)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
	{
		uint64_t out = qoff[t];
		const uint64_t end = qoff[t + 1];
		if (out == end)
			continue;
		const TriRows r = tri_rows(tris, t, erec, src, above);
		const uint32_t a = __ldg(tris + 3 * t), b = __ldg(tris + 3 * t + 1), c = __ldg(tris + 3 * t + 2);
		const uint32_t u = __ldg(src + b), W = r.ra.y >> 16, ou = __ldg(O + u);
		const uint64_t iu = in_off[u];
		const uint2 rc = __ldg(reinterpret_cast<const uint2 *>(erec + c));
		const uint2 la = __ldg(in_live + a), lb = __ldg(in_live + b);
		const uint32_t Win = la.x && lb.x ? la.y : 0u;
		uint32_t q = 0, z = 0, x = NO_VERTEX; // rows: next word, bits left of the one before, next vertex
		uint32_t iq = r.first_in >> 5, iz = 0, y = NO_VERTEX;
		uint4 cv = make_uint4(0, 0, 0, 0), cw = cv, iv = cv, iw = cv;
		auto next_x = [&] {
			while (!z && q < W)
			{
				cw = __ldg(rows + r.ra.x + q);
				cv = __ldg(rows + r.rb.x + q);
				z = cw.z & cv.z & own_row(r, cv, cw, q);
				++q;
			}
			x = z ? __ldg(E + ou + (q - 1) * 32 + (__ffs(z) - 1)) : NO_VERTEX;
		};
		auto next_y = [&] {
			while (!iz && iq < Win)
			{
				iw = __ldg(in_rows + r.ra.z + iq);
				iv = __ldg(in_rows + r.rb.z + iq);
				iz = iw.x & iv.x & from_mask(r.first_in, iq);
				++iq;
			}
			y = iz ? uint32_t(in_edges[iu + (iq - 1) * 32 + (__ffs(iz) - 1)] >> 32) : NO_VERTEX;
		};
		next_x();
		next_y();
		while (out < end && (x != NO_VERTEX || y != NO_VERTEX))
		{
			uint32_t id1, id2;
			uint2 h, l;
			if (x < y) // a vertex is not both: x is an out-neighbour of u, y an in-neighbour
			{
				const uint32_t bit = __ffs(z) - 1, ix = (q - 1) * 32 + bit, below = (1u << bit) - 1u;
				z &= z - 1;
				const uint4 *row_x = rows + (r.ra.x + (ix - r.p) * W);
				const bool xv = (cv.x >> bit) & 1u, xw = (cw.x >> bit) & 1u;
				if (xv)
					id1 = cv.y + __popc(cv.x & below);
				else
				{
					const uint2 d = __ldg(reinterpret_cast<const uint2 *>(row_x + (r.j >> 5)));
					id1 = d.y + __popc(d.x & ((1u << (r.j & 31)) - 1u));
				}
				if (xw)
					id2 = cw.y + __popc(cw.x & below);
				else
				{
					const uint2 d = __ldg(reinterpret_cast<const uint2 *>(row_x + (r.p >> 5)));
					id2 = d.y + __popc(d.x & ((1u << (r.p & 31)) - 1u));
				}
				// x -> v: head x -> w, tail x -> v; v -> x -> w: head v -> w, tail
				// v -> x; v -> w -> x: the reverse
				const uint2 r1 = __ldg(reinterpret_cast<const uint2 *>(erec + __ldg(tris + 3 * uint64_t(id1) + 2)));
				const uint2 r2 =
					xv ? __ldg(reinterpret_cast<const uint2 *>(erec + __ldg(tris + 3 * uint64_t(id2) + 2))) : rc;
				h = xv || xw ? r2 : r1;
				l = xv || xw ? r1 : r2;
				next_x();
			}
			else
			{
				const uint32_t bit = __ffs(iz) - 1, below = (1u << bit) - 1u;
				iz &= iz - 1;
				// (y, u, v) and (y, u, w): their a edges are tail and head of (y, v, w)
				id1 = __ldg(in_tri + iv.y + __popc(iv.x & below));
				id2 = __ldg(in_tri + iw.y + __popc(iw.x & below));
				l = __ldg(reinterpret_cast<const uint2 *>(erec + __ldg(tris + 3 * uint64_t(id1))));
				h = __ldg(reinterpret_cast<const uint2 *>(erec + __ldg(tris + 3 * uint64_t(id2))));
				next_y();
			}
			uint32_t id3 = tri_id(rows, h, l);
			sort2(id1, id2);
			sort2(id2, id3);
			sort2(id1, id2);
			quds[out++] = make_uint4(uint32_t(t), id1, id2, id3);
		}
	}
}

// cursor[t] = end of t's own cliques in its list, which come first
__global__ void k_csr_cursors(const uint64_t *__restrict__ off, const uint64_t *__restrict__ qoff, uint64_t T,
							  unsigned long long *__restrict__ cursor)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
		cursor[t] = off[t] + (qoff[t + 1] - qoff[t]);
}

// The triangle -> clique lists: own cliques by their place in the clique list,
// the others by a cursor (the order inside a list does not matter).
__global__ void k_csr_fill(const uint4 *__restrict__ quds, uint64_t Q, const uint64_t *__restrict__ off,
						   const uint64_t *__restrict__ qoff, unsigned long long *__restrict__ cursor,
						   uint32_t *__restrict__ ids, uint32_t *__restrict__ err)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t q = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < Q; q += stride)
	{
		const uint4 x = quds[q];
		ids[off[x.x] + (q - qoff[x.x])] = uint32_t(q);
		unsigned long long at[3];
		at[0] = atomicAdd(cursor + x.y, 1ull);
		at[1] = atomicAdd(cursor + x.z, 1ull);
		at[2] = atomicAdd(cursor + x.w, 1ull);
#pragma unroll
		for (int r = 0; r < 3; ++r)
		{
			if (at[r] < 4 * Q) // capacity guard: the supports size every list exactly
				ids[at[r]] = uint32_t(q);
			else
				atomicOr(err, 1u);
		}
	}
}

} // namespace

static int build_above(Ctx &c, const InMats &in, uint2 **above)
{
	N34_TRY(dalloc(c, above, c.n, "vertex bounds"));
	k_above<<<grid_for(c, c.n, 256), 256, 0, c.stream>>>(c.dO, c.dE, c.n, in.in_off, in.in_edges, *above);
	c.launches++;
	return NUCLEUS34_OK;
}

int count_support_bits(Ctx &c, const BitMats &mats, const InMats &in, int32_t *support, uint64_t *total,
					   uint32_t *own, bool *acyclic)
{
	unsigned long long *dtot = nullptr, h[2] = {0, 0};
	uint2 *above = nullptr;
	int rc = dalloc(c, &dtot, 2, "support total");
	if (!rc && own)
		rc = build_above(c, in, &above);
	if (!rc && cudaMemsetAsync(dtot, 0, 16, c.stream) != cudaSuccess)
		rc = fail(NUCLEUS34_E_CUDA, "memset");
	if (!rc)
	{
		const uint32_t grid = grid_for(c, c.T, CL_THREADS, 32);
		if (own)
			k_support_bits<true><<<grid, CL_THREADS, 0, c.stream>>>(c.dtris, c.T, mats.erec, mats.cells, in.cells,
																	in.live, c.dsrc, above, support, own, dtot);
		else
			k_support_bits<false><<<grid, CL_THREADS, 0, c.stream>>>(c.dtris, c.T, mats.erec, mats.cells, in.cells,
																	 in.live, c.dsrc, above, support, own, dtot);
		c.launches++;
		if (cudaGetLastError() != cudaSuccess ||
			cudaMemcpyAsync(h, dtot, 16, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaStreamSynchronize(c.stream) != cudaSuccess)
			rc = fail(NUCLEUS34_E_CUDA, "support count");
	}
	c.release(dtot);
	c.release(above);
	*total = h[0];
	*acyclic = h[1] == 3 * (h[0] - h[1]);
	return rc;
}

int list_cliques_bits(Ctx &c, BitMats &mats, InMats &in, const int32_t *support, const uint32_t *own,
					  CliqueCsr &csr)
{
	const uint64_t T = c.T;
	uint64_t *qoff = nullptr;
	unsigned long long *cursor = nullptr;
	uint32_t *errf = nullptr;
	uint2 *above = nullptr;
	int rc = NUCLEUS34_OK;
	do
	{
		uint64_t Q = 0;
		if ((rc = dalloc(c, &qoff, T + 1, "clique offsets")) || (rc = scan_u32(c, own, qoff, T)))
			break;
		if (cudaMemcpyAsync(&Q, qoff + T, 8, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaStreamSynchronize(c.stream) != cudaSuccess)
		{
			rc = fail(NUCLEUS34_E_CUDA, "clique count");
			break;
		}
		if (Q > 0xffffffffull)
		{
			rc = fail(NUCLEUS34_E_RANGE32, "four-clique count " + std::to_string(Q) +
											   " exceeds the 32-bit clique id range of the direct variant; "
											   "use the on-demand variant");
			break;
		}
		c.Q = Q;
		if (Q == 0)
			break;
		if ((rc = dalloc(c, &c.dquds, 4 * Q, "four-cliques")) || (rc = build_above(c, in, &above)))
			break;
		uint4 *quds = reinterpret_cast<uint4 *>(c.dquds);
		k_cliques_bits<<<grid_for(c, T, CL_THREADS, 32), CL_THREADS, 0, c.stream>>>(
			c.dtris, T, c.dO, c.dE, c.dsrc, mats.erec, mats.cells, in.cells, in.live, in.tri, in.in_off, in.in_edges,
			above, qoff, quds);
		c.launches++;
		// The peel over the clique list (20 to 35 % faster than over the rows on
		// small graphs) pays for its lists while these stay in cache: lists and
		// peel together 3.7 ms against 4.1 at Q = 4 million, 3.8 against 4.1 at
		// 14, 4.1 against 4.6 and 7.8 against 7.7 at 16 to 19; 6.4 against 5.7
		// at 26, 12.3 against 10.2 at 35 and 20.1 against 13.9 at 64. It also
		// takes over where the peel over the rows (support apart: k, two
		// frontiers, death rounds, the ordering bitmap) has no room.
		constexpr uint64_t CSR_MAX = uint64_t(1) << 24;
		const uint64_t room = c.budget > c.in_use ? c.budget - c.in_use : 0;
		if (Q <= CSR_MAX || room < 16 * T + T / 8 + (uint64_t(1) << 20))
		{
			free_mats(c, mats);
			free_in_rows(c, in);
			if ((rc = dalloc(c, &csr.off, T + 1, "clique csr offsets")) ||
				(rc = scan_u32(c, reinterpret_cast<const uint32_t *>(support), csr.off, T)) ||
				(rc = dalloc(c, &csr.ids, 4 * Q, "clique csr ids")) ||
				(rc = dalloc(c, &cursor, T, "clique csr cursors")) || (rc = dalloc(c, &errf, 1, "clique check")))
				break;
			if (cudaMemsetAsync(errf, 0, 4, c.stream) != cudaSuccess)
			{
				rc = fail(NUCLEUS34_E_CUDA, "memset");
				break;
			}
			k_csr_cursors<<<grid_for(c, T, 256), 256, 0, c.stream>>>(csr.off, qoff, T, cursor);
			k_csr_fill<<<grid_for(c, Q, 256), 256, 0, c.stream>>>(quds, Q, csr.off, qoff, cursor, csr.ids, errf);
			c.launches += 2;
		}
		uint32_t herr = 0;
		if (cudaGetLastError() != cudaSuccess ||
			(errf && cudaMemcpyAsync(&herr, errf, 4, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess) ||
			cudaStreamSynchronize(c.stream) != cudaSuccess)
			rc = fail(NUCLEUS34_E_CUDA, "clique kernels");
		else if (herr)
			rc = fail(NUCLEUS34_E_CUDA, "internal: clique incidence overflow");
	} while (false);
	c.release(qoff);
	c.release(cursor);
	c.release(errf);
	c.release(above);
	return rc;
}

} // namespace n34
