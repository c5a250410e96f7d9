// The peel on bit matrices, and the in-rows that it and the support count
// (bitcliques.cu) share.
//
// Reference: count_support and debit_partners (nucleus/cuNucleus34_ondemand.cu:
// 176-194, 203-305) find a triangle's cliques by a 3-way zipper over the
// incidence lists of its three edges (3T entries, sorted).
//
// Here a four-clique {u, v, w, x} with source u (u -> v, w, x) is found in one
// of two ways, depending on which of its triangles looks for it:
//   - by its three triangles of source u. The triangles of u are the bits of
//     u's symmetric matrix (BitMats), and the cliques of triangle (u, v, w)
//     that have source u are the set bits of row v AND row w: 32 candidates
//     per word pair, no list and no search. The peel clears the bits of dead
//     triangles, so a candidate's two triangles of source u are known to live.
//   - by its fourth ("top") triangle (v, w, x). In its names (u -> v -> w, with
//     x = y the clique's source): the in-row of edge u -> v has a bit for every
//     in-edge y -> u with a triangle (y, u, v), the in-row of u -> w one for
//     every (y, u, w), so the cliques are again the set bits of two rows.
// Every clique is in three row ANDs and one AND of in-rows. The ids of the
// partners come from the cells (a word's first id + the bits below), and the
// last one, which is not in hand, from the cell of its own source: the c edges
// of the two triangles found (their a edges, for the in-rows) tell its row and
// its position. So a clique costs a fixed chain of loads, where the lists
// needed a binary search of the longest list. An in-row whose triangles are all
// dead is passed by a count (R-MAT scale 18: 5.8e7 bits taken up, where the
// in-lists of the dying hold 4.8e9 entries).
//
// What bounds the debit: scattered accesses. Of a clique's three atomics and
// about five gathers, the third partner's cell and support are nowhere near
// the others. On one B200 atomics with a result run at 1.25e11 per second on
// 32 MB, 2.8e10 on 320 MB (loads of 4 bytes: 2.7e11, 5.8e10; of 16 bytes:
// 1.4e11, 3.8e10), so R-MAT scale 18's 2.3e9 cliques take 129 ms of its peel's
// 164. Hence: state bits beside the ids in the cell (one gather tells both; a
// separate word cost 330 ms), no loads of supports that other warps debit, and
// row words that leave out what a dying partner of lower id owns (2.3e9
// cliques settled instead of 3.8e9). A pipeline of asynchronous copies that kept
// four batches in flight changed nothing: latency is not the bound.
#include "pipeline.cuh"

#include <algorithm>

#include "form.h"
#include "peel_loop.cuh"

namespace n34 {

namespace {

// ---- in-rows -----------------------------------------------------------------

// column of every edge among its head's in-edges, and the in-degrees
__global__ void k_in_columns(const uint32_t *__restrict__ E, uint64_t m, uint32_t *__restrict__ indeg,
							 uint4 *__restrict__ erec)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
		erec[e].w = atomicAdd(indeg + E[e], 1u);
}

// key of every in-edge at its place among its head's (any order)
__global__ void k_in_keys(const uint32_t *__restrict__ E, const uint32_t *__restrict__ src, uint64_t m,
						  const uint64_t *__restrict__ in_off, const uint4 *__restrict__ erec,
						  unsigned long long *__restrict__ keys)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
		keys[in_off[E[e]] + erec[e].w] = (unsigned long long)src[e] << 32 | e;
}

// columns in the order of the sorted keys
__global__ void k_in_sorted_columns(const uint32_t *__restrict__ E, const unsigned long long *__restrict__ keys,
									uint64_t m, const uint64_t *__restrict__ in_off, uint4 *__restrict__ erec)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += stride)
	{
		const uint32_t e = uint32_t(keys[i]);
		erec[e].w = uint32_t(i - in_off[E[e]]);
	}
}

// What the rows and the lists would cost (rows_pay), summed over the edges.
struct EdgeSums
{
	unsigned long long sum_sq;  // of the triangles on an edge (k_in_counts)
	// row and in-row words of all triangles; the triangles that have a triangle's
	// head edge as head or tail, over all triangles; those that have its tail edge
	unsigned long long words, heads, tails;
	unsigned long long cells; // of the in-rows
};

// cells of every edge's in-row; cnt: triangles whose head or tail edge it is
__global__ void k_in_widths(const uint32_t *__restrict__ src, uint64_t m, const uint32_t *__restrict__ indeg,
							const uint4 *__restrict__ erec, const uint4 *__restrict__ rows,
							uint32_t *__restrict__ width, uint32_t *__restrict__ cnt, EdgeSums *__restrict__ sums)
{
	unsigned long long acc[4] = {0, 0, 0, 0}; // words, heads, tails, cells
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
	{
		const uint2 r = __ldg(reinterpret_cast<const uint2 *>(erec + e));
		const uint32_t W = r.y >> 16, in = (indeg[src[e]] + 31) >> 5;
		uint32_t head = 0, sym = 0;
		for (uint32_t q = 0; q < W; ++q)
		{
			const uint4 c = __ldg(rows + r.x + q);
			head += __popc(c.x);
			sym += __popc(c.z);
		}
		width[e] = in;
		cnt[e] = sym;
		acc[0] += uint64_t(head) * (W + in);
		acc[1] += uint64_t(head) * sym;
		acc[2] += uint64_t(sym - head) * sym;
		acc[3] += in;
	}
	block_sums(acc, &sums->words);
}

__global__ void k_in_starts(const uint64_t *__restrict__ off, uint64_t m, uint4 *__restrict__ erec)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
		erec[e].z = uint32_t(off[e]);
}

// the bit of every triangle (y, u, v): in-row of c = u -> v, column of b = y -> u
__global__ void k_in_set(const uint32_t *__restrict__ tris, uint64_t T, const uint4 *__restrict__ erec,
						 uint4 *__restrict__ cells)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
	{
		const uint32_t col = __ldg(&erec[tris[3 * t + 1]].w), row = __ldg(&erec[tris[3 * t + 2]].z);
		atomicOr(&cells[row + (col >> 5)].x, 1u << (col & 31));
	}
}

// triangles per in-row, in place of those with the edge as head or tail, and the
// sum over edges of (triangles on the edge)^2
__global__ void k_in_counts(const uint4 *__restrict__ erec, uint64_t m, const uint4 *__restrict__ cells,
							const uint32_t *__restrict__ width, uint32_t *__restrict__ cnt,
							uint2 *__restrict__ live, unsigned long long *__restrict__ sum_sq)
{
	unsigned long long acc[1] = {0};
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
	{
		const uint32_t first = erec[e].z, W = width[e], rest = cnt[e];
		uint32_t n = 0;
		for (uint32_t q = 0; q < W; ++q)
			n += __popc(cells[first + q].x);
		const unsigned long long d = uint64_t(n) + rest;
		cnt[e] = n;
		live[e] = make_uint2(n, W);
		acc[0] += d * d;
	}
	block_sums(acc, sum_sq);
}

// first positions of the cells' triangles in tri; all not dead, none dying. A
// warp takes 32 edges, whose in-rows lie behind one another, as their triangles
// do in tri: a running sum over their cells (one thread per edge wrote them at
// scattered places: 3.2 ms on R-MAT scale 18, 0.3 now).
__global__ void k_in_firsts(const uint4 *__restrict__ erec, uint64_t m, const uint32_t *__restrict__ width,
							const uint64_t *__restrict__ off, uint4 *__restrict__ cells)
{
	const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
	const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
	const uint32_t lane = lane_id();
	for (uint64_t e0 = warp * 32; e0 < m; e0 += nwarps * 32)
	{
		const uint64_t last = min(e0 + 32, m) - 1;
		const uint32_t first = erec[e0].z, end = erec[last].z + width[last];
		uint32_t at = uint32_t(off[e0]);
		for (uint32_t w0 = first; w0 < end; w0 += 32)
		{
			const uint32_t w = w0 + lane, x = w < end ? cells[w].x : 0u, n = __popc(x);
			uint32_t sum = n; // inclusive over the lanes
#pragma unroll
			for (uint32_t o = 1; o < 32; o <<= 1)
			{
				const uint32_t y = __shfl_up_sync(FULL, sum, o);
				if (lane >= o)
					sum += y;
			}
			if (w < end)
				cells[w] = make_uint4(x, at + sum - n, x, 0u);
			at += __shfl_sync(FULL, sum, 31);
		}
	}
}

__global__ void k_in_place(const uint32_t *__restrict__ tris, uint64_t T, const uint4 *__restrict__ erec,
						   const uint4 *__restrict__ cells, uint32_t *__restrict__ tri)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
	{
		const uint32_t col = __ldg(&erec[tris[3 * t + 1]].w), row = __ldg(&erec[tris[3 * t + 2]].z);
		const uint2 c = __ldg(reinterpret_cast<const uint2 *>(cells + row + (col >> 5)));
		tri[c.y + __popc(c.x & ((1u << (col & 31)) - 1u))] = uint32_t(t);
	}
}

// ---- peel ----------------------------------------------------------------------

// crec[t] = record of t's c edge: its row and position
__global__ void k_c_records(const uint32_t *__restrict__ tris, uint64_t T, const uint4 *__restrict__ erec,
							uint2 *__restrict__ crec)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
		crec[t] = __ldg(reinterpret_cast<const uint2 *>(erec + __ldg(tris + 3 * t + 2)));
}

// LIVE: counts of the live triangles of every in-row follow the peel, so that
// in-rows without any are passed by. Of use where in-rows are long (R-MAT scale
// 18, 8 words a row: peel 170 ms with them, 178 without; scale 16: 32.1 and
// 33.6); where they are two words or less, a word costs no more than its count
// (geometric graphs of 1.1e8 and 4.5e7 triangles: 52.8 and 22.9 ms with the
// counts, 50.9 and 22.4 without).
template <bool LIVE>
struct BitPath
{
	const uint32_t *tris;
	const uint4 *erec;
	uint4 *cells;
	uint4 *in_cells;
	const uint32_t *in_tri;
	uint2 *in_live;
	const uint2 *crec; // record of each triangle's c edge, or null (then looked up through tris)

	// Sets (mark) or clears (retire) the two bits of t in its source's matrix
	// and its bit in the in-row of its c edge.
	__device__ __forceinline__ void mark(uint32_t t) const
	{
		const uint32_t b = __ldg(tris + 3 * uint64_t(t) + 1), c = __ldg(tris + 3 * uint64_t(t) + 2);
		const uint4 ra = __ldg(erec + __ldg(tris + 3 * uint64_t(t))), rb = __ldg(erec + b);
		const uint32_t in = __ldg(&erec[c].z), p = ra.y & 0xffffu, j = rb.y & 0xffffu, col = rb.w;
		atomicOr(&cells[ra.x + (j >> 5)].w, 1u << (j & 31));
		atomicOr(&cells[rb.x + (p >> 5)].w, 1u << (p & 31));
		atomicOr(&in_cells[in + (col >> 5)].w, 1u << (col & 31));
	}

	__device__ __forceinline__ void retire(uint32_t t) const
	{
		const uint32_t b = __ldg(tris + 3 * uint64_t(t) + 1), c = __ldg(tris + 3 * uint64_t(t) + 2);
		const uint4 ra = __ldg(erec + __ldg(tris + 3 * uint64_t(t))), rb = __ldg(erec + b);
		const uint32_t in = __ldg(&erec[c].z), p = ra.y & 0xffffu, j = rb.y & 0xffffu, col = rb.w;
		atomicAnd(&cells[ra.x + (j >> 5)].z, ~(1u << (j & 31)));
		atomicAnd(&cells[rb.x + (p >> 5)].z, ~(1u << (p & 31)));
		atomicAnd(&in_cells[in + (col >> 5)].z, ~(1u << (col & 31)));
		if (LIVE)
			atomicSub(&in_live[c].x, 1u);
	}

	__device__ __forceinline__ uint2 row_of(uint32_t e) const
	{
		return __ldg(reinterpret_cast<const uint2 *>(erec + e));
	}

	__device__ __forceinline__ uint2 c_record(uint32_t t) const
	{
		return crec ? __ldg(crec + t) : row_of(__ldg(tris + 3 * uint64_t(t) + 2));
	}

	// Cliques found, up to 32 at a time, one per lane when they are settled:
	// HEAD_V / HEAD_W: x -> v / x -> w; DIES_1 / DIES_2: the partner (u, v, x) /
	// (u, w, x) dies this round; IN: found in the in-rows.
	static constexpr uint32_t HEAD_V = 4, HEAD_W = 8, DIES_1 = 16, DIES_2 = 32, IN = 64;
	struct Batch
	{
		// slot << 8 | flags, position of x, two partners (as far as known; IN:
		// their positions in in_tri)
		uint32_t flags[32], ix[32], id1[32], id2[32];
	};
	struct WarpMem
	{
		Batch batch;
		// the triangles of the unit in hand: {id, first cell of the row of its
		// head w, W << 16 | position of w, position of v}
		uint4 slot[32];
		uint32_t next[Appender::CAP];
	};
	static constexpr uint32_t SMEM = uint32_t(sizeof(WarpMem)) * LOOP_WARPS;

	// bits of word q that stand for positions below i
	__device__ __forceinline__ static uint32_t below_mask(uint32_t i, uint32_t q)
	{
		return q < (i >> 5) ? FULL : (q == (i >> 5) ? (1u << (i & 31)) - 1u : 0u);
	}

	// What a warp has found and not settled yet.
	struct Settler
	{
		const BitPath &p;
		WarpMem &m;
		int32_t *S;
		Appender next;
		int32_t level;
		uint32_t queued; // cliques in the batch

		__device__ __forceinline__ Settler(const BitPath &path, WarpMem &mem, const LoopArgs &g, uint32_t *Fn,
										   PhaseSlot *slot, int32_t lv)
			: p(path), m(mem), S(g.S), next{mem.next, Fn, &slot->n, &g.ctl->c.error, g.T, 0u}, level(lv), queued(0)
		{
		}

		// A clique found, at place `at` of the batch.
		__device__ __forceinline__ void put(uint32_t at, uint32_t slot, uint32_t ix, uint32_t flags, uint32_t id1,
											uint32_t id2)
		{
			m.batch.flags[at] = slot << 8 | flags;
			m.batch.ix[at] = ix;
			m.batch.id1[at] = id1;
			m.batch.id2[at] = id2;
		}

		// Settles the batch: one clique per lane. All lanes call.
		__device__ __forceinline__ void settle()
		{
			__syncwarp();
			const uint32_t lane = lane_id();
			bool ok = lane < queued, live1 = false, live2 = false, live3 = false;
			uint32_t t = 0, id1 = 0, id2 = 0, id3 = 0;
			if (ok)
			{
				const uint32_t f = m.batch.flags[lane], ix = m.batch.ix[lane];
				id1 = m.batch.id1[lane];
				id2 = m.batch.id2[lane];
				const uint4 a = m.slot[f >> 8];
				t = a.x;
				live1 = !(f & DIES_1);
				live2 = !(f & DIES_2);
				uint2 h = make_uint2(0, 0), l = h;
				if (f & IN)
				{
					// (y, u, v) and (y, u, w): their a edges are tail y -> v and head
					// y -> w of the third, (y, v, w)
					id1 = __ldg(p.in_tri + id1);
					id2 = __ldg(p.in_tri + id2);
					ok = (live1 || id1 > t) && (live2 || id2 > t);
					if (ok)
					{
						l = p.row_of(__ldg(p.tris + 3 * uint64_t(id1)));
						h = p.row_of(__ldg(p.tris + 3 * uint64_t(id2)));
					}
				}
				else
				{
					const uint32_t W = a.z >> 16, pw = a.z & 0xffffu, pv = a.w;
					// (plain loads: the state words beside the ids change between phases)
					const uint4 *row_x = p.cells + (a.y + (ix - pw) * W);
					const bool xv = f & HEAD_V, xw = f & HEAD_W;
					uint2 rv = make_uint2(0, 0), rw = rv;
					if (!xv)
						rv = *reinterpret_cast<const uint2 *>(row_x + (pv >> 5));
					if (!xw)
						rw = *reinterpret_cast<const uint2 *>(row_x + (pw >> 5));
					if (!xv)
						id1 = rv.y + __popc(rv.x & ((1u << (pv & 31)) - 1u));
					if (!xw)
						id2 = rw.y + __popc(rw.x & ((1u << (pw & 31)) - 1u));
					ok = (xv || (rv.x >> (pv & 31)) & 1u) && (xw || (rw.x >> (pw & 31)) & 1u);
					if (ok)
					{
						// x -> v: head x -> w, tail x -> v; v -> x -> w: head v -> w
						// (t's own c edge), tail v -> x; v -> w -> x: the reverse
						const uint2 r1 = p.c_record(id1), r2 = p.c_record(xv ? id2 : t);
						h = xv || xw ? r2 : r1;
						l = xv || xw ? r1 : r2;
					}
				}
				const uint32_t it = l.y & 0xffffu;
				ok = ok && (it >> 5) < (h.y >> 16);
				if (ok)
				{
					const uint4 c = p.cells[h.x + (it >> 5)];
					const uint32_t bit = it & 31;
					id3 = c.y + __popc(c.x & ((1u << bit) - 1u));
					live3 = !((c.w >> bit) & 1u);
					ok = (((c.x & c.z) >> bit) & 1u) && (live3 || id3 > t);
				}
			}
			const uint32_t id[3] = {id1, id2, id3};
			const bool live[3] = {live1, live2, live3};
			next.debit(ok, id, live, S, level);
			queued = 0;
			__syncwarp();
		}

	};

	// Deals the set bits of the warp's words out to the places of a batch: lane s
	// owns `words` words, word q of lane s is load(s, q, on). put(o, s, i, bit,
	// mine), all lanes: the bit is bit i of lane s's words and bit `bit` of the
	// word that lane o holds; the lanes with mine set take it, each for its own
	// place. queued counts the places taken; full() is called at 32 and frees
	// them. One of several warps that share a triangle takes its own 32s of each
	// 32 words' bits. one: only lane 0 owns words.
	template <class Load, class Put, class Full>
	__device__ __forceinline__ static void deal_bits(uint32_t words, bool one, uint32_t stripe, uint32_t shift,
													 uint32_t &queued, Load &&load, Put &&put, Full &&full)
	{
		const uint32_t lane = lane_id();
		const uint32_t incl = one ? words : warp_incl_scan(words), excl = incl - words;
		const uint32_t items = __shfl_sync(FULL, incl, one ? 0 : 31);
		for (uint32_t k0 = 0; k0 < items; k0 += 32)
		{
			const uint32_t k = k0 + lane;
			const uint32_t s = one ? 0u : warp_owner(incl, k);
			const uint32_t q = one ? k : k - __shfl_sync(FULL, excl, s);
			const uint32_t z = load(s, q, k < items);
			const uint32_t cnt = __popc(z);
			const uint32_t zi = warp_incl_scan(cnt);
			const uint32_t bits = __shfl_sync(FULL, zi, 31);
			uint32_t pos = 32 * stripe, end = shift ? min(pos + 32, bits) : bits;
			while (pos < bits) // warp-uniform
			{
				const uint32_t take = min(32u - queued, end - pos);
				const uint32_t r = pos + lane - queued; // this lane's bit
				const uint32_t o = warp_owner(zi, r);
				const uint32_t zz = __shfl_sync(FULL, z, o), first = __shfl_sync(FULL, zi - cnt, o),
							   qq = __shfl_sync(FULL, q, o), ss = __shfl_sync(FULL, s, o);
				const uint32_t bit = nth_bit(zz, r - first);
				put(o, ss, qq * 32 + bit, bit, lane >= queued && lane < queued + take);
				queued += take;
				pos += take;
				if (queued == 32)
					full();
				if (pos == end && shift)
				{
					pos += (32u << shift) - 32;
					end = min(pos + 32, bits);
				}
			}
		}
	}

	// A warp takes a unit of consecutive frontier triangles, one per lane for
	// the loads of their records. The words of their row pairs, and then of
	// their pairs of in-rows, are dealt out to the lanes across the unit; the
	// cliques found are settled 32 at a time, one lane per clique.
	__device__ __forceinline__ void debit(const LoopArgs &g, const uint32_t *F, uint32_t nF, uint32_t *Fn, PhaseSlot *slot,
										  int32_t level) const
	{
		extern __shared__ uint4 loop_smem[];
		WarpMem &m = reinterpret_cast<WarpMem *>(loop_smem)[threadIdx.x >> 5];
		Settler found(*this, m, g, Fn, slot, level);
		const uint32_t lane = lane_id();
		const Units u = debit_units(nF, loop_warps());
		claim_units(u.total, &slot->work, &g.ctl->c.error, [&](uint32_t unit) {
			// of the warps that share a triangle, half take its rows and half its
			// in-rows (R-MAT scale 12: 3% less than one after the other)
			const uint32_t shift = u.shift ? u.shift - 1 : 0u;
			const uint32_t stripe = (unit & ((1u << u.shift) - 1u)) >> (u.shift ? 1 : 0);
			const bool do_rows = !u.shift || !(unit & 1u), do_in = !u.shift || (unit & 1u);
			const uint32_t base = (unit >> u.shift) * u.ch;
			uint32_t row_w = 0, row_v = 0, W = 0, pos = 0, in_w = 0, in_v = 0, Win = 0;
			if (lane < u.ch && base + lane < nF)
			{
				const uint32_t t = F[base + lane];
				const uint32_t a = __ldg(tris + 3 * uint64_t(t)), b = __ldg(tris + 3 * uint64_t(t) + 1),
							   c = __ldg(tris + 3 * uint64_t(t) + 2);
				const uint4 ra = __ldg(erec + a), rb = __ldg(erec + b);
				// none live under one of the edges: no clique through the in-rows
				const uint2 lb = in_live[b];
				const uint32_t na = LIVE ? in_live[a].x : 1u, nc = LIVE ? in_live[c].x : 1u;
				row_w = ra.x;
				row_v = rb.x;
				W = do_rows ? ra.y >> 16 : 0u;
				pos = ra.y << 16 | (rb.y & 0xffffu);
				in_w = ra.z;
				in_v = rb.z;
				Win = do_in && min(min(lb.x, na), nc) ? lb.y : 0u;
				m.slot[lane] = make_uint4(t, ra.x, ra.y, rb.y & 0xffffu);
			}
			__syncwarp();
			uint4 cw = make_uint4(0, 0, 0, 0), cv = cw; // this lane's word pair
			auto put = [&](uint32_t o, uint32_t s, uint32_t ix, uint32_t bit, bool mine, uint32_t kind) {
				const uint32_t vx = __shfl_sync(FULL, cv.x, o), vy = __shfl_sync(FULL, cv.y, o),
							   vd = __shfl_sync(FULL, cv.w, o);
				const uint32_t wx = __shfl_sync(FULL, cw.x, o), wy = __shfl_sync(FULL, cw.y, o),
							   wd = __shfl_sync(FULL, cw.w, o);
				if (!mine)
					return;
				const uint32_t below = (1u << bit) - 1u;
				found.put(lane, s, ix,
						  kind | ((vx >> bit) & 1u ? HEAD_V : 0u) | ((wx >> bit) & 1u ? HEAD_W : 0u) |
							  ((vd >> bit) & 1u ? DIES_1 : 0u) | ((wd >> bit) & 1u ? DIES_2 : 0u),
						  vy + __popc(vx & below), wy + __popc(wx & below));
			};
			auto full = [&]() { found.settle(); };
			deal_bits(
				W, u.ch == 1, stripe, shift, found.queued,
				[&](uint32_t s, uint32_t q, bool on) {
					const uint32_t rw = __shfl_sync(FULL, row_w, s), rv = __shfl_sync(FULL, row_v, s);
					const uint32_t pj = __shfl_sync(FULL, pos, s), p = pj >> 16, j = pj & 0xffffu;
					if (!on)
						return 0u;
					cw = cells[rw + q];
					cv = cells[rv + q];
					// not the cliques that a dying partner of lower id owns: ids of u's
					// triangles ascend with the head's position, then the tail's, and
					// this triangle's are p and j
					const uint32_t below_p = below_mask(p, q), below_j = below_mask(j, q);
					const uint32_t low_v = (cv.x & (j < p ? FULL : 0u)) | (~cv.x & below_p);
					const uint32_t low_w = (cw.x & below_j) | (~cw.x & below_p);
					return cw.z & cv.z & ~(cv.w & low_v) & ~(cw.w & low_w);
				},
				[&](uint32_t o, uint32_t s, uint32_t ix, uint32_t bit, bool mine) { put(o, s, ix, bit, mine, 0u); },
				full);
			if (__any_sync(FULL, Win != 0))
				deal_bits(
					Win, u.ch == 1, stripe, shift, found.queued,
					[&](uint32_t s, uint32_t q, bool on) {
						const uint32_t rw = __shfl_sync(FULL, in_w, s), rv = __shfl_sync(FULL, in_v, s);
						if (!on)
							return 0u;
						cw = in_cells[rw + q];
						cv = in_cells[rv + q];
						return cw.z & cv.z;
					},
					[&](uint32_t o, uint32_t s, uint32_t ix, uint32_t bit, bool mine) { put(o, s, ix, bit, mine, IN); },
					full);
			if (found.queued)
				found.settle();
			__syncwarp(); // the slots are rewritten by the next unit
		});
		found.next.finish();
	}
};

} // namespace

// The bit form serves the direct variant, and the on-demand variant unless a
// flag asks for the list form (a layout, an owner test or a schedule of it); a
// graph with an edge in both directions goes to the lists, as one bit would stand
// for two triangles.
bool bit_form_wanted(const Ctx &c, int variant)
{
	constexpr uint32_t LIST_FORM = NUCLEUS34_OPT_STAMP_PEEL | NUCLEUS34_OPT_LEAN_MEMORY | NUCLEUS34_OPT_HOST_LOOP |
								   NUCLEUS34_OPT_NO_SMALL_ROUNDS | NUCLEUS34_OPT_FRONTIER_BY_C |
								   NUCLEUS34_OPT_CHUNKED_DEBIT | NUCLEUS34_OPT_SCALAR_SCANS |
								   NUCLEUS34_OPT_PIPELINED_DEBIT | NUCLEUS34_OPT_DEBIT_CURSOR;
	return c.one_way && !c.force_lists && (variant == NUCLEUS34_DIRECT || !(c.opt_flags & LIST_FORM));
}

int build_in_rows(Ctx &c, const BitMats &mats, InMats &in, int variant, bool *fits)
{
	const uint64_t T = c.T, m = c.m;
	const bool by_source = variant == NUCLEUS34_DIRECT;
	*fits = false;
	uint32_t *indeg = nullptr, *width = nullptr, *cnt = nullptr;
	uint64_t *off = nullptr;
	EdgeSums *sums = nullptr, hsums{};
	const uint32_t gm = grid_for(c, m, 256), gt = grid_for(c, T, 256);
	int rc = NUCLEUS34_OK;
	do
	{
		if ((rc = dalloc(c, &indeg, c.n, "in-degrees")) || (rc = dalloc(c, &width, m, "in-row widths")) ||
			(rc = dalloc(c, &cnt, m, "in-row counts")) || (rc = dalloc(c, &sums, 1, "edge sums")) ||
			(rc = dalloc(c, &off, m + 1, "in-row offsets")))
			break;
		if (cudaMemsetAsync(indeg, 0, c.n * 4, c.stream) != cudaSuccess ||
			cudaMemsetAsync(sums, 0, sizeof(EdgeSums), c.stream) != cudaSuccess)
		{
			rc = fail(NUCLEUS34_E_CUDA, "memset");
			break;
		}
		k_in_columns<<<gm, 256, 0, c.stream>>>(c.dE, m, indeg, mats.erec);
		k_in_widths<<<gm, 256, 0, c.stream>>>(c.dsrc, m, indeg, mats.erec, mats.cells, width, cnt, sums);
		c.launches += 2;
		if ((rc = scan_u32(c, width, off, m)))
			break;
		if (cudaMemcpyAsync(&hsums, sums, sizeof(EdgeSums), cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaStreamSynchronize(c.stream) != cudaSuccess)
		{
			rc = fail(NUCLEUS34_E_CUDA, "in-row widths");
			break;
		}
		in.nwords = hsums.cells;
		if (!rows_pay(variant, hsums.words, std::min(hsums.heads, hsums.tails)))
			break;
		if (by_source)
		{
			if ((rc = dalloc(c, &in.in_off, c.n + 1, "in-edge offsets")) || (rc = scan_u32(c, indeg, in.in_off, c.n)) ||
				(rc = dalloc(c, &in.in_edges, m, "in-edges")))
				break;
			k_in_keys<<<gm, 256, 0, c.stream>>>(c.dE, c.dsrc, m, in.in_off, mats.erec, in.in_edges);
			if ((rc = sort_segments_u64(c, in.in_edges, in.in_off, c.n)))
				break;
			k_in_sorted_columns<<<gm, 256, 0, c.stream>>>(c.dE, in.in_edges, m, in.in_off, mats.erec);
			c.launches += 2;
		}
		c.release(indeg);
		indeg = nullptr;
		const uint64_t room = c.budget > c.in_use ? c.budget - c.in_use : 0;
		if (!rows_fit(in.nwords, T, m, c.opt_flags & NUCLEUS34_OPT_VERIFIABLE, room))
			break;
		if ((rc = dalloc(c, &in.cells, in.nwords, "in-rows")) || (rc = dalloc(c, &in.live, m, "in-row counts")))
			break;
		if (cudaMemsetAsync(in.cells, 0, in.nwords * 16, c.stream) != cudaSuccess)
		{
			rc = fail(NUCLEUS34_E_CUDA, "memset");
			break;
		}
		k_in_starts<<<gm, 256, 0, c.stream>>>(off, m, mats.erec);
		k_in_set<<<gt, 256, 0, c.stream>>>(c.dtris, T, mats.erec, in.cells);
		k_in_counts<<<gm, 256, 0, c.stream>>>(mats.erec, m, in.cells, width, cnt, in.live, &sums->sum_sq);
		c.launches += 3;
		if ((rc = scan_u32(c, cnt, off, m)))
			break;
		if ((rc = dalloc(c, &in.tri, T, "in-row triangles")))
			break;
		k_in_firsts<<<gm, 256, 0, c.stream>>>(mats.erec, m, width, off, in.cells);
		k_in_place<<<gt, 256, 0, c.stream>>>(c.dtris, T, mats.erec, in.cells, in.tri);
		c.launches += 2;
		uint64_t placed = 0;
		if (cudaMemcpyAsync(&in.sum_te_sq, &sums->sum_sq, 8, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaMemcpyAsync(&placed, off + m, 8, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaStreamSynchronize(c.stream) != cudaSuccess || cudaGetLastError() != cudaSuccess)
		{
			rc = fail(NUCLEUS34_E_CUDA, "in-row kernels");
			break;
		}
		if (placed != T)
			rc = fail(NUCLEUS34_E_CUDA, "internal: in-rows do not hold every triangle once");
		*fits = true;
	} while (false);
	c.release(indeg);
	c.release(width);
	c.release(cnt);
	c.release(off);
	c.release(sums);
	if (rc || !*fits)
		free_in_rows(c, in);
	if (rc == NUCLEUS34_E_OOM_BUDGET)
	{
		clear_error();
		*fits = false;
		return NUCLEUS34_OK;
	}
	return rc;
}

void free_in_rows(Ctx &c, InMats &in)
{
	c.release(in.cells);
	c.release(in.tri);
	c.release(in.live);
	c.release(in.in_edges);
	c.release(in.in_off);
	in = InMats{};
}

int peel_bits(Ctx &c, const BitMats &mats, const InMats &in, int32_t *support, int32_t *K, PeelCtl *hctl)
{
	LoopBuffers b;
	uint2 *crec = nullptr;
	int rc = loop_alloc(c, b);
	if (!rc)
	{
		// optional: without room for it the records are looked up
		if (dalloc(c, &crec, c.T, "c edge records"))
		{
			crec = nullptr;
			clear_error();
		}
		else
		{
			k_c_records<<<grid_for(c, c.T, 256), 256, 0, c.stream>>>(c.dtris, c.T, mats.erec, crec);
			c.launches++;
		}
		if (in.nwords > 2 * c.m)
			rc = run_peel_loop(c, b, BitPath<true>{c.dtris, mats.erec, mats.cells, in.cells, in.tri, in.live, crec},
							   support, K);
		else
			rc = run_peel_loop(c, b, BitPath<false>{c.dtris, mats.erec, mats.cells, in.cells, in.tri, in.live, crec},
							   support, K);
	}
	if (!rc)
		rc = loop_finish(c, b, hctl);
	c.release(crec);
	loop_release(c, b);
	return rc;
}

} // namespace n34
