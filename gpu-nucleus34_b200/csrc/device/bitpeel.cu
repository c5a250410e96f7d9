// The on-demand variant on bit matrices: four-clique support and peel.
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
//   - by its fourth ("top") triangle (v, w, x), whose cliques {u; v, w, x} are
//     the common sources of two of the in-lists of its three edges (the
//     in-list of v -> w: the sources u of the triangles (u, v, w), ascending,
//     with their ids). T entries in all, a third of the incidence.
// Every clique is in three row ANDs and one list intersection. The ids of the
// partners come from the cells (a word's first id + the bits below), and the
// last one, which is not in hand, from the cell of its own source: the c edges
// of the two triangles found tell its row and its position. So a clique costs
// a fixed chain of loads, where the lists needed a binary search of the longest
// list, and of the in-lists the peel reads little: a live-entry bitmap and a
// live count per edge pass over the dead (R-MAT scale 18: 5.8e7 entries looked
// up in all, of 4.8e9 in the lists of the dying).
//
// What bounds the debit: scattered accesses. Of a clique's three atomics and
// about five gathers, the third partner's cell and support are nowhere near
// the others. On one B200 atomics with a result run at 1.25e11 per second on
// 32 MB, 2.8e10 on 320 MB (loads of 4 bytes: 2.7e11, 5.8e10; of 16 bytes:
// 1.4e11, 3.8e10), so R-MAT scale 18's 2.3e9 cliques take 128 ms of its peel's
// 175. Hence: state bits beside the ids in the cell (one gather tells both; a
// separate word cost 330 ms), no loads of supports that other warps debit, and
// row words that leave out what a dying partner of lower id owns (2.3e9
// cliques settled instead of 3.8e9). A pipeline of asynchronous copies that kept
// four batches in flight changed nothing: latency is not the bound.
#include "pipeline.cuh"

#include "peel_loop.cuh"

namespace n34 {

namespace {

constexpr int SUP_THREADS = 256;

// The two shorter of a triangle's three in-lists: A, to be looked up in B.
// Roles: 0 = under b (u -> v), 1 = under a (u -> w), 2 = under c (v -> w).
struct InPair
{
	uint32_t a0, a1, b0, b1;
	uint32_t ra, rb;
};

__device__ __forceinline__ InPair in_pair(uint2 sb, uint2 sa, uint2 sc)
{
	uint2 p = sb, q = sa, r = sc;
	uint32_t rp = 0, rq = 1, rr = 2;
	uint2 t;
	uint32_t rt;
	if (q.y - q.x < p.y - p.x)
	{
		t = p; p = q; q = t;
		rt = rp; rp = rq; rq = rt;
	}
	if (r.y - r.x < q.y - q.x)
	{
		t = q; q = r; r = t;
		rt = rq; rq = rr; rr = rt;
	}
	if (q.y - q.x < p.y - p.x)
	{
		t = p; p = q; q = t;
		rt = rp; rp = rq; rq = rt;
	}
	return InPair{p.x, p.y, q.x, q.y, rp, rq};
}

// support[t] = cliques on t. A warp takes 32 triangles: each lane counts the
// row ANDs of its own triangle (neighbours share their source, so the rows
// come from L1); the in-list entries of all 32 are then dealt out to the
// lanes one by one, each a binary search in the other list.
__global__ void __launch_bounds__(SUP_THREADS) k_support_bits(
	const uint32_t *__restrict__ tris, uint64_t T, const uint2 *__restrict__ erec, const uint4 *__restrict__ cells,
	const uint2 *__restrict__ span, const uint32_t *__restrict__ third, int32_t *__restrict__ support,
	unsigned long long *__restrict__ total)
{
	const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
	const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
	const uint32_t lane = lane_id();
	unsigned long long acc = 0;
	for (uint64_t base = warp * 32; base < T; base += nwarps * 32)
	{
		const uint64_t t = base + lane;
		uint32_t cnt = 0;
		InPair L{0, 0, 0, 0, 0, 0};
		if (t < T)
		{
			const uint32_t a = __ldg(tris + 3 * t), b = __ldg(tris + 3 * t + 1), c = __ldg(tris + 3 * t + 2);
			const uint2 ra = __ldg(erec + a), rb = __ldg(erec + b);
			const uint32_t W = ra.y >> 16;
			for (uint32_t q = 0; q < W; ++q)
				cnt += __popc(__ldg(&cells[ra.x + q].z) & __ldg(&cells[rb.x + q].z));
			L = in_pair(__ldg(span + b), __ldg(span + a), __ldg(span + c));
		}
		const uint32_t len = L.a1 - L.a0;
		const uint32_t incl = warp_incl_scan(len), excl = incl - len;
		const uint32_t items = __shfl_sync(FULL, incl, 31);
		for (uint32_t k0 = 0; k0 < items; k0 += 32)
		{
			const uint32_t k = k0 + lane;
			const uint32_t s = warp_owner(incl, k);
			const uint32_t i = __shfl_sync(FULL, L.a0, s) + k - __shfl_sync(FULL, excl, s);
			const uint32_t b0 = __shfl_sync(FULL, L.b0, s), b1 = __shfl_sync(FULL, L.b1, s);
			bool found = false;
			if (k < items)
			{
				const uint32_t x = __ldg(third + i);
				const uint32_t p = lower_bound32(third, b0, b1, x);
				found = p < b1 && __ldg(third + p) == x;
			}
			// each lane takes the matches among its own triangle's items
			const uint32_t fm = __ballot_sync(FULL, found);
			const uint32_t lo = excl > k0 ? excl - k0 : 0u, hi = incl > k0 ? incl - k0 : 0u;
			if (lo < 32 && hi > lo)
				cnt += __popc(fm & ((hi >= 32 ? FULL : (1u << hi) - 1u) & ~((1u << lo) - 1u)));
		}
		if (t < T)
			support[t] = int32_t(cnt);
		acc += cnt;
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
		acc += __shfl_xor_sync(FULL, acc, o);
	if (lane == 0 && acc)
		atomicAdd(total, acc);
}

// crec[t] = record of t's c edge
__global__ void k_c_records(const uint32_t *__restrict__ tris, uint64_t T, const uint2 *__restrict__ erec,
							uint2 *__restrict__ crec)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < T; t += stride)
		crec[t] = __ldg(erec + __ldg(tris + 3 * t + 2));
}

// live[e] = entries of e's in-list
__global__ void k_in_lengths(const uint2 *__restrict__ span, uint64_t m, uint32_t *__restrict__ live)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += stride)
		live[e] = span[e].y - span[e].x;
}

// tpos[t] = position of t's in-list entry
__global__ void k_in_positions(const uint32_t *__restrict__ tri, uint64_t T, uint32_t *__restrict__ tpos)
{
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
	for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < T; i += stride)
		tpos[tri[i]] = uint32_t(i);
}

struct BitPath
{
	const uint32_t *tris, *src;
	const uint2 *erec;
	uint4 *cells;
	const uint2 *span;
	const uint32_t *third, *tri;
	uint32_t *inlive;     // per edge: in-list entries whose triangle is not dead
	uint32_t *inbits;     // bit per in-list entry: its triangle is not dead
	const uint32_t *tpos; // position of each triangle's in-list entry, or null (then searched)
	const uint2 *crec;    // record of each triangle's c edge, or null (then looked up through tris)

	__device__ __forceinline__ void mark(uint32_t t) const
	{
		const uint2 ra = __ldg(erec + __ldg(tris + 3 * uint64_t(t))),
					rb = __ldg(erec + __ldg(tris + 3 * uint64_t(t) + 1));
		const uint32_t p = ra.y & 0xffffu, j = rb.y & 0xffffu;
		atomicOr(&cells[ra.x + (j >> 5)].w, 1u << (j & 31));
		atomicOr(&cells[rb.x + (p >> 5)].w, 1u << (p & 31));
	}

	__device__ __forceinline__ void retire(uint32_t t) const
	{
		const uint32_t b = __ldg(tris + 3 * uint64_t(t) + 1);
		const uint2 ra = __ldg(erec + __ldg(tris + 3 * uint64_t(t))), rb = __ldg(erec + b);
		const uint32_t p = ra.y & 0xffffu, j = rb.y & 0xffffu;
		atomicAnd(&cells[ra.x + (j >> 5)].z, ~(1u << (j & 31)));
		atomicAnd(&cells[rb.x + (p >> 5)].z, ~(1u << (p & 31)));
		const uint32_t c = __ldg(tris + 3 * uint64_t(t) + 2);
		atomicSub(inlive + c, 1u);
		uint32_t i;
		if (tpos)
			i = __ldg(tpos + t);
		else
		{
			const uint2 sc = __ldg(span + c);
			i = lower_bound32(third, sc.x, sc.y, __ldg(src + b));
		}
		atomicAnd(inbits + (i >> 5), ~(1u << (i & 31)));
	}

	__device__ __forceinline__ uint2 c_record(uint32_t t) const
	{
		return __ldg(erec + __ldg(tris + 3 * uint64_t(t) + 2));
	}

	// Cliques found, up to 32 at a time, one per lane when they are settled:
	// HEAD_V / HEAD_W: x -> v / x -> w; DIES_1 / DIES_2: the partner (u, v, x) /
	// (u, w, x) dies this round; LIST: found in the in-lists.
	static constexpr uint32_t HEAD_V = 4, HEAD_W = 8, DIES_1 = 16, DIES_2 = 32, LIST = 64;
	struct Batch
	{
		// slot << 8 | flags, position of x / role pair, two partners (as far as known)
		uint32_t flags[32], ix[32], id1[32], id2[32];
	};
	struct WarpMem
	{
		Batch batch;
		// the triangles of the batch in hand: {id, first cells of the rows of
		// its head w and tail v, first word of list A as an entry}, {W << 16 |
		// position of w, role pair and order << 16 | position of v, list B}
		uint4 s0[32], s1[32];
		uint32_t q0[32], q1[32]; // list entries dealt out: triangle, entry
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
		uint32_t stamp;
		uint32_t queued; // cliques in the batch

		__device__ __forceinline__ Settler(const BitPath &path, WarpMem &mem, const LoopArgs &g, uint32_t *Fn,
										   PhaseSlot *slot, int32_t lv, uint32_t st)
			: p(path), m(mem), S(g.S), next{mem.next, Fn, &slot->n, &g.ctl->c.error, g.T, 0u}, level(lv), stamp(st),
			  queued(0)
		{
		}

		// A clique found in the rows, at place `at` of the batch: slot s, x at
		// position ix; id1 and id2 as far as v's and w's row tell them.
		__device__ __forceinline__ void put_row(uint32_t at, uint32_t s, uint32_t ix, uint32_t flags, uint32_t id1,
												uint32_t id2)
		{
			m.batch.flags[at] = s << 8 | flags;
			m.batch.ix[at] = ix;
			m.batch.id1[at] = id1;
			m.batch.id2[at] = id2;
		}

		// A match of two in-lists: partners id1 and id2 of slot s's triangle, by
		// role pair. With two of the triangles (y, u, v), (y, u, w), (y, v, w) of y
		// in hand, the edges of y in them give the row and the position of the
		// third: uv + uw (0): head y -> w, tail y -> v, their a edges; uv + vw (1):
		// head y -> w from vw's a, tail y -> u from uv's b; uw + vw (2): head
		// y -> v from vw's b, tail y -> u from uw's b.
		__device__ __forceinline__ void put_list(uint32_t at, uint32_t s, uint32_t kind, uint32_t id1, uint32_t id2)
		{
			put_row(at, s, kind, LIST, id1, id2);
		}

		__device__ __forceinline__ uint2 c_rec(uint32_t t) const
		{
			return p.crec ? __ldg(p.crec + t) : p.c_record(t);
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
				const uint4 a = m.s0[f >> 8];
				t = a.x;
				uint2 h, l;
				if (f & LIST)
				{
					const int32_t s1 = ld_support(S + id1), s2 = ld_support(S + id2);
					l = __ldg(p.erec + __ldg(p.tris + 3 * uint64_t(id1) + (ix == 0 ? 0 : 1)));
					h = __ldg(p.erec + __ldg(p.tris + 3 * uint64_t(id2) + (ix == 2 ? 1 : 0)));
					live1 = s1 >= 0;
					live2 = s2 >= 0;
					ok = !partner_blocks(s1, id1, t, stamp) && !partner_blocks(s2, id2, t, stamp);
				}
				else
				{
					const uint4 b = m.s1[f >> 8];
					const uint32_t W = b.x >> 16, pw = b.x & 0xffffu, pv = b.y & 0xffffu;
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
					live1 = !(f & DIES_1);
					live2 = !(f & DIES_2);
					ok = (xv || (rv.x >> (pv & 31)) & 1u) && (xw || (rw.x >> (pw & 31)) & 1u);
					h = l = make_uint2(0, 0);
					if (ok)
					{
						// x -> v: head x -> w, tail x -> v; v -> x -> w: head v -> w
						// (t's own c edge), tail v -> x; v -> w -> x: the reverse
						const uint2 r1 = c_rec(id1), r2 = c_rec(xv ? id2 : t);
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

	// A warp takes a batch of consecutive frontier triangles, one per lane for
	// the loads of their records. The words of their row pairs, and then the
	// live entries of their shortest in-lists, are dealt out to the lanes across
	// the batch; the cliques found go through the found.
	__device__ __forceinline__ void debit(const LoopArgs &g, const uint32_t *F, uint32_t nF, uint32_t *Fn, PhaseSlot *slot,
										  int32_t level, uint32_t stamp) const
	{
		extern __shared__ uint4 loop_smem[];
		WarpMem &m = reinterpret_cast<WarpMem *>(loop_smem)[threadIdx.x >> 5];
		Settler found(*this, m, g, Fn, slot, level, stamp);
		const uint32_t lane = lane_id();
		const Units u = debit_units(nF, (gridDim.x * blockDim.x) >> 5);
		claim_units(u.total, &slot->work, [&](uint32_t unit) {
			const uint32_t stripe = unit & ((1u << u.shift) - 1u);
			const uint32_t base = (unit >> u.shift) * u.ch;
			const bool have = lane < u.ch && base + lane < nF;
			uint32_t row_w = 0, row_v = 0, W = 0, pos = 0;
			uint2 la = make_uint2(0, 0); // in-list A
			if (have)
			{
				const uint32_t t = F[base + lane];
				const uint32_t a = __ldg(tris + 3 * uint64_t(t)), b = __ldg(tris + 3 * uint64_t(t) + 1),
							   c = __ldg(tris + 3 * uint64_t(t) + 2);
				const uint2 ra = __ldg(erec + a), rb = __ldg(erec + b);
				// the two in-lists with the fewest live entries, the least first
				// (role 0: under b, 1: under a, 2: under c); none live, no clique
				const uint32_t nb = inlive[b], na = inlive[a], nc = inlive[c];
				row_w = ra.x;
				row_v = rb.x;
				W = ra.y >> 16;
				pos = ra.y << 16 | (rb.y & 0xffffu);
				uint32_t meta = 0;
				uint2 lb = la;
				if (min(min(na, nb), nc))
				{
					const uint32_t most = nc >= na && nc >= nb ? 2u : (na >= nb ? 1u : 0u);
					// the pair without `most`: lower role first, swapped if the other has fewer
					const uint32_t e0 = most == 0 ? a : b, e1 = most == 2 ? a : c;
					const bool swap = (most == 0 ? na : nb) > (most == 2 ? na : nc);
					la = __ldg(span + (swap ? e1 : e0));
					lb = __ldg(span + (swap ? e0 : e1));
					// role pair 0: uv + uw, 1: uv + vw, 2: uw + vw; swap: A holds the higher role
					meta = (2 - most) << 1 | (swap ? 1u : 0u);
				}
				m.s0[lane] = make_uint4(t, ra.x, rb.x, la.x & ~31u);
				m.s1[lane] = make_uint4(ra.y, (rb.y & 0xffffu) | meta << 16, lb.x, lb.y);
			}
			__syncwarp();
			uint4 cw = make_uint4(0, 0, 0, 0), cv = cw; // this lane's word pair
			deal_bits(
				W, u.ch == 1, stripe, u.shift, found.queued,
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
				[&](uint32_t o, uint32_t s, uint32_t ix, uint32_t bit, bool mine) {
					const uint32_t vx = __shfl_sync(FULL, cv.x, o), vy = __shfl_sync(FULL, cv.y, o),
								   vd = __shfl_sync(FULL, cv.w, o);
					const uint32_t wx = __shfl_sync(FULL, cw.x, o), wy = __shfl_sync(FULL, cw.y, o),
								   wd = __shfl_sync(FULL, cw.w, o);
					if (!mine)
						return;
					const uint32_t below = (1u << bit) - 1u;
					found.put_row(lane, s, ix,
								 ((vx >> bit) & 1u ? HEAD_V : 0u) | ((wx >> bit) & 1u ? HEAD_W : 0u) |
									 ((vd >> bit) & 1u ? DIES_1 : 0u) | ((wd >> bit) & 1u ? DIES_2 : 0u),
								 vy + __popc(vx & below), wy + __popc(wx & below));
				},
				[&]() { found.settle(); });
			// entries [a0, a1) as bits of the words that hold them
			const uint32_t nw = la.y > la.x ? ((la.y - 1) >> 5) - (la.x >> 5) + 1 : 0u;
			if (!__any_sync(FULL, nw != 0))
			{
				if (found.queued)
					found.settle();
				__syncwarp(); // the slots are rewritten by the next batch
				return;
			}
			uint32_t dealt = 0;
			auto search = [&]() {
				__syncwarp();
				bool live = false;
				uint32_t ia = 0, ib = 0, s = 0;
				if (lane < dealt)
				{
					s = m.q0[lane];
					const uint32_t i = m.s0[s].w + m.q1[lane], x = __ldg(third + i);
					const uint32_t b1 = m.s1[s].w, p = lower_bound32(third, m.s1[s].z, b1, x);
					if (p < b1 && __ldg(third + p) == x)
					{
						live = (inbits[p >> 5] >> (p & 31)) & 1u;
						ia = __ldg(tri + i);
						ib = __ldg(tri + p);
					}
				}
				dealt = 0;
				const uint32_t lm = __ballot_sync(FULL, live);
				const uint32_t at = found.queued + __popc(lm & lanemask_lt()), sum = found.queued + __popc(lm);
				const uint32_t meta = m.s1[s].y >> 16;
				if (live && at < 32)
					found.put_list(at, s, meta >> 1, meta & 1u ? ib : ia, meta & 1u ? ia : ib);
				found.queued = min(sum, 32u);
				if (sum >= 32)
				{
					found.settle();
					if (live && at >= 32)
						found.put_list(at - 32, s, meta >> 1, meta & 1u ? ib : ia, meta & 1u ? ia : ib);
					found.queued = sum - 32;
				}
				__syncwarp();
			};
			deal_bits(
				nw, u.ch == 1, stripe, u.shift, dealt,
				[&](uint32_t s, uint32_t q, bool on) {
					const uint32_t a0 = __shfl_sync(FULL, la.x, s), a1 = __shfl_sync(FULL, la.y, s);
					if (!on)
						return 0u;
					const uint32_t w = (a0 >> 5) + q;
					uint32_t z = inbits[w];
					if (q == 0)
						z &= FULL << (a0 & 31);
					if (a1 - w * 32 < 32)
						z &= (1u << (a1 & 31)) - 1u;
					return z;
				},
				[&](uint32_t, uint32_t s, uint32_t i, uint32_t, bool mine) {
					if (mine)
					{
						m.q0[lane] = s;
						m.q1[lane] = i;
					}
				},
				search);
			if (dealt)
				search();
			if (found.queued)
				found.settle();
			__syncwarp(); // the slots are rewritten by the next batch
		});
		found.next.finish();
	}
};

} // namespace

// The bit form serves the on-demand variant unless a flag asks for one of the
// list forms (a layout, an owner test or a schedule of theirs).
bool bit_form_wanted(const Ctx &c, int variant)
{
	constexpr uint32_t LIST_FORM = NUCLEUS34_OPT_STAMP_PEEL | NUCLEUS34_OPT_LEAN_MEMORY | NUCLEUS34_OPT_HOST_LOOP |
								   NUCLEUS34_OPT_NO_SMALL_ROUNDS | NUCLEUS34_OPT_FRONTIER_BY_C |
								   NUCLEUS34_OPT_CHUNKED_DEBIT | NUCLEUS34_OPT_SCALAR_SCANS |
								   NUCLEUS34_OPT_PIPELINED_DEBIT | NUCLEUS34_OPT_DEBIT_CURSOR;
	return variant == NUCLEUS34_ONDEMAND && !(c.opt_flags & LIST_FORM);
}

// Room for the in-lists (8 bytes per triangle), support, k and two frontiers
// (16), the two bitmaps, and the per-edge arrays of the in-list build.
bool bit_form_fits(const Ctx &c, const BitMats &mats)
{
	const uint64_t room = c.budget > c.in_use ? c.budget - c.in_use : 0;
	return mats.cells && 24 * c.T + c.T / 4 + 28 * c.m + (uint64_t(1) << 20) <= room;
}

int count_support_bits(Ctx &c, const BitMats &mats, const Incidence &in, int32_t *support, uint64_t *total)
{
	unsigned long long *dtot = nullptr;
	N34_TRY(dalloc(c, &dtot, 1, "support total"));
	unsigned long long h = 0;
	int rc = NUCLEUS34_OK;
	if (cudaMemsetAsync(dtot, 0, 8, c.stream) != cudaSuccess)
		rc = fail(NUCLEUS34_E_CUDA, "memset");
	if (!rc)
	{
		const uint32_t grid = grid_for(c, (c.T + 31) / 32, SUP_THREADS / 32, 32);
		k_support_bits<<<grid, SUP_THREADS, 0, c.stream>>>(c.dtris, c.T, mats.erec, mats.cells, in.span, in.third,
														   support, dtot);
		c.launches++;
		if (cudaGetLastError() != cudaSuccess ||
			cudaMemcpyAsync(&h, dtot, 8, cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
			cudaStreamSynchronize(c.stream) != cudaSuccess)
			rc = fail(NUCLEUS34_E_CUDA, "support count");
	}
	c.release(dtot);
	*total = h;
	return rc;
}

int peel_bits(Ctx &c, const BitMats &mats, const Incidence &in, int32_t *support, int32_t *K, PeelCtl *hctl)
{
	const uint64_t T = c.T, words = (T + 31) / 32;
	LoopBuffers b;
	uint2 *crec = nullptr;
	uint32_t *inbits = nullptr, *inlive = nullptr, *tpos = nullptr;
	int rc = loop_alloc(c, b);
	if (!rc)
		rc = dalloc(c, &inbits, words, "in-list entry bits");
	if (!rc)
		rc = dalloc(c, &inlive, c.m, "in-list live counts");
	if (!rc && cudaMemsetAsync(inbits, 0xff, words * 4, c.stream) != cudaSuccess)
		rc = fail(NUCLEUS34_E_CUDA, "memset");
	if (!rc)
	{
		k_in_lengths<<<grid_for(c, c.m, 256), 256, 0, c.stream>>>(in.span, c.m, inlive);
		c.launches++;
		// both optional: without room for them they are looked up
		if (dalloc(c, &tpos, T, "in-list positions"))
		{
			tpos = nullptr;
			clear_error();
		}
		else
		{
			k_in_positions<<<grid_for(c, T, 256), 256, 0, c.stream>>>(in.tri, T, tpos);
			c.launches++;
		}
		if (dalloc(c, &crec, T, "c edge records"))
		{
			crec = nullptr;
			clear_error();
		}
		else
		{
			k_c_records<<<grid_for(c, T, 256), 256, 0, c.stream>>>(c.dtris, T, mats.erec, crec);
			c.launches++;
		}
		const BitPath path{c.dtris, c.dsrc, mats.erec, mats.cells, in.span, in.third, in.tri, inlive, inbits, tpos, crec};
		rc = run_peel_loop(c, b, path, support, K);
	}
	if (!rc)
		rc = loop_finish(c, b, hctl);
	c.release(crec);
	c.release(tpos);
	c.release(inbits);
	c.release(inlive);
	loop_release(c, b);
	return rc;
}

} // namespace n34
