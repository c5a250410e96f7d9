// The direct variant's peel: the one-launch loop over the materialised clique
// list and the triangle -> clique CSR.
//
// Reference: peel_fourcliques over all triangles once per level, with claim
// flags per clique (nucleus/cuNucleus34.cu:107-141, 675-714).
//
// A clique is destroyed by the member that owns it in the round in which its
// first members die (the lowest id among those that die); the owner sets the
// clique's byte in `destroyed`, so a later member passes it with one byte load.
// A clique whose byte is clear has therefore only live members and members
// that die this round, which `dying` (a byte per triangle, set when it begins
// to die and left set) tells apart: no support is read beside the atomics.
//
// As launches (11 per round, half of them empty) a round took 34 us on R-MAT
// scale 14 and 55 us on the geometric graph with 50k points; here 16.5 and 25.
// The clique ids and members of a round stream from L2 or memory (R-MAT scale
// 14 holds 1.1 GB of them, and takes the rows instead: see list_cliques_bits);
// the atomics and the barriers are the rest.
#include "pipeline.cuh"

#include "peel_loop.cuh"

namespace n34 {

namespace {

struct DirectPath
{
	const uint64_t *off;
	const uint32_t *ids;
	const uint4 *quds;
	uint8_t *destroyed;
	uint8_t *dying;

	struct WarpMem
	{
		uint32_t next[Appender::CAP];
	};
	static constexpr uint32_t SMEM = uint32_t(sizeof(WarpMem)) * LOOP_WARPS;

	__device__ __forceinline__ void mark(uint32_t t) const { dying[t] = 1; }
	__device__ __forceinline__ void retire(uint32_t) const {}

	// A warp takes a batch of consecutive frontier triangles; the entries of
	// their clique lists are dealt out to the lanes across the batch.
	__device__ __forceinline__ void debit(const LoopArgs &g, const uint32_t *F, uint32_t nF, uint32_t *Fn, PhaseSlot *slot,
										  int32_t level) const
	{
		extern __shared__ uint4 loop_smem[];
		WarpMem &m = reinterpret_cast<WarpMem *>(loop_smem)[threadIdx.x >> 5];
		Appender next{m.next, Fn, &slot->n, &g.ctl->c.error, g.T, 0u};
		const uint32_t lane = lane_id();
		const Units u = debit_units(nF, loop_warps());
		claim_units(u.total, &slot->work, &g.ctl->c.error, [&](uint32_t unit) {
			const uint32_t stripe = unit & ((1u << u.shift) - 1u);
			const uint32_t base = (unit >> u.shift) * u.ch;
			uint32_t t = 0, len = 0;
			uint64_t begin = 0;
			if (lane < u.ch && base + lane < nF)
			{
				t = F[base + lane];
				begin = __ldg(off + t);
				len = uint32_t(__ldg(off + t + 1) - begin);
			}
			const bool one = u.ch == 1;
			const uint32_t incl = one ? len : warp_incl_scan(len), excl = incl - len;
			const uint32_t items = __shfl_sync(FULL, incl, one ? 0 : 31);
			for (uint32_t k0 = 32 * stripe; k0 < items; k0 += 32u << u.shift)
			{
				const uint32_t k = k0 + lane;
				const uint32_t s = one ? 0u : warp_owner(incl, k);
				const uint32_t ts = __shfl_sync(FULL, t, s);
				const uint64_t first = __shfl_sync(FULL, begin, s);
				const uint32_t at = k - __shfl_sync(FULL, excl, s);
				bool own = false;
				uint32_t id[3] = {0, 0, 0};
				bool live[3] = {false, false, false};
				if (k < items)
				{
					const uint32_t q = __ldg(ids + first + at);
					if (!destroyed[q])
					{
						const uint4 x = __ldg(quds + q);
						// the members other than ts (ascending ids)
						id[0] = x.x == ts ? x.y : x.x;
						id[1] = x.x == ts || x.y == ts ? x.z : x.y;
						id[2] = x.w == ts ? x.z : x.w;
						own = true;
#pragma unroll
						for (int r = 0; r < 3; ++r)
						{
							live[r] = !dying[id[r]];
							own = own && (live[r] || id[r] > ts);
						}
						if (own)
							destroyed[q] = 1;
					}
				}
				next.debit(own, id, live, g.S, level);
			}
		});
		next.finish();
	}
};

} // namespace

int peel_direct(Ctx &c, const CliqueCsr &csr, int32_t *support, int32_t *K, PeelCtl *hctl)
{
	LoopBuffers b;
	uint8_t *destroyed = nullptr, *dying = nullptr;
	int rc = loop_alloc(c, b);
	if (!rc)
		rc = dalloc(c, &destroyed, c.Q, "clique destroyed flags");
	if (!rc)
		rc = dalloc(c, &dying, c.T, "triangle dying flags");
	if (!rc && (cudaMemsetAsync(destroyed, 0, c.Q, c.stream) != cudaSuccess ||
				cudaMemsetAsync(dying, 0, c.T, c.stream) != cudaSuccess))
		rc = fail(NUCLEUS34_E_CUDA, "memset");
	if (!rc)
	{
		const DirectPath path{csr.off, csr.ids, reinterpret_cast<const uint4 *>(c.dquds), destroyed, dying};
		rc = run_peel_loop(c, b, path, support, K);
	}
	if (!rc)
		rc = loop_finish(c, b, hctl);
	c.release(destroyed);
	c.release(dying);
	loop_release(c, b);
	return rc;
}

} // namespace n34
