// The level-synchronous peel as one cooperative launch.
//
// All blocks of the launch are resident at once and run every round of the
// peel, phases separated by grid barriers; nothing is launched and no size is
// read by the host in between. A round is two phases:
//   mark    the frontier's triangles get their k and leave the scans (the
//           support word becomes negative); the frontier before it
//           is retired (what a path keeps per dead triangle is cleared)
//   debit   every dying triangle enumerates its live four-cliques and debits
//           the partners still alive; a partner that falls to the level is
//           appended to the next frontier
// An empty next frontier is a level change: one more phase scans the supports
// for the triangles at level + 1 (and the minimum, should none sit there). A
// large next frontier is put in id order through a bitmap (two phases), so
// that neighbouring warps work on triangles that share their rows and lists.
//
// Round-to-round cost is what bounds the small graphs and the long tails of
// the large ones: with every step of a round a kernel of its own (13 launches
// in a CUDA graph's while node) a round took 38 us on R-MAT scale 12 and 66 us
// on scale 16, with most of the launches empty; here it takes 11.5 and 28 us, of
// which a barrier is 1.4.
//
// Figures given as pairs in this file and in the paths' were taken when the step
// was made, each against the code before it. Peels now, ms: R-MAT scale 12 3.56, 14
// (direct) 8.66, 16 31.9, 18 164; geometric, 2e7 triangles 9.15, 1.1e8 48.9.
//
// The counters that a phase fills (appended triangles, minimum support) live
// in one of four slots taken in turn; every block reads the slot right after
// the phase's barrier, and it is cleared two phases later, when no block can
// still read it.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace n34 {

// Two blocks of 512 threads per SM, 64 registers each (three blocks of 40
// registers: 13% slower on R-MAT scale 18; one of 1024: 2% slower).
constexpr uint32_t LOOP_THREADS = 512;
constexpr uint32_t LOOP_WARPS = LOOP_THREADS / 32;
constexpr uint32_t NO_SUPPORT = 0xffffffffu;
// A barrier wait longer than this ends the launch (every block leaves at its
// next barrier and the call returns E_TIMEOUT); so does a peel longer than
// LOOP_TIME_LIMIT_NS. R-MAT scale 20 peels in about a second.
constexpr unsigned long long LOOP_WAIT_LIMIT_NS = 60ull * 1000000000ull;
constexpr unsigned long long LOOP_TIME_LIMIT_NS = 600ull * 1000000000ull;

constexpr uint32_t CLAIM_TRIES = 1u << 24; // of 32 ns or more

struct alignas(16) PhaseSlot
{
	uint32_t arrived; // blocks at the phase's barrier
	uint32_t n;       // triangles appended in the phase (read with arrived, in one 64-bit load)
	uint32_t mn;      // least support above the gathered level (scan phase)
	uint32_t work;    // units of the debit phase claimed beyond the first of each warp
};

struct LoopCtl
{
	PeelCtl c; // results: peeled, ksum, kmax, rounds, error
	uint32_t timed_out;
	uint32_t abort;
	uint32_t scans, ordered;
	PhaseSlot slot[4];
	unsigned long long ns[4]; // time per phase kind: mark, debit, scan, order
};

struct LoopArgs
{
	LoopCtl *ctl;
	int32_t *S; // support; of peeled triangles ~k
	int32_t *K;
	uint32_t *R; // death rounds kept for the certificate, or null
	uint32_t *F0, *F1;
	uint32_t *fbits; // T bits, all zero (null: frontiers keep their order)
	uint64_t T;
	uint32_t sort_min; // frontiers at least this large are put in id order
};

// A warp's number in the launch: the first warps of all blocks, then their
// second warps, and so on, so that few warps' work is on as many SMs.
__device__ __forceinline__ uint32_t loop_warp() { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }
__device__ __forceinline__ uint32_t loop_warps() { return (gridDim.x * blockDim.x) >> 5; }

// f(i) for i in [0, n): every block takes an equal, contiguous share (whole
// warps), so that a small n is spread over all SMs and a large one keeps
// neighbours on one SM.
template <class Fn>
__device__ __forceinline__ void block_shares(uint64_t n, Fn &&f)
{
	const uint64_t share = ((n + gridDim.x - 1) / gridDim.x + 31) & ~uint64_t(31);
	const uint64_t end = min(n, (blockIdx.x + 1) * share);
	for (uint64_t i = blockIdx.x * share + threadIdx.x; i < end; i += blockDim.x)
		f(i);
}

__device__ __forceinline__ unsigned long long loop_ns()
{
	unsigned long long t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
	const uint32_t lane = lane_id();
#pragma unroll
	for (uint32_t o = 1; o < 32; o <<= 1)
	{
		const uint32_t y = __shfl_up_sync(FULL, v, o);
		if (lane >= o)
			v += y;
	}
	return v;
}

// First lane whose inclusive sum exceeds k (31 if none): the lane that item k
// of the warp's concatenated items belongs to.
__device__ __forceinline__ uint32_t warp_owner(uint32_t incl, uint32_t k)
{
	uint32_t s = 0;
#pragma unroll
	for (uint32_t step = 16; step > 0; step >>= 1)
		if (__shfl_sync(FULL, incl, s + step - 1) <= k)
			s += step;
	return s;
}

// Position of the r-th (from 0) set bit of z; r < popc(z).
__device__ __forceinline__ uint32_t nth_bit(uint32_t z, uint32_t r)
{
	uint32_t pos = 0;
#pragma unroll
	for (uint32_t w = 16; w > 0; w >>= 1)
	{
		const uint32_t c = __popc(z & ((1u << w) - 1u));
		if (r >= c)
		{
			r -= c;
			z >>= w;
			pos += w;
		}
	}
	return pos;
}

// A warp's triangles for the next frontier, collected in shared memory and
// handed over many at a time: atomics of all warps on the one counter of the
// frontier take about 5.5 cycles each (2.8 ns, whole GPU), which bounded the
// debit when every step with a crossing appended by itself (peel of the random
// geometric graph with 500k points: 106 ms, 69 with the buffer; R-MAT scale 18:
// 265 and 233 ms).
struct Appender
{
	static constexpr uint32_t CAP = 128;
	uint32_t *buf;  // CAP entries of this warp
	uint32_t *Fn;   // next frontier
	uint32_t *n;    // its size
	uint32_t *err;
	uint64_t T;     // capacity
	uint32_t count; // entries in buf (warp-uniform)

	// t for the lanes with hit set (all lanes call)
	__device__ __forceinline__ void push(bool hit, uint32_t t)
	{
		const uint32_t m = __ballot_sync(FULL, hit);
		if (hit)
			buf[count + __popc(m & lanemask_lt())] = t;
		count += __popc(m);
	}
	// A clique that the lanes with own set destroy: debits its live partners and
	// collects those that fall to the level (all lanes call).
	__device__ __forceinline__ void debit(bool own, const uint32_t id[3], const bool live[3], int32_t *S, int32_t level)
	{
		// all three in flight before the first result is used
		int32_t old[3];
#pragma unroll
		for (int r = 0; r < 3; ++r)
		{
			old[r] = 0x7fffffff;
			if (own && live[r])
				old[r] = atomicSub(S + id[r], 1);
		}
		if (!__any_sync(FULL, old[0] == level + 1 || old[1] == level + 1 || old[2] == level + 1))
			return;
#pragma unroll
		for (int r = 0; r < 3; ++r)
			push(old[r] == level + 1, id[r]);
		drain();
	}
	// makes room for three pushes (all lanes call)
	__device__ __forceinline__ void drain()
	{
		if (count <= CAP - 96)
			return;
		__syncwarp();
		uint32_t base = 0;
		if (lane_id() == 0)
			base = atomicAdd(n, count);
		write(__shfl_sync(FULL, base, 0));
	}
	__device__ __forceinline__ void write(uint32_t base)
	{
		for (uint32_t i = lane_id(); i < count; i += 32)
		{
			if (uint64_t(base) + i < T)
				Fn[base + i] = buf[i];
			else
				atomicOr(err, 1u);
		}
		__syncwarp();
		count = 0;
	}
	// the rest of all warps of the block, with one atomic (all threads call)
	__device__ __forceinline__ void finish()
	{
		__shared__ uint32_t s_at[LOOP_WARPS];
		if (lane_id() == 0)
			s_at[threadIdx.x >> 5] = count;
		__syncthreads();
		if (threadIdx.x < 32)
		{
			const uint32_t c = threadIdx.x < LOOP_WARPS ? s_at[threadIdx.x] : 0u;
			const uint32_t x = warp_incl_scan(c);
			uint32_t base = 0;
			if (threadIdx.x == 31 && x)
				base = atomicAdd(n, x);
			base = __shfl_sync(FULL, base, 31);
			if (threadIdx.x < LOOP_WARPS)
				s_at[threadIdx.x] = base + x - c;
		}
		__syncthreads();
		write(s_at[threadIdx.x >> 5]);
	}
};

// Ownership of a clique among the members that die this round: the lowest id
// (debit_partners' rule, cuNucleus34_ondemand.cu:237-276). Paths tell dying
// members by flags of their own, set in the mark phase: a support word is never
// read while other warps debit it.

// How a debit phase is cut into units, which are claimed as the warps go:
// batches of ch consecutive frontier triangles, at least sixteen per warp (a
// fixed stride over two per warp took 325 ms of debit on R-MAT scale 18,
// claimed units of that size 247); or, where the frontier has at most half as many triangles as
// there are warps, one triangle shared by 2^shift warps (twice or four times as
// many warps per triangle: 17% and 35% slower on R-MAT scale 12).
struct Units
{
	uint32_t ch, total;
	uint32_t shift; // log2 of the warps that share a triangle
};

__device__ __forceinline__ Units debit_units(uint32_t nF, uint32_t nwarps)
{
	Units u{1u, 0u, 0u};
	while (u.ch < 32 && uint64_t(u.ch) * 16 * nwarps <= nF)
		u.ch <<= 1;
	while (u.shift < 6 && (nF << (u.shift + 1)) <= nwarps)
		++u.shift;
	u.total = ((nF + u.ch - 1) / u.ch) << u.shift;
	return u;
}

// f(unit) for every unit of the phase (all lanes call f together; all threads
// of the block call). A block claims `grab` consecutive units at a time and its
// warps take them one by one, so that the warps of an SM work on neighbouring
// triangles, whose rows and supports are in the same lines and pages: against
// claims by single warps the peel takes 175 ms instead of 250 on R-MAT scale
// 18, 36 instead of 44 on scale 16, 56 instead of 62 on the geometric graph
// with 500k points (address translation limits scattered accesses: 1.3e5 lines
// that stay in L2 are read 2.7e11 times a second from 128 MB of addresses, 5.3e10
// from 512 MB; up to 256 units per claim make no difference). Every warp begins
// with a unit of its own and at least four are claimed at a time: a claim is a
// round trip for one warp while the others of its block wait, which cost the
// middle-sized rounds (a few units per warp) most: peel of R-MAT scale 14,
// direct, 8.84 -> 8.59 ms, scale 12 3.89 -> 3.79 and 10, direct, 1.63 -> 1.56,
// scale 16 31.4 -> 31.2.
template <class Fn>
__device__ __forceinline__ void claim_units(uint32_t total, uint32_t *work, uint32_t *err, Fn &&f)
{
	const uint32_t nwarps = loop_warps();
	if (total <= nwarps)
	{
		// one unit each, on as many SMs as there are units
		if (loop_warp() < total)
			f(loop_warp());
		return;
	}
	// high word: end of the claimed range, low word: its next unit
	__shared__ unsigned long long s_range;
	const uint32_t grab = min(max(total / (gridDim.x * 8), 4u), 16u);
	if (threadIdx.x == 0)
	{
		// a unit for each warp to begin with (total > nwarps), without a claim
		const uint32_t b = blockIdx.x * LOOP_WARPS;
		s_range = (unsigned long long)(b + LOOP_WARPS) << 32 | b;
	}
	__syncthreads();
	for (;;)
	{
		uint32_t unit = total;
		if (lane_id() == 0)
		{
			for (;;)
			{
				const unsigned long long r = atomicAdd(&s_range, 1ull);
				const uint32_t at = uint32_t(r), end = uint32_t(r >> 32);
				if (at < end)
				{
					unit = at;
					break;
				}
				if (end == total)
					break; // nothing lies past it
				if (at == end)
				{
					// this warp fetches the next range
					const uint32_t b = nwarps + atomicAdd(work, grab);
					if (b >= total)
					{
						atomicExch(&s_range, (unsigned long long)total << 32 | total);
						break;
					}
					atomicExch(&s_range, (unsigned long long)min(b + grab, total) << 32 | (b + 1));
					unit = b;
					break;
				}
				// another warp is fetching it: one atomic's round trip. After a second
				// or so the call ends with an error instead.
				uint32_t tries = 0;
				while ((uint32_t)(*(volatile unsigned long long *)&s_range >> 32) == end && ++tries < CLAIM_TRIES)
					__nanosleep(32);
				if (tries >= CLAIM_TRIES)
				{
					atomicOr(err, 1u);
					break;
				}
			}
		}
		unit = __shfl_sync(FULL, unit, 0);
		if (unit >= total)
			break;
		f(unit);
	}
}

// End of a phase: grid barrier; n gets the phase's appended triangles and mn,
// with scan set, its least support. False: leave.
__device__ __forceinline__ bool phase_end(LoopCtl *ctl, uint32_t &phase, uint32_t &n, uint32_t &mn, bool scan)
{
	__shared__ uint32_t s_n, s_mn, s_ok;
	__syncthreads();
	if (threadIdx.x == 0)
	{
		PhaseSlot *slot = &ctl->slot[phase & 3];
		if (blockIdx.x == 0)
			ctl->slot[(phase + 2) & 3] = PhaseSlot{0u, 0u, NO_SUPPORT, 0u};
		// the block's writes before its arrival
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&slot->arrived) : "memory");
		uint32_t spins = 0, ok = 1;
		unsigned long long t0 = 0, v;
		for (;;)
		{
			asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(slot) : "memory");
			if (uint32_t(v) >= gridDim.x)
				break;
			if ((++spins & 1023u) == 0)
			{
				if (__ldcg(&ctl->abort))
				{
					ok = 0;
					break;
				}
				const unsigned long long now = loop_ns();
				if (!t0)
					t0 = now;
				else if (now - t0 > LOOP_WAIT_LIMIT_NS)
					atomicExch(&ctl->abort, 1u);
			}
		}
		asm volatile("fence.acq_rel.gpu;" ::: "memory");
		s_n = uint32_t(v >> 32);
		if (scan)
			s_mn = __ldcg(&slot->mn);
		s_ok = ok;
	}
	__syncthreads();
	++phase;
	n = s_n;
	mn = s_mn;
	return s_ok != 0;
}

// Appends every live triangle with support <= hi to F and takes the minimum of
// the others. A warp reads up to 1024 supports per step, eight per thread at a
// time (two 16-byte loads), and appends them with one atomic. gone: the warp's
// steps that hold no live triangle any more and are passed by (its first 64: it
// takes the same ones in every scan). Ids of one source lie together and die at
// close levels: over all levels 35 % of the steps of R-MAT graphs are gone, 27 %
// of geometric ones (scans of R-MAT scale 18: 10.6 -> 8.2 ms, geometric graph of
// 1.1e8 triangles 4.3 -> 3.9).
__device__ __forceinline__ void scan_level(const LoopArgs &g, uint32_t hi, uint32_t *__restrict__ F, PhaseSlot *slot,
										   unsigned long long &gone)
{
	const uint32_t lane = lane_id();
	const uint64_t warp = loop_warp();
	// 1024 supports a step, 256 where that leaves warps without any
	const uint32_t chunks = g.T >= uint64_t(loop_warps()) * 1024 ? 4 : 1;
	const uint64_t stride = uint64_t(loop_warps()) * chunks * 256;
	uint32_t mn = NO_SUPPORT;
	uint32_t step = 0;
	for (uint64_t b0 = warp * chunks * 256; b0 < g.T; b0 += stride, ++step)
	{
		if (step < 64 && (gone >> step & 1ull))
			continue;
		uint32_t left = NO_SUPPORT;
		uint32_t mask = 0; // bit 8c + j: support j of this lane's chunk c
#pragma unroll
		for (uint32_t c = 0; c < 4; ++c)
		{
			if (c >= chunks)
				break;
			const uint64_t t0 = b0 + c * 256 + lane * 8;
			int32_t v[8];
			if (t0 + 8 <= g.T)
			{
				const int4 a = *reinterpret_cast<const int4 *>(g.S + t0);
				const int4 b = *reinterpret_cast<const int4 *>(g.S + t0 + 4);
				v[0] = a.x;
				v[1] = a.y;
				v[2] = a.z;
				v[3] = a.w;
				v[4] = b.x;
				v[5] = b.y;
				v[6] = b.z;
				v[7] = b.w;
			}
			else
			{
#pragma unroll
				for (uint32_t j = 0; j < 8; ++j)
					v[j] = t0 + j < g.T ? g.S[t0 + j] : -1;
			}
#pragma unroll
			for (uint32_t j = 0; j < 8; ++j)
				if (v[j] >= 0)
				{
					if (uint32_t(v[j]) <= hi)
						mask |= 1u << (c * 8 + j);
					else
						left = min(left, uint32_t(v[j]));
				}
		}
		mn = min(mn, left);
		if (step < 64 && !__any_sync(FULL, left != NO_SUPPORT))
			gone |= 1ull << step;
		if (!__ballot_sync(FULL, mask != 0))
			continue;
		uint32_t base = 0;
		const uint32_t total = __shfl_sync(FULL, warp_incl_scan(__popc(mask)), 31);
		if (lane == 0)
			base = atomicAdd(&slot->n, total);
		base = __shfl_sync(FULL, base, 0);
		for (uint32_t c = 0; c < chunks; ++c)
		{
			uint32_t z = (mask >> (c * 8)) & 0xffu;
			const uint32_t x = warp_incl_scan(__popc(z));
			uint32_t pos = base + x - __popc(z);
			while (z)
			{
				const uint32_t j = __ffs(z) - 1;
				z &= z - 1;
				if (pos < g.T)
					F[pos] = uint32_t(b0 + c * 256 + lane * 8 + j);
				else
					atomicOr(&g.ctl->c.error, 1u);
				++pos;
			}
			base += __shfl_sync(FULL, x, 31);
		}
	}
	// one atomic per block
	__shared__ uint32_t s_min;
	if (threadIdx.x == 0)
		s_min = NO_SUPPORT;
	__syncthreads();
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
		mn = min(mn, __shfl_xor_sync(FULL, mn, o));
	if (lane == 0 && mn != NO_SUPPORT)
		atomicMin(&s_min, mn);
	__syncthreads();
	if (threadIdx.x == 0 && s_min != NO_SUPPORT)
		atomicMin(&slot->mn, s_min);
}

// Order phase 1: the bits of F[0, n).
__device__ __forceinline__ void order_set(const LoopArgs &g, const uint32_t *F, uint32_t n)
{
	block_shares(n, [&](uint64_t i) {
		const uint32_t t = F[i];
		if (t < g.T)
			atomicOr(g.fbits + (t >> 5), 1u << (t & 31));
	});
}

// Order phase 2: the ids back to F, clearing the bits. A warp takes 128 words
// (4096 ids) at a time, in id order inside and in the order the warps reach
// them outside, which is close to id order.
__device__ __forceinline__ void order_write(const LoopArgs &g, uint32_t *__restrict__ F, PhaseSlot *slot)
{
	const uint32_t lane = lane_id();
	const uint64_t words = (g.T + 31) / 32;
	const uint64_t warp = loop_warp();
	const uint64_t stride = uint64_t(loop_warps()) * 128;
	for (uint64_t w0 = warp * 128; w0 < words; w0 += stride)
	{
		uint32_t z[4], cnt = 0;
#pragma unroll
		for (uint32_t c = 0; c < 4; ++c)
		{
			const uint64_t w = w0 + c * 32 + lane;
			z[c] = w < words ? g.fbits[w] : 0u;
			cnt += __popc(z[c]);
		}
		if (!__ballot_sync(FULL, cnt != 0))
			continue;
		const uint32_t total = __shfl_sync(FULL, warp_incl_scan(cnt), 31);
		uint32_t base = 0;
		if (lane == 0)
			base = atomicAdd(&slot->n, total);
		base = __shfl_sync(FULL, base, 0);
#pragma unroll
		for (uint32_t c = 0; c < 4; ++c)
		{
			const uint64_t w = w0 + c * 32 + lane;
			if (z[c])
				g.fbits[w] = 0;
			const uint32_t x = warp_incl_scan(__popc(z[c]));
			uint32_t pos = base + x - __popc(z[c]);
			while (z[c])
			{
				const uint32_t b = __ffs(z[c]) - 1;
				z[c] &= z[c] - 1;
				if (pos < g.T)
					F[pos] = uint32_t(w * 32 + b);
				++pos;
			}
			base += __shfl_sync(FULL, x, 31);
		}
	}
}

// Path: struct with
//   SMEM           bytes of dynamic shared memory per block
//   mark(t)        a triangle begins to die
//   retire(t)      it died in the round before
//   debit(g, F, nF, Fn, slot, level)  the debit phase (all threads call)
template <class Path>
__global__ void __launch_bounds__(LOOP_THREADS, 2) k_peel_loop(LoopArgs g, Path path)
{
	uint32_t phase = 0, n = 0, mn = 0;
	uint32_t nF = 0, nPrev = 0, cur = 0, level = 0xffffffffu, round = 0, rounds = 0;
	const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
	unsigned long long peeled = 0, ksum = 0, t_start = 0, t_last = 0, ns[4] = {0, 0, 0, 0};
	if (lead)
		t_start = t_last = loop_ns();
	__shared__ unsigned long long s_gone[LOOP_WARPS]; // see scan_level
	if (lane_id() == 0)
		s_gone[threadIdx.x >> 5] = 0;
	__syncwarp();
	bool ok = true, late = false;
	auto lap = [&](int kind) {
		if (lead)
		{
			const unsigned long long now = loop_ns();
			ns[kind] += now - t_last;
			t_last = now;
			if (now - t_start > LOOP_TIME_LIMIT_NS)
				late = true;
		}
	};
	while (peeled < g.T)
	{
		if (late) // the lead block leaves; the others find it at their next barrier
			atomicExch(&g.ctl->abort, 1u);
		if (__syncthreads_or(late))
		{
			ok = false;
			break;
		}
		uint32_t *F = cur ? g.F1 : g.F0, *Fp = cur ? g.F0 : g.F1;
		if (nF == 0)
		{
			// level change: level + 1 first, else the minimum of the rest
			unsigned long long gone = s_gone[threadIdx.x >> 5];
			scan_level(g, level + 1, F, &g.ctl->slot[phase & 3], gone);
			if (!(ok = phase_end(g.ctl, phase, n, mn, true)))
				break;
			++level;
			if (lead)
				g.ctl->scans++;
			if (n == 0)
			{
				if (mn == NO_SUPPORT)
					break; // nothing alive (cannot happen while peeled < T)
				level = mn;
				scan_level(g, level, F, &g.ctl->slot[phase & 3], gone);
				if (!(ok = phase_end(g.ctl, phase, n, mn, true)))
					break;
			}
			if (lane_id() == 0)
				s_gone[threadIdx.x >> 5] = gone;
			__syncwarp();
			nF = n;
			lap(2);
		}
		block_shares(uint64_t(nF) + nPrev, [&](uint64_t i) {
			if (i < nF)
			{
				const uint32_t t = F[i];
				g.S[t] = ~int32_t(level);
				if (g.R)
					g.R[t] = round;
				path.mark(t);
			}
			else
				path.retire(Fp[i - nF]);
		});
		if (!(ok = phase_end(g.ctl, phase, n, mn, false)))
			break;
		lap(0);
		path.debit(g, F, nF, Fp, &g.ctl->slot[phase & 3], int32_t(level));
		if (!(ok = phase_end(g.ctl, phase, n, mn, false)))
			break;
		lap(1);
		peeled += nF;
		ksum += (unsigned long long)level * nF;
		++rounds;
		++round;
		nPrev = nF;
		nF = n;
		cur ^= 1u;
		if (nF >= g.sort_min && nF <= g.T && g.fbits)
		{
			order_set(g, Fp, nF);
			uint32_t unused, m2;
			if (!(ok = phase_end(g.ctl, phase, unused, m2, false)))
				break;
			order_write(g, Fp, &g.ctl->slot[phase & 3]);
			if (!(ok = phase_end(g.ctl, phase, unused, m2, false)))
				break;
			if (lead)
				g.ctl->ordered++;
			lap(3);
		}
	}
	// k from the support words: a pass in order at the end in place of a second
	// scattered write per triangle in the mark phases (geometric graph of 1.1e8
	// triangles: peel 50.9 -> 49.4 ms; R-MAT scale 18: 171 -> 169)
	if (ok)
		block_shares(g.T, [&](uint64_t t) { g.K[t] = ~g.S[t]; });
	if (lead)
	{
		PeelCtl &c = g.ctl->c;
		c.peeled = peeled;
		c.ksum = ksum;
		c.kmax = peeled ? level : 0u;
		c.unpeeled = uint32_t(g.T - peeled);
		c.rounds = rounds;
		c.round = round;
		c.level = level;
		c.done = ok;
		for (int i = 0; i < 4; ++i)
			g.ctl->ns[i] = ns[i];
		if (!ok)
			g.ctl->timed_out = 1;
	}
}

// Runs the loop on the context's stream and waits for it (peel_loop.cu holds
// the rest of the host side).
struct LoopBuffers
{
	LoopCtl *ctl = nullptr;
	uint32_t *R = nullptr, *F0 = nullptr, *F1 = nullptr, *fbits = nullptr;
};
int loop_alloc(Ctx &c, LoopBuffers &b);
void loop_release(Ctx &c, LoopBuffers &b);
int loop_finish(Ctx &c, LoopBuffers &b, PeelCtl *hctl);

template <class Path>
int run_peel_loop(Ctx &c, LoopBuffers &b, const Path &path, int32_t *S, int32_t *K)
{
	int per_sm = 0;
	if (cudaFuncSetAttribute(k_peel_loop<Path>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Path::SMEM)) !=
			cudaSuccess ||
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_peel_loop<Path>, LOOP_THREADS, Path::SMEM) !=
			cudaSuccess ||
		per_sm < 1)
		return fail(NUCLEUS34_E_CUDA, "peel loop occupancy");
	const nucleus34_tune tn = tune_filled(c.tune);
	LoopArgs g{b.ctl, S, K, b.R, b.F0, b.F1, b.fbits, c.T, 0xffffffffu};
	// Frontiers are put in id order from T / 2^(sort_shift - 3) triangles on (an
	// eighth of the list form's rule: the append buffers leave runs of
	// neighbours), on graphs of 2^24 triangles and more, whose supports alone
	// are as large as half of L2, and wherever the caller pins a threshold. Peel of R-MAT scale 18 (8.3e7 triangles) with
	// T/2^14, 2^12, 2^9, never: 176, 172, 170, 173 ms; geometric, 1.1e8: 53.4,
	// 53.2, 52.9, 57.2; R-MAT scale 16 (1.6e7) 35.5, 35.5, 33.4, 32.0; geometric,
	// 2e7: 9.8, 9.7, 9.6, 9.5.
	if (tn.sort_shift != NUCLEUS34_TUNE_NEVER && (c.T >= ORDER_MIN_TRIANGLES || c.order_pinned))
		g.sort_min = uint32_t(std::max<uint64_t>(c.T >> (tn.sort_shift > 3 ? tn.sort_shift - 3 : 0), 4096));
	// as many blocks as fit at once, fewer for small graphs, whose frontiers do
	// not fill them (a quarter as many blocks: 19% slower on R-MAT scale 12; one
	// per SM: 17 to 20% slower on the direct variant's graphs of 3M triangles)
	uint64_t blocks = (c.T + LOOP_THREADS * 4 - 1) / (LOOP_THREADS * 4);
	blocks = std::min<uint64_t>(std::max<uint64_t>(blocks, 4), uint64_t(per_sm) * uint64_t(c.sm_count));
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(uint32_t(blocks));
	cfg.blockDim = dim3(LOOP_THREADS);
	cfg.dynamicSmemBytes = Path::SMEM;
	cfg.stream = c.stream;
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeCooperative;
	at[0].val.cooperative = 1;
	cfg.attrs = at;
	cfg.numAttrs = 1;
	if (cudaLaunchKernelEx(&cfg, k_peel_loop<Path>, g, path) != cudaSuccess)
		return fail(NUCLEUS34_E_CUDA, std::string("peel loop: ") + cudaGetErrorString(cudaGetLastError()));
	c.launches++;
	return NUCLEUS34_OK;
}

} // namespace n34
