// Host side of the one-launch peel (peel_loop.cuh): its buffers and results.
#include "pipeline.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "peel_loop.cuh"

namespace n34 {

namespace {

__global__ void k_loop_init(LoopCtl *ctl)
{
	LoopCtl z{};
	for (int i = 0; i < 4; ++i)
		z.slot[i].mn = NO_SUPPORT;
	*ctl = z;
}

} // namespace

int loop_alloc(Ctx &c, LoopBuffers &b)
{
	const uint64_t T = c.T;
	if (c.opt_flags & NUCLEUS34_OPT_VERIFIABLE)
		N34_TRY(dalloc(c, &b.R, T, "peel death rounds"));
	N34_TRY(dalloc(c, &b.F0, T, "frontier 0"));
	N34_TRY(dalloc(c, &b.F1, T, "frontier 1"));
	N34_TRY(dalloc(c, &b.ctl, 1, "peel control"));
	// the ordering bitmap is optional: without it frontiers keep their order
	if (dalloc(c, &b.fbits, (T + 31) / 32, "frontier order bitmap"))
	{
		b.fbits = nullptr;
		clear_error();
	}
	else
		N34_CUDA(cudaMemsetAsync(b.fbits, 0, (T + 31) / 32 * 4, c.stream));
	N34_LAUNCH(c, k_loop_init, 1, 1, 0, b.ctl);
	return NUCLEUS34_OK;
}

void loop_release(Ctx &c, LoopBuffers &b)
{
	c.release(b.R);
	c.release(b.F0);
	c.release(b.F1);
	c.release(b.ctl);
	c.release(b.fbits);
	b = LoopBuffers{};
}

int loop_finish(Ctx &c, LoopBuffers &b, PeelCtl *hctl)
{
	LoopCtl h{};
	if (cudaMemcpyAsync(&h, b.ctl, sizeof(LoopCtl), cudaMemcpyDeviceToHost, c.stream) != cudaSuccess ||
		cudaStreamSynchronize(c.stream) != cudaSuccess)
		return fail(NUCLEUS34_E_CUDA, std::string("peel loop: ") + cudaGetErrorString(cudaGetLastError()));
	*hctl = h.c;
	if (h.timed_out)
		return fail(NUCLEUS34_E_TIMEOUT, "peel did not end within its time bounds");
	if (h.c.error)
		return fail(NUCLEUS34_E_CUDA, "internal: peel check failed (frontier overflow)");
	if (c.opt_flags & NUCLEUS34_OPT_PROFILE_PEEL)
	{
		std::fprintf(stderr,
					 "[peel-profile] rounds=%u scans=%u ordered=%u mark=%.3fms debit=%.3fms scan=%.3fms order=%.3fms\n",
					 h.c.rounds, h.scans, h.ordered, h.ns[0] * 1e-6, h.ns[1] * 1e-6, h.ns[2] * 1e-6, h.ns[3] * 1e-6);
		c.peel_debit_sec = h.ns[1] * 1e-9;
	}
	if (b.R)
	{
		c.dR = b.R; // kept for nucleus34_ctx_verify
		b.R = nullptr;
	}
	return NUCLEUS34_OK;
}

} // namespace n34
