// Stages of the device pipeline and the data they hand to each other.
#pragma once

#include "common.cuh"

namespace n34 {

// Edge -> triangle incidence, per edge sorted by third vertex. Edge e's list
// is [span[e].x, span[e].y) in third[] / tri[] (32-bit positions: the
// incidence holds 3T < 2^32 entries). The peel may shorten a list in place
// (dead entries dropped, span[e].y lowered); begins never move.
struct Incidence
{
	uint2 *span = nullptr;     // m
	uint32_t *third = nullptr; // 3T
	uint32_t *tri = nullptr;   // 3T
	// optional (on-demand peel with death flags): tpos[3t + r] = position of
	// triangle t's entry under its edge b (r=0), a (r=1), c (r=2)
	uint32_t *tpos = nullptr;
	unsigned long long sum_te_sq = 0; // sum over edges of (list length)^2
};

// Bit of an incidence entry's tri word that marks a peeled triangle (on-demand
// peel with death flags; the incidence is discarded after the peel).
constexpr uint32_t INC_DEAD = 0x80000000u;
// Most triangles the on-demand peel keeps its death flags in the incidence
// for (ids leave the top two bits of a tri word free); above it the slower
// round-stamp peel runs. Union passes (batched form, serving) are cut below it,
// as a pass may have to run on the lists; the bit form itself has no such limit.
constexpr uint64_t FLAG_PEEL_MAX_TRIANGLES = 0x3fffffffull;

// The triangle listing's bit matrices, kept for the bit form of both variants.
// Source u of out-degree d has a d x d matrix of W = ceil(d / 32) cells per row. Row
// ia belongs to edge O[u] + ia, so an edge stands for its row.
struct BitMats
{
	// x, y: bit ib of row ia is the triangle with head edge a = O[u] + ia and
	// tail edge b = O[u] + ib; its id is y + the set bits of x below it.
	// z: symmetric (bit i of row j and bit j of row i are the triangle of u
	// with the vertices at i and j); the peel clears both when it is dead.
	// w: symmetric, zero at first; the peel sets both when it begins to die.
	// One 16-byte load tells a triangle's id and state.
	uint4 *cells = nullptr;
	// per oriented edge, in the same allocation: {first cell of its row, W << 16 | its position in
	// N+(u), first cell of its in-row, its column among its head's in-edges}
	uint4 *erec = nullptr;
	uint64_t nwords = 0;
};

// The same for the triangles that lie on an edge as its c edge. Edge u -> v has
// an in-row of ceil(in-degree of u / 32) cells over u's in-edges y -> u (in any
// order, or by y: see build_in_rows): a bit is the triangle (y, u, v).
struct InMats
{
	uint4 *cells = nullptr; // as above, y counting positions in tri
	uint32_t *tri = nullptr; // triangle ids, in-row by in-row
	uint2 *live = nullptr;  // per oriented edge: {triangles of its in-row not dead, cells of the in-row}
	uint64_t nwords = 0;
	unsigned long long sum_te_sq = 0; // sum over edges of (triangles on the edge)^2
	// with by_source only (the direct variant's clique list): every vertex's
	// in-edges as y << 32 | edge, ascending, and where they start
	unsigned long long *in_edges = nullptr; // m
	uint64_t *in_off = nullptr;             // n + 1
};

// Triangle -> four-clique incidence of the direct variant.
struct CliqueCsr
{
	uint64_t *off = nullptr; // T+1
	uint32_t *ids = nullptr; // 4Q clique ids
};

int build_src(Ctx &c);
// Triangle-listing passes on caller-owned memory (no bitmap cache).
cudaError_t launch_tri_count(const uint32_t *O, const uint32_t *E, uint64_t n, uint32_t *cnt, int sm_count,
							 cudaStream_t s);
cudaError_t launch_tri_write(const uint32_t *O, const uint32_t *E, uint64_t n, const uint64_t *toff,
							 uint32_t *tris, int sm_count, cudaStream_t s);
int list_triangles(Ctx &c, BitMats *keep, uint64_t keep_min);
void free_mats(Ctx &c, BitMats &mats);
// lean: no 64-bit key array (entries sorted in place as pairs) and no tpos.
int build_incidence(Ctx &c, Incidence &inc, bool want_tpos, bool lean = false);
void free_incidence(Ctx &c, Incidence &inc);
// Sorts every segment [off[s], off[s+1]) of keys ascending (incidence.cu's
// segmented sort; nseg < 2^32).
int sort_segments_u64(Ctx &c, unsigned long long *keys, const uint64_t *off, uint64_t nseg);
// Oriented CSR of an edge list built on the device and made resident in c
// (csr_build.cu), with the host build's semantics.
int upload_edges(Ctx &c, const uint32_t *src, const uint32_t *dst, uint64_t count);
// support[t] = number of four-cliques on t; returns sum(support) in *total.
// own (optional): cliques whose lowest triangle is t (direct variant sizes).
int count_support(Ctx &c, const Incidence &inc, int32_t *support, uint64_t *total, uint32_t *own);
// Direct variant: canonical clique list (c.dquds, c.Q) and triangle->clique CSR.
int list_cliques(Ctx &c, const Incidence &inc, const int32_t *support, const uint32_t *own, CliqueCsr &csr);
void free_clique_csr(Ctx &c, CliqueCsr &csr);
// Per-segment statistics of a batched (disjoint union) run; no-ops when the
// context holds a single graph. After listing: triangle offsets per member
// graph; after the support count: clique counts; after the peel: k max/sum.
int segments_after_listing(Ctx &c);
int segments_after_support(Ctx &c, const int32_t *support);
int segments_after_peel(Ctx &c);
// The bit-matrix form of the support count, the clique list and the peel.
bool bit_form_wanted(const Ctx &c, int variant);
// Builds the in-rows; *fits is false, and nothing is left, when they and what
// the form needs beside them exceed the room left, or when the lists are the less
// work. In the direct variant columns ascend with the in-edge's source (by_source).
int build_in_rows(Ctx &c, const BitMats &mats, InMats &in, int variant, bool *fits);
void free_in_rows(Ctx &c, InMats &in);
// own (optional, needs by_source): cliques whose lowest triangle is t. *acyclic:
// no three vertices above one source form a directed cycle (the rows would take
// them for a clique).
int count_support_bits(Ctx &c, const BitMats &mats, const InMats &in, int32_t *support, uint64_t *total,
					   uint32_t *own, bool *acyclic);
// Direct variant: the clique list and, where the peel uses them in place of the
// rows (which it then gives back), the triangle -> clique lists.
int list_cliques_bits(Ctx &c, BitMats &mats, InMats &in, const int32_t *support, const uint32_t *own,
					  CliqueCsr &csr);
int peel_bits(Ctx &c, const BitMats &mats, const InMats &in, int32_t *support, int32_t *K, PeelCtl *hctl);
// The direct variant's peel over the clique list.
int peel_direct(Ctx &c, const CliqueCsr &csr, int32_t *support, int32_t *K, PeelCtl *hctl);
// Device-resident peel of the on-demand variant's list form; K receives the final k of every triangle.
int peel(Ctx &c, const Incidence &inc, int32_t *support, int32_t *K, PeelCtl *hctl);

// Certificate check of the last run (verify.cu); needs the kept death rounds.
int verify(Ctx &c, uint64_t *violations, uint64_t *checked);
// Context entry points shared by the C-ABI front ends (api.cu, batch.cu).
int upload(Ctx &c, const nucleus34_csr *csr);
int run(Ctx &c, int variant, nucleus34_result *out);
int copy_to_host(Ctx &c, void *dst, const void *src, uint64_t bytes);
int create_ctx(const nucleus34_opts *opts, nucleus34_ctx *out);
void destroy_ctx(nucleus34_ctx x);

} // namespace n34

struct nucleus34_ctx_s
{
	n34::Ctx c;
};
