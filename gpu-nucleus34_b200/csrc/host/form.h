// When a decomposition runs on the listing's bit matrices (the bit form) and when
// on incidence lists: host-only arithmetic, shared by the device code that asks and
// by tests without a GPU.
#pragma once

#include "nucleus34.h"

#include <cstdint>

namespace n34 {

// The rows are worth their words: every triangle's words are read in the support
// count and once more when it dies, however few bits they hold, where the lists
// cost by what they hold. `lists` is the lesser of the entries on the triangles'
// head and tail edges (those with the edge as head or tail: the others are not
// counted before the in-rows are built). Words and entries of R-MAT and geometric
// graphs are 0.1 to 1.1 to one. Hubs that are joined to each other and to many
// vertices of degree 1 to 3 (in-rows long and nearly empty) cross over between
// 2.9 and 4.7 on demand, where the lists' rounds take longer (incidence, support
// and peel, rows against lists, ms: 8.1 and 14.1 at 1.1, 14.7 and 15.6 at 2.9,
// 20.5 and 15.6 at 4.7, 94 and 33 at 26), and between 1.5 and 2 in the direct
// variant, which peels over the clique list in either form (19.7 and 25 at 1.5,
// 19.0 and 15.5 at 2.0, 237 and 32 at 26). On demand the lists also take 1 to 2
// ms for the launches of their rounds: the time of 1e8 words.
inline bool rows_pay(int variant, uint64_t words, uint64_t lists)
{
	return variant == NUCLEUS34_DIRECT ? words <= lists + lists / 2 : words <= 3 * lists + lists / 2 + 100000000;
}

// From this many triangles on the listing keeps its matrices: building in-rows is
// several passes over the edges, whatever the triangles. On demand that is 0.03
// ns an edge against 1 ms for the launches of the lists' rounds (if any: road-like
// grids have no cliques); the direct variant also sorts the in-edges, 0.2 ns an
// edge, and has no such launches. Incidence, support, cliques and peel, rows against
// lists, ms: on demand, 2e6 edges and 2e5 triangles 0.25 and 0.26, 3.2e7 and 6e5
// 1.86 and 0.98, 1.2e7 and 4e4 (with rounds) 1.2 and 1.5; direct, 8e6 and 1.5e6
// 2.0 and 1.3, 6e6 and 3.5e6 2.76 and 2.81, 1e7 and 1e7 5.7 and 7.4.
inline uint64_t rows_least_triangles(int variant, uint64_t m)
{
	return variant == NUCLEUS34_DIRECT ? m / 2 : m > (uint64_t(1) << 23) ? m / 16 : 0;
}

// The in-rows (cells of 16 bytes) and their triangles, the counts; then support, k,
// two frontiers, the ordering bitmap and, if kept, the death rounds. Cells are
// addressed by 32 bits, by warps that step over 32 at a time and must not wrap.
inline bool rows_fit(uint64_t cells, uint64_t T, uint64_t m, bool rounds, uint64_t room)
{
	return cells <= 0xffffffffull - 31 && 16 * cells + (rounds ? 24 : 20) * T + T / 8 + 16 * m + (uint64_t(1) << 20) <= room;
}

} // namespace n34
