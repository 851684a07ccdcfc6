// The four boundary sides of a domain as one launch.
//
// The reference draws East, North, West, South one after another (engine.cpp:1342-1438), each side
// reading what the earlier ones wrote.  Two sides meet only in a corner, so the strips split into
// eight rectangles that touch no common texel: four segments, where one side alone writes and reads
// texels that no side writes (or the texel itself), and four corners, in which one CTA takes its two
// sides in order with a barrier between them.  A wall reads texels up to 4 (W, S) or from n - 2
// (E, N), so a corner reaches to those as well as to the strips' ends.
#pragma once

#include <algorithm>

#include "celeris_internal.hpp"

namespace cel {

struct Rect { int x0, y0, x1, y1; };   // texels [x0, x1) x [y0, y1)

constexpr int BND_REGIONS = 8;         // segments of the sides N, E, S, W, then the corners EN, NW, ES, WS
// The sides of corner EN, NW, ES, WS (0 .. 3) in drawing order (0 = N, 1 = E, 2 = S, 3 = W); q = 0, 1.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int corner_side(int corner, int q) {
    return q == 0 ? (corner == 1 ? 0 : corner == 3 ? 3 : 1) : (corner == 0 ? 0 : corner == 1 ? 3 : 2);
}
// The plain form takes a corner in one CTA; with larger ones (two very wide sponges) each side keeps its launch.
constexpr int BND_CORNER_MAX = 16384;

// How a corner may be cut into pieces that take its two sides independently: a wall reads texels along its
// own axis only, and every other kind the texel itself.
enum CornerCut { CUT_NONE, CUT_ROWS, CUT_COLUMNS };
inline CornerCut corner_cut(int corner, const int type[4]) {
    const int a = corner_side(corner, 0), b = corner_side(corner, 1);
    const int xside = (a == 1 || a == 3) ? a : b, yside = a + b - xside;
    return type[yside] != CEL_BC_SOLID ? CUT_ROWS : type[xside] != CEL_BC_SOLID ? CUT_COLUMNS : CUT_NONE;
}

// put(Rect): the corner r cut into pieces of at most `cells` texels (or one row or column of a wall's corner), each
// of which takes the two sides by itself.  Where neither side is a wall every texel stands alone, and the
// corner is cut both ways: in whole rows, a wave-maker along a sponge of 2000 cells left two rows to two CTAs
// (compensated form, 64 waves, 8192 x 64 cells: 778 us a step, 4000 cells 1413; cut both ways 188 and 222).
template <class F>
inline void corner_pieces(int corner, const int type[4], const Rect& r, int cells, F&& put) {
    if (r.x1 <= r.x0 || r.y1 <= r.y0) return;
    const int a = corner_side(corner, 0), b = corner_side(corner, 1);
    const CornerCut cut = corner_cut(corner, type);
    int w = r.x1 - r.x0, h = r.y1 - r.y0;
    if (type[a] != CEL_BC_SOLID && type[b] != CEL_BC_SOLID) {
        w = std::min(w, cells);
        h = std::min(h, std::max(1, cells / w));
    } else if (cut == CUT_ROWS) {
        h = std::min(h, std::max(1, cells / w));
    } else if (cut == CUT_COLUMNS) {
        w = std::min(w, std::max(1, cells / h));
    }
    for (int y = r.y0; y < r.y1; y += h)
        for (int x = r.x0; x < r.x1; x += w) put(Rect{x, y, std::min(x + w, r.x1), std::min(y + h, r.y1)});
}

// Fills the eight rectangles (empty ones have no texels); false where the sides have to be launched
// one after another: walls wide enough to read their own strip (W, S from 3, E, N from 4 cells), or
// a domain so small that opposite corners meet.
inline bool plan_boundary(int nx, int ny, const int type[4], const int width[4], Rect out[BND_REGIONS]) {
    const int NX = nx + 4, NY = ny + 4;
    auto wall = [&](int s) { return type[s] == CEL_BC_SOLID && width[s] > 0; };
    if ((wall(0) && width[0] > 3) || (wall(1) && width[1] > 3) || (wall(2) && width[2] > 2) || (wall(3) && width[3] > 2))
        return false;
    const int w[4] = {std::min(width[0], NY), std::min(width[1], NX), std::min(width[2], NY), std::min(width[3], NX)};
    const int xe = std::min(NX - w[1], wall(1) ? nx - 2 : NX), yn = std::min(NY - w[0], wall(0) ? ny - 2 : NY);
    const int xw = std::max(w[3], wall(3) ? 4 : 0), ys = std::max(w[2], wall(2) ? 4 : 0);
    if (xw > xe || ys > yn) return false;
    out[0] = {xw, NY - w[0], xe, NY};
    out[1] = {NX - w[1], ys, NX, yn};
    out[2] = {xw, 0, xe, w[2]};
    out[3] = {0, ys, w[3], yn};
    out[4] = {xe, yn, NX, NY};
    out[5] = {0, yn, xw, NY};
    out[6] = {xe, 0, NX, ys};
    out[7] = {0, 0, xw, ys};
    for (int k = 4; k < BND_REGIONS; ++k)
        if ((long long)(out[k].x1 - out[k].x0) * (out[k].y1 - out[k].y0) > BND_CORNER_MAX) return false;
    return true;
}

}  // namespace cel
