// The pieces of the boundary corners (boundary_plan.hpp) over random domains, side types and widths: they cover
// a corner once, none is more work than an item (or than two walls' corner, which cannot be cut), and taking
// them in any order gives what the sides drawn one after another give, on symbolic texel values.  Prints
// "corners uncovered too_large wrong".
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "boundary_plan.hpp"

using namespace cel;
typedef uint64_t u64;

static u64 mix(u64 a, u64 b) {
    u64 x = (a ^ (b * 0x9E3779B97F4A7C15ull)) + 0x7F4A7C15ull + (a << 6);
    x ^= x >> 29;
    x *= 0xBF58476D1CE4E5B9ull;
    return x ^ (x >> 32);
}

int main() {
    std::mt19937 r(7);
    long corners = 0, uncovered = 0, too_large = 0, wrong = 0;
    for (int it = 0; it < 20000; ++it) {
        const int nx = 2 + r() % 70, ny = 2 + r() % 70, NX = nx + 4, NY = ny + 4;
        int type[4], width[4];
        for (int s = 0; s < 4; ++s) {
            type[s] = r() % 5;
            width[s] = type[s] == CEL_BC_SOLID ? r() % 4 : r() % 3 ? r() % 12 : r() % 60;
        }
        Rect R[BND_REGIONS];
        if (!plan_boundary(nx, ny, type, width, R)) continue;
        const int cells = 1 << (r() % 8);
        auto strip = [&](int s) {
            const int w = width[s];
            return s == 0 ? Rect{0, std::max(NY - w, 0), NX, NY} : s == 1 ? Rect{std::max(NX - w, 0), 0, NX, NY}
                 : s == 2 ? Rect{0, 0, NX, std::min(w, NY)} : Rect{0, 0, std::min(w, NX), NY};
        };
        auto meet = [](Rect a, const Rect& b) {
            return Rect{std::max(a.x0, b.x0), std::max(a.y0, b.y0), std::min(a.x1, b.x1), std::min(a.y1, b.y1)};
        };
        auto draw = [&](std::vector<u64>& v, int s, const Rect& q) {   // side s on the texels of q
            const std::vector<u64> src = v;
            for (int y = q.y0; y < q.y1; ++y)
                for (int x = q.x0; x < q.x1; ++x) {
                    int qx = x, qy = y;
                    if (type[s] == CEL_BC_SOLID) {   // mirrored: 3 - x, 2 n + 1 - x
                        if (s == 3) qx = 3 - x;
                        if (s == 1) qx = 2 * nx + 1 - x;
                        if (s == 2) qy = 3 - y;
                        if (s == 0) qy = 2 * ny + 1 - y;
                    }
                    const bool in = qx >= 0 && qy >= 0 && qx < NX && qy < NY;
                    const u64 from = type[s] > CEL_BC_SPONGE ? u64(y) * 1000 + x : in ? src[size_t(qy) * NX + qx] : 0;
                    v[size_t(y) * NX + x] = mix(from, 10 * type[s] + s + 1);
                }
        };
        std::vector<u64> pre(size_t(NX) * NY);
        for (u64& v : pre) v = (u64(r()) << 32) | r();
        std::vector<u64> want = pre, got = pre;
        for (int s : {1, 0, 3, 2}) draw(want, s, strip(s));
        struct Item { int k; Rect q; };
        std::vector<Item> items;
        for (int k = 0; k < 4; ++k) items.push_back({k, R[k]});
        for (int k = 4; k < BND_REGIONS; ++k) {
            const Rect& c = R[k];
            if (c.x1 <= c.x0 || c.y1 <= c.y0) continue;
            ++corners;
            std::vector<int> seen(size_t(NX) * NY, 0);
            corner_pieces(k - 4, type, c, cells, [&](const Rect& q) {
                items.push_back({k, q});
                if ((q.x1 - q.x0) * (q.y1 - q.y0) > std::max(cells, 36)) ++too_large;
                for (int y = q.y0; y < q.y1; ++y)
                    for (int x = q.x0; x < q.x1; ++x) ++seen[size_t(y) * NX + x];
            });
            for (int y = 0; y < NY; ++y)
                for (int x = 0; x < NX; ++x)
                    if (seen[size_t(y) * NX + x] != (x >= c.x0 && x < c.x1 && y >= c.y0 && y < c.y1)) { ++uncovered; x = NX; y = NY; }
        }
        std::shuffle(items.begin(), items.end(), r);
        for (const Item& i : items)
            for (int q = 0; q < (i.k < 4 ? 1 : 2); ++q) {
                const int s = i.k < 4 ? i.k : corner_side(i.k - 4, q);
                const Rect m = meet(i.q, strip(s));
                if (m.x1 > m.x0 && m.y1 > m.y0) draw(got, s, m);
            }
        if (got != want) ++wrong;
    }
    std::printf("%ld %ld %ld %ld\n", corners, uncovered, too_large, wrong);
    return 0;
}
