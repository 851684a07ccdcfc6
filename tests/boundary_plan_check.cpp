// Compares the one-launch split of the boundary sides (boundary_plan.hpp) with the sides drawn one
// after another, over random domains, side types and widths, on symbolic texel values; also checks that
// no region reads or writes what another one writes.  Prints "planned refused wrong races".
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "boundary_plan.hpp"

using namespace cel;
typedef uint64_t u64;

static u64 mix(u64 a, u64 b) {
    u64 x = a * 0x9E3779B97F4A7C15ull ^ (b + 0x7F4A7C15ull + (a << 6) + (a >> 2));
    x ^= x >> 29;
    x *= 0xBF58476D1CE4E5B9ull;
    return x ^ (x >> 32);
}
static int mirror(int c, int x) { return int(float(c) - (float(x) + 0.5f)); }

int main() {
    std::mt19937 r(1);
    long planned = 0, refused = 0, wrong = 0, races = 0;
    for (int it = 0; it < 60000; ++it) {
        const int nx = 2 + r() % (it % 3 ? 40 : 9), ny = 2 + r() % (it % 3 ? 40 : 9);
        int type[4], width[4];
        for (int s = 0; s < 4; ++s) {
            type[s] = r() % 5;
            width[s] = type[s] == CEL_BC_SOLID ? r() % 5 : r() % 12;
        }
        Rect R[BND_REGIONS];
        if (!plan_boundary(nx, ny, type, width, R)) { ++refused; continue; }
        ++planned;
        const int NX = nx + 4, NY = ny + 4;
        std::vector<u64> pre(size_t(NX) * NY);
        for (u64& v : pre) v = (u64(r()) << 32) | r();
        auto strip = [&](int s) {
            Rect q = s == 0 ? Rect{0, NY - width[0], NX, NY} : s == 1 ? Rect{NX - width[1], 0, NX, NY}
                   : s == 2 ? Rect{0, 0, NX, width[2]} : Rect{0, 0, width[3], NY};
            return Rect{std::max(0, q.x0), std::max(0, q.y0), std::min(NX, q.x1), std::min(NY, q.y1)};
        };
        // a side's value at a texel; reads: the texel it comes from
        auto value = [&](const std::vector<u64>& src, int s, int x, int y, std::vector<int>* reads) -> u64 {
            if (type[s] == CEL_BC_SOLID) {
                int qx = x, qy = y;
                if (s == 3) qx = mirror(4, x);
                else if (s == 1) qx = mirror(2 * nx + 2, x);
                else if (s == 2) qy = mirror(4, y);
                else qy = mirror(2 * ny + 2, y);
                if (qx < 0 || qy < 0 || qx >= NX || qy >= NY) return mix(0, s + 1);
                if (reads) reads->push_back(qy * NX + qx);
                return mix(src[size_t(qy) * NX + qx], s + 1);
            }
            if (type[s] == CEL_BC_SPONGE) {
                if (reads) reads->push_back(y * NX + x);
                return mix(src[size_t(y) * NX + x], 100 + s);
            }
            return mix(u64(y) * 1000 + x, 200 + s + type[s] * 10);
        };
        std::vector<u64> want = pre;
        for (int s : {1, 0, 3, 2}) {
            const Rect q = strip(s);
            const std::vector<u64> src = want;
            for (int y = q.y0; y < q.y1; ++y)
                for (int x = q.x0; x < q.x1; ++x) want[size_t(y) * NX + x] = value(src, s, x, y, nullptr);
        }
        // the regions, the corners cut into single rows or columns where that is allowed
        struct Piece { int k; Rect r; };
        std::vector<Piece> pieces;
        for (int k = 0; k < BND_REGIONS; ++k) {
            const CornerCut cut = k < 4 ? CUT_NONE : corner_cut(k - 4, type);
            if (cut == CUT_ROWS)
                for (int y = R[k].y0; y < R[k].y1; ++y) pieces.push_back({k, {R[k].x0, y, R[k].x1, y + 1}});
            else if (cut == CUT_COLUMNS)
                for (int x = R[k].x0; x < R[k].x1; ++x) pieces.push_back({k, {x, R[k].y0, x + 1, R[k].y1}});
            else
                pieces.push_back({k, R[k]});
        }
        std::vector<int> writer(pre.size(), -1);
        std::vector<std::vector<int>> reads(pieces.size());
        std::vector<u64> got = pre;
        for (int q = 0; q < int(pieces.size()); ++q) {
            const int k = pieces[q].k;
            const Rect rect = pieces[q].r;
            std::vector<u64> local = pre;   // a region sees the state before the launch, and its own writes
            for (int turn = 0; turn < (k < 4 ? 1 : 2); ++turn) {
                const int s = k < 4 ? k : corner_side(k - 4, turn);
                Rect t = strip(s);
                t = {std::max(t.x0, rect.x0), std::max(t.y0, rect.y0), std::min(t.x1, rect.x1), std::min(t.y1, rect.y1)};
                const std::vector<u64> src = local;
                for (int y = t.y0; y < t.y1; ++y)
                    for (int x = t.x0; x < t.x1; ++x) {
                        const int e = y * NX + x;
                        const size_t seen = reads[q].size();
                        local[e] = got[e] = value(src, s, x, y, &reads[q]);
                        if (writer[e] >= 0 && writer[e] != q) ++races;
                        writer[e] = q;
                        for (size_t i = seen; i < reads[q].size(); ++i) {   // written in place in the same sweep
                            const int ry = reads[q][i] / NX, rx = reads[q][i] % NX;
                            if (reads[q][i] != e && rx >= t.x0 && rx < t.x1 && ry >= t.y0 && ry < t.y1) ++races;
                        }
                    }
            }
        }
        for (int q = 0; q < int(pieces.size()); ++q)
            for (int e : reads[q])
                if (writer[e] >= 0 && writer[e] != q) ++races;
        if (got != want) ++wrong;
    }
    std::printf("%ld %ld %ld %ld\n", planned, refused, wrong, races);
    return 0;
}
