// A serial model of the Danielsson block iteration (csrc/k_dan_blocks.cu), for
// the CPU test of its round limit (csrc/dan_rounds.h): the same blocks, inputs,
// first guesses, comparisons and rounds, with each row's x passes as the plain
// loops they stand for.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "dan_rounds.h"

namespace {

struct Cell {
    int16_t x, y, z;
    bool operator!=(const Cell& o) const { return x != o.x || y != o.y || z != o.z; }
};
struct Opt {   // a cell or none
    bool has;
    Cell c;
    bool operator!=(const Opt& o) const { return has != o.has || (has && c != o.c); }
};
using Row = std::vector<Opt>;

int32_t len(Cell c)
{
    return (int32_t)((uint32_t)((int)c.x * c.x) + (uint32_t)((int)c.y * c.y) + (uint32_t)((int)c.z * c.z));
}
Cell add(Cell c, int x, int y, int z)
{
    return Cell{(int16_t)(c.x + x), (int16_t)(c.y + y), (int16_t)(c.z + z)};
}
void take(Cell& own, const Opt& from, int x, int y, int z)
{
    if (!from.has) return;
    const Cell c = add(from.c, x, y, z);
    if (len(own) > len(c)) own = c;
}

struct Model {
    int w, h, d, cw, R, Z, BX, dir, zfirst, nchain, nc, nx, nk;
    std::vector<Cell> A;
    struct Out {   // what a block's run leaves, per slice of its chain part
        std::vector<std::vector<Row>> rows;   // [slice][row]: results
        std::vector<Row> down;                // [slice]: last row after the down sweep
        std::vector<std::vector<Opt>> right, left;   // [slice][step]: side cells
    };
    std::vector<Out> cur;

    Cell a(int x, int y, int z) const { return A[((size_t)z * h + y) * w + x]; }
    int block(int k, int c, int xb) const { return (k * nc + c) * nx + xb; }

    Out guess(int b) const
    {
        const int xb = b % nx, c = b / nx % nc, k = b / nx / nc;
        const int x0 = xb * BX, nw = std::min(BX, w - x0), y0 = c * R, L = std::min(R, h - y0);
        const int nsl = std::min(Z, nchain - k * Z);
        Out o;
        for (int j = 0; j < nsl; j++) {
            const int z = zfirst + dir * (k * Z + j);
            std::vector<Row> rows(L, Row(nw));
            for (int q = 0; q < L; q++)
                for (int i = 0; i < nw; i++) rows[q][i] = Opt{true, a(x0 + i, y0 + q, z)};
            o.rows.push_back(rows);
            o.down.push_back(rows[L - 1]);
            o.right.emplace_back(2 * L, Opt{});
            o.left.emplace_back(2 * L, Opt{});
        }
        return o;
    }
    Out run(int b, const std::vector<Out>& in) const
    {
        const int xb = b % nx, c = b / nx % nc, k = b / nx / nc;
        const int x0 = xb * BX, nw = std::min(BX, w - x0), y0 = c * R, L = std::min(R, h - y0);
        const int nsl = std::min(Z, nchain - k * Z), dz = -dir * cw;
        Out o = guess(b);
        for (int j = 0; j < nsl; j++) {
            const int z = zfirst + dir * (k * Z + j);
            Row P(nw);   // the row before (nothing at the field's edge)
            if (c > 0) P = in[block(k, c - 1, xb)].down[j];
            for (int i = 0; i < 2 * L; i++) {
                const bool downw = i < L;
                const int q = downw ? i : 2 * L - 1 - i, y = y0 + q;
                if (i == L) {
                    P = Row(nw);
                    if (y0 + L < h) P = in[block(k, c + 1, xb)].rows[j][0];
                }
                Row C(nw);
                for (int x = 0; x < nw; x++) {
                    Cell v;
                    if (downw) {
                        v = a(x0 + x, y, z);
                        Opt before{};
                        if (d > 1) {
                            if (j > 0) before = o.rows[j - 1][q][x];
                            else if (k > 0) before = in[block(k - 1, c, xb)].rows.back()[q][x];
                            else before = Opt{true, a(x0 + x, y, z - dir)};
                        }
                        take(v, before, 0, 0, dz);
                    } else {
                        v = o.rows[j][q][x].c;
                    }
                    take(v, P[x], 0, downw ? -cw : cw, 0);
                    C[x] = Opt{true, v};
                }
                if (downw ? y > 0 : y < h - 1) {
                    Opt s = xb > 0 ? in[block(k, c, xb - 1)].right[j][i] : Opt{};
                    for (int x = 0; x < nw; x++) {
                        take(C[x].c, s, -cw, 0, 0);
                        s = C[x];
                    }
                    o.right[j][i] = s;
                    s = xb + 1 < nx ? in[block(k, c, xb + 1)].left[j][i] : Opt{};
                    for (int x = nw - 1; x >= 0; x--) {
                        take(C[x].c, s, cw, 0, 0);
                        s = C[x];
                    }
                    o.left[j][i] = s;
                }
                o.rows[j][q] = C;
                if (i == L - 1) o.down[j] = C;
                P = C;
            }
        }
        return o;
    }
    // rounds until nothing changes; the results go to A
    int iterate()
    {
        nc = (h + R - 1) / R;
        nx = (w + BX - 1) / BX;
        nk = (nchain + Z - 1) / Z;
        const int n = nk * nc * nx;
        cur.clear();
        for (int b = 0; b < n; b++) cur.push_back(guess(b));
        std::vector<char> dirty(n, 1);
        int round = 0;
        for (;; round++) {
            std::vector<char> next(n, 0);
            std::vector<Out> out(n);
            std::vector<int> ran;
            for (int b = 0; b < n; b++)
                if (dirty[b]) {
                    out[b] = run(b, cur);
                    ran.push_back(b);
                }
            bool any = false;
            for (int b : ran) {
                const int xb = b % nx, c = b / nx % nc, k = b / nx / nc;
                const Out &o = out[b], &p = cur[b];
                auto mark = [&](int m) {
                    next[m] = 1;
                    any = true;
                };
                auto differ = [](const Row& r, const Row& s) {
                    for (size_t i = 0; i < r.size(); i++)
                        if (r[i] != s[i]) return true;
                    return false;
                };
                for (size_t j = 0; j < o.rows.size(); j++) {
                    if (c + 1 < nc && differ(o.down[j], p.down[j])) mark(block(k, c + 1, xb));
                    if (c > 0 && differ(o.rows[j][0], p.rows[j][0])) mark(block(k, c - 1, xb));
                    if (j + 1 == o.rows.size() && k + 1 < nk)
                        for (size_t q = 0; q < o.rows[j].size(); q++)
                            if (differ(o.rows[j][q], p.rows[j][q])) mark(block(k + 1, c, xb));
                    if (xb + 1 < nx && differ(o.right[j], p.right[j])) mark(b + 1);
                    if (xb > 0 && differ(o.left[j], p.left[j])) mark(b - 1);
                }
            }
            for (int b : ran) cur[b] = out[b];
            if (!any) break;
            dirty = next;
        }
        for (int b = 0; b < n; b++) {
            const int xb = b % nx, c = b / nx % nc, k = b / nx / nc;
            for (size_t j = 0; j < cur[b].rows.size(); j++) {
                const int z = zfirst + dir * (k * Z + (int)j);
                for (size_t q = 0; q < cur[b].rows[j].size(); q++)
                    for (size_t i = 0; i < cur[b].rows[j][q].size(); i++)
                        A[((size_t)z * h + c * R + q) * w + xb * BX + i] = cur[b].rows[j][q][i].c;
            }
        }
        return round + 1;
    }
};

}  // namespace

// Danielsson of a field (int16 deltas, 2 or 3 per cell) by the model, in place.
// *limit: the least of the phases' limits less their rounds; returns the most
// rounds of a phase.
extern "C" int dan_rounds_model(int dim, int w, int h, int d, int cw, int R, int Z, int BX, int16_t* cells, long long* limit,
                                int* blocks)
{
    Model m{};
    m.w = w; m.h = h; m.d = dim == 3 ? d : 1; m.cw = cw; m.R = R; m.BX = BX;
    m.A.resize((size_t)w * h * m.d);
    for (size_t i = 0; i < m.A.size(); i++)
        m.A[i] = Cell{cells[dim * i], cells[dim * i + 1], dim == 3 ? cells[dim * i + 2] : (int16_t)0};
    int most = 0;
    *limit = 1LL << 40;
    for (int pass = 0; pass < (dim == 3 ? 2 : 1); pass++) {
        m.dir = pass ? -1 : 1;
        m.nchain = dim == 3 ? d - 1 : 1;
        m.zfirst = dim == 3 ? (pass ? d - 2 : 1) : 0;
        m.Z = std::min(Z, m.nchain);
        const int r = m.iterate();
        *blocks = m.nk * m.nc * m.nx;
        most = std::max(most, r);
        *limit = std::min(*limit, (long long)dolk::dan_max_rounds(m.nchain, h, m.nx) - r);
    }
    for (size_t i = 0; i < m.A.size(); i++) {
        cells[dim * i] = m.A[i].x;
        cells[dim * i + 1] = m.A[i].y;
        if (dim == 3) cells[dim * i + 2] = m.A[i].z;
    }
    return most;
}

extern "C" int dan_rounds_limit(long long nchain, long long h, long long nx) { return dolk::dan_max_rounds(nchain, h, nx); }
