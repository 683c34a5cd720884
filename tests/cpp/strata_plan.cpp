// Host check of the dense-phase solve plan (csrc/arap_strata.h): on a mesh's
// constrained Laplacian with random weights, the plan's groups, tiles, update
// lists and inversion items give the solution of L L^T x = b. The products run
// tile by tile with the kernels' index arithmetic; every access is checked
// against its array.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "arap_strata.h"
#include "arap_symbolic.h"

using namespace arapgpu;

#define REQUIRE(c)                                            \
    do {                                                      \
        if (!(c)) {                                           \
            std::printf("FAILED %s line %d\n", #c, __LINE__); \
            return 1;                                         \
        }                                                     \
    } while (0)

static void grid(int nx, int ny, int off, std::vector<int32_t> &f) {
    for (int i = 0; i + 1 < nx; ++i)
        for (int j = 0; j + 1 < ny; ++j) {
            const int a = off + i * ny + j, b = a + ny, c = b + 1, d = a + 1;
            f.insert(f.end(), {a, b, c, a, c, d});
        }
}

static int check(int nx, int ny, int copies, StrataKind kind, int sms) {
    const bool fp64 = kind == kStFp64, poses = kind == kStPoses;
    std::vector<int32_t> faces;
    for (int c = 0; c < copies; ++c) grid(nx, ny, c * nx * ny, faces);
    const int V = copies * nx * ny;
    Topology topo;
    std::string err;
    REQUIRE(build_topology(V, (int)faces.size() / 3, faces.data(), topo, err));
    std::vector<uint8_t> fixed(V, 0);
    for (int c = 0; c < copies; ++c) fixed[c * nx * ny] = fixed[c * nx * ny + 1] = 1;
    Symbolic s;
    bool singular;
    REQUIRE(build_symbolic(topo, fixed, s, err, singular));
    Strata p;
    REQUIRE(build_strata(s, kind, sms, p));
    const int m = s.m;
    // the matrix in elimination order, its dense Cholesky factor
    std::mt19937 rng(7);
    std::uniform_real_distribution<double> u(0.5, 1.5);
    std::vector<double> L((size_t)m * m, 0.0);
    for (int k = 0; k < m; ++k)
        for (int e = s.drow[k]; e < s.drow[k + 1]; ++e) {
            const int l = s.dcol[e];
            if (l == k) continue;
            if (l >= m) L[(size_t)k * m + k] += 1.0;
            else if (l > k) {
                const double w = u(rng);
                L[(size_t)l * m + k] = -w;
                L[(size_t)k * m + k] += w;
                L[(size_t)l * m + l] += w;
            }
        }
    const std::vector<double> A = L;
    for (int k = 0; k < m; ++k) {
        const double d = std::sqrt(L[(size_t)k * m + k]);
        REQUIRE(d > 0);
        std::vector<int> nz;
        for (int i = k; i < m; ++i)
            if (i == k) L[(size_t)k * m + k] = d;
            else if (L[(size_t)i * m + k] != 0) {
                L[(size_t)i * m + k] /= d;
                nz.push_back(i);
            }
        for (size_t a = 0; a < nz.size(); ++a)
            for (size_t b = 0; b <= a; ++b)
                L[(size_t)nz[a] * m + nz[b]] -= L[(size_t)nz[a] * m + k] * L[(size_t)nz[b] * m + k];
    }
    // the inversion's items cover every column once, phase by phase
    std::vector<double> M(p.m_size, 0.0);
    std::vector<int> seen(m, 0);
    int items = 0;
    for (const StPhase &ph : p.ph) {
        REQUIRE(ph.i0 == items);
        items += ph.in;
        for (int q = ph.i0; q < ph.i0 + ph.in; ++q) {
            const int j = p.items[2 * q], c0 = p.items[2 * q + 1];
            const SnInfo &d = s.sn[j];
            REQUIRE(d.nrow <= ph.front && c0 % ph.rc == 0 && c0 < d.ncol);
            REQUIRE(ph.rc == 8 || ph.rc == 4 || ph.rc == 2);
            for (int c = c0; c < std::min(c0 + ph.rc, (int)d.ncol); ++c) {
                ++seen[d.first + c];
                // column of M: forward substitution along j's ancestors in the group
                const StSn &g = p.sn[j];
                std::vector<double> e(m, 0.0);
                e[d.first + c] = 1.0;
                int node = j;
                for (;;) {
                    const SnInfo &x = s.sn[node];
                    REQUIRE(p.sn[node].m_off == g.m_off && p.sn[node].ld == g.ld && p.sn[node].n == g.n);
                    for (int k = 0; k < x.ncol; ++k) {
                        const int col = x.first + k;
                        e[col] /= L[(size_t)col * m + col];
                        const int64_t at = g.m_off + (int64_t)(p.sn[node].pos + k) * g.ld + g.pos + c;
                        REQUIRE(at >= 0 && at < p.m_size);
                        if (e[col] != 0.0) M[at] = e[col];
                        for (int i = col + 1; i < m; ++i) e[i] -= L[(size_t)i * m + col] * e[col];
                    }
                    if (p.sn[node].root) {
                        for (int i = 0; i < x.nrow - x.ncol; ++i)
                            M[g.m_off + (int64_t)(g.n + i) * g.ld + g.pos + c] = e[s.rows[x.rows_off + i]];
                        break;
                    }
                    node = x.parent;
                    REQUIRE(node >= 0);
                }
            }
        }
    }
    REQUIRE((int)p.items.size() == 2 * items);
    for (int k = 0; k < m; ++k) REQUIRE(seen[k] == 1);
    std::vector<double> b(m), sol, y(m, 0.0), uv(s.uvec_size, 0.0), x(m);
    for (double &v : b) v = u(rng) - 1.0;
    sol = b;
    std::vector<int> wrote(m, 0), uwrote(s.uvec_size, 0);
    const int np = (int)p.ph.size();
    auto gathered = [&](int c) {
        double v = sol[p.col[c]];
        for (int q = 4 * p.gptr[c]; q < 4 * p.gptr[c + 1]; ++q)
            if (p.gidx[q] >= 0) v += uv[p.gidx[q]];
        return v;
    };
    for (int k = 0; k < np; ++k) {
        const StPhase &ph = p.ph[k];
        if (k == 0)
            for (int c = ph.c0; c < ph.c0 + ph.cn; ++c) REQUIRE(p.gptr[c] == p.gptr[c + 1]);
        for (int c = ph.c0; c < ph.c0 + ph.cn; ++c)
            for (int q = p.gptr[c]; q < p.gptr[c + 1]; ++q) REQUIRE(p.gidx[4 * q] >= 0);
        if (ph.big) {
            REQUIRE(k == np - 1 && p.big_n == ph.cn && ph.c0 == p.big_col && p.big_n <= kStMaxCols);
            for (int r = 0; r < p.big_n; ++r) {
                double v = 0;
                for (int c = 0; c <= r; ++c) {
                    double f = sol[p.col[p.big_col + c]];
                    for (int q = p.top_gptr[c]; q < p.top_gptr[c + 1]; ++q) f += uv[p.top_gidx[q]];
                    v += M[p.big_off + (int64_t)r * ((p.big_n + 3) & ~3) + c] * f;
                }
                y[p.col[p.big_col + r]] = v;
                ++wrote[p.col[p.big_col + r]];
            }
            continue;
        }
        if (poses) REQUIRE(!ph.big && ph.TC == 32);
        if (!poses) REQUIRE(ph.G == 8 || ph.G == 32 || (fp64 && (ph.G == 1 || ph.G == 4)));
        if (fp64) REQUIRE(ph.RW == 1);
        if (!poses) REQUIRE(ph.RW == 1 || ph.RW == 2 || ph.RW == 4);
        for (int t = ph.f0; t < ph.f0 + ph.fn; ++t) {
            const StTile &d = p.tiles[t];
            REQUIRE(d.count > 0 && d.first >= 0 && d.first + d.count <= d.n + d.r && d.ld == ((d.n + 3) & ~3));
            if (poses) REQUIRE(d.count <= 32);
            REQUIRE(d.n <= ph.nmax && d.n + d.r <= ph.vmax && d.m_off % 4 == 0);
            REQUIRE(d.m_off + (int64_t)(d.n + d.r) * d.ld <= p.m_size);
            for (int c = 0; c < d.n; ++c) REQUIRE(d.base < 0 || p.col[d.col_off + c] == d.base + c);
            const int ncol = d.first + d.count > d.n ? d.n : d.first + d.count;
            for (int r = d.first; r < d.first + d.count; ++r) {
                double v = 0;
                for (int c = 0; c < ncol; ++c) v += M[d.m_off + (int64_t)r * d.ld + c] * gathered(d.col_off + c);
                if (r < d.n) {
                    y[p.col[d.col_off + r]] = v;
                    ++wrote[p.col[d.col_off + r]];
                } else {
                    REQUIRE(d.u_off + r - d.n < s.uvec_size);
                    uv[d.u_off + r - d.n] = v;
                    ++uwrote[d.u_off + r - d.n];
                }
            }
        }
    }
    for (int k = 0; k < m; ++k) REQUIRE(wrote[k] == 1);
    size_t used = 0, sent = 0;
    for (int q : p.gidx) used += q >= 0;
    for (int w : uwrote) {
        REQUIRE(w <= 1);
        sent += w;
    }
    REQUIRE(used == sent);
    std::vector<int> solved(m, 0);
    for (int k = np - 1; k >= 0; --k) {
        const StPhase &ph = p.ph[k];
        if (ph.big) {
            for (int c = 0; c < p.big_n; ++c) {
                double v = 0;
                for (int r = c; r < p.big_n; ++r)
                    v += M[p.big_off + (int64_t)r * ((p.big_n + 3) & ~3) + c] * y[p.col[p.big_col + r]];
                x[p.col[p.big_col + c]] = v;
                ++solved[p.col[p.big_col + c]];
            }
            continue;
        }
        REQUIRE(ph.TC == 4 || ph.TC == 8 || ph.TC == 16 || ph.TC == 32 || ph.TC == 64);
        for (int t = ph.b0; t < ph.b0 + ph.bn; ++t) {
            const StTile &d = p.tiles[t];
            REQUIRE(d.count > 0 && d.count <= ph.TC && d.first % 4 == 0 && d.first + d.count <= d.n);
            for (int c = d.first; c < d.first + d.count; ++c) {
                double v = 0;
                for (int r = d.first; r < d.n + d.r; ++r) {
                    if (r >= d.n) REQUIRE(solved[s.rows[d.row_off + r - d.n]] == 1);
                    const double w = r < d.n ? y[p.col[d.col_off + r]] : x[s.rows[d.row_off + r - d.n]];
                    v += M[d.m_off + (int64_t)r * d.ld + c] * w;
                }
                x[p.col[d.col_off + c]] = v;
            }
        }
        for (int t = ph.b0; t < ph.b0 + ph.bn; ++t)
            for (int c = 0; c < p.tiles[t].count; ++c) ++solved[p.col[p.tiles[t].col_off + p.tiles[t].first + c]];
    }
    double worst = 0;
    for (int k = 0; k < m; ++k) {
        REQUIRE(solved[k] == 1);
        double r = b[k];
        for (int l = 0; l < m; ++l) r -= (l <= k ? A[(size_t)k * m + l] : A[(size_t)l * m + k]) * x[l];
        worst = std::max(worst, std::fabs(r));
    }
    std::printf("%dx%d x%d kind %d sms %d: m %d, %d phases, residual %.1e\n", nx, ny, copies, (int)kind, sms, m, np, worst);
    // x is O(m) at most here; 1e-16 x condition (about m) x sqrt(m) of rounding
    REQUIRE(worst < 1e-16 * (double)m * 64.0);
    return 0;
}

int main() {
    for (const StrataKind kind : {kStFp32, kStFp64, kStPoses}) {
        if (check(3, 2, 1, kind, 152)) return 1;     // four unknowns
        if (check(9, 8, 1, kind, 152)) return 1;     // one leaf
        if (check(23, 17, 2, kind, 152)) return 1;   // two components
        if (check(60, 33, 1, kind, 152)) return 1;
        if (check(47, 41, 1, kind, 4)) return 1;     // tiles of several row steps
    }
    std::printf("ok\n");
    return 0;
}
