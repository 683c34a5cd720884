// arap_strata.cpp -- cuts the elimination tree into the dense phases of the
// solves (arap_strata.h). Integer work on the host, O(S log m).
#include "arap_strata.h"

#include <algorithm>
#include <limits>

#include "arap_symbolic.h"

namespace arapgpu {

namespace {

// Cost of a sweep's phase in us: a latency per launch (measured 4 to 6 us a
// phase with overlapped launches) and per gather, the matrix entries at the
// rate that bounds them (FP32: bytes from L2; FP64: three FMAs per entry at
// about 0.55 T FMA/s), and the entries' formation spread over the sweeps of a
// deform. The minimum is flat in FP32: 3 us for 5, or 3 TB/s for 5, move the
// bar and the level-7 sphere by 2%; 10 us for 5 takes one phase less of the
// level-6 sphere, 113 -> 143 us per iteration. FP64: a tiled last phase with
// the FP32 constants 290 against 271 us (bar).
constexpr double kPhaseUs = 5.0, kBytesPerUs = 5e6, kFma64PerUs = 0.55e6, kFma32PerUs = 8e6;
constexpr double kGatherUs[2] = {1.0, 2.5}, kBigTopUs[2] = {0.0, 3.0};  // FP32, FP64
constexpr double kSweepsPerFactor[2] = {40.0, 20.0};
// many poses: FP32 FMAs at about half the peak, for 256 poses, and the chain of
// a CTA's chunks by the largest group (without it 16 poses 300 instead of 276
// us per iteration, 5 poses of 642 vertices 141 instead of 90)
constexpr double kPosesUs = 8.0, kPosesGatherUs = 4.0, kPoses = 256.0, kPosesFmaPerUs = 18e6, kPosesColUs = 0.05;

int ld_of(int n) { return (n + 3) & ~3; }

}  // namespace

bool build_strata(const Symbolic &sym, StrataKind kind, int sms, Strata &out) {
    out = Strata();
    const bool fp64 = kind == kStFp64, poses = kind == kStPoses;
    const int S = sym.S, m = sym.m;
    if (S == 0 || sym.uvec_size >= std::numeric_limits<int32_t>::max()) return false;
    const std::vector<SnInfo> &sn = sym.sn;
    // columns and factor entries of every supernode's subtree (children come first)
    std::vector<int32_t> full(S, 0);
    std::vector<double> fent(S, 0.0);
    int maxfull = 0;
    for (int s = 0; s < S; ++s) {
        const double nc = sn[s].ncol, nb = sn[s].nrow - sn[s].ncol;
        full[s] += sn[s].ncol;
        fent[s] += nc * nc / 2 + nc * nb;
        if (sn[s].parent >= 0) {
            full[sn[s].parent] += full[s];
            fent[sn[s].parent] += fent[s];
        }
        maxfull = std::max(maxfull, full[s]);
    }
    // candidate cuts: subtrees of at most thr[j] columns lie below cut j
    std::vector<int32_t> thr(1, 0);
    for (double t = 32; t < maxfull; t *= t < 512 ? 1.25 : 1.4) thr.push_back((int32_t)t);
    thr.push_back(maxfull);
    const int K = (int)thr.size();
    std::vector<std::vector<int32_t>> roots(K);  // maximal subtrees below cut j
    for (int j = 1; j < K; ++j)
        for (int s = 0; s < S; ++s)
            if (full[s] <= thr[j] && (sn[s].parent < 0 || full[sn[s].parent] > thr[j])) roots[j].push_back(s);
    const double inf = 1e30;
    const int vlim = fp64 ? 5600 : 11200;  // rows whose vector fits the backward product's shared memory
    std::vector<double> best(K, inf);
    std::vector<int> from(K, -1);
    best[0] = 0.0;
    std::vector<int32_t> dcol(S);
    std::vector<double> dent(S);
    for (int i = 0; i + 1 < K; ++i) {
        if (best[i] >= inf) continue;
        // columns / entries of every subtree that lie below cut i
        std::fill(dcol.begin(), dcol.end(), 0);
        std::fill(dent.begin(), dent.end(), 0.0);
        for (int s = 0; s < S; ++s) {
            if (full[s] <= thr[i]) {
                dcol[s] = full[s];
                dent[s] = fent[s];
            }
            if (sn[s].parent >= 0) {
                dcol[sn[s].parent] += dcol[s];
                dent[sn[s].parent] += dent[s];
            }
        }
        for (int j = i + 1; j < K; ++j) {
            double ent = 0.0, form = 0.0;
            int nmax = 0, cnt = 0;
            bool fits = true;
            for (const int32_t s : roots[j]) {
                const int n = full[s] - dcol[s], r = sn[s].nrow - sn[s].ncol;
                if (n == 0) continue;
                ent += 0.5 * n * (n + 1.0) + (double)n * r;
                form += 0.5 * n * (fent[s] - dent[s]);
                nmax = std::max(nmax, n);
                fits = fits && n <= kStMaxCols && n + r <= vlim;
                ++cnt;
            }
            if (!fits) continue;
            double c;
            if (poses) {
                c = kPosesUs + kPosesColUs * nmax + ent * 3 * kPoses / kPosesFmaPerUs + (i > 0 ? 0.5 * kPosesGatherUs : 0.0);
            } else {
                c = kPhaseUs + std::max(ent * (fp64 ? 8 : 4) / kBytesPerUs, fp64 ? ent * 3 / kFma64PerUs : 0.0) +
                    form / (fp64 ? kFma64PerUs : kFma32PerUs) / kSweepsPerFactor[fp64];
                if (j == K - 1 && cnt == 1 && nmax > kStBigTop) c += kBigTopUs[fp64];
                else if (i > 0) c += 0.5 * kGatherUs[fp64];  // forward sweeps only
            }
            if (best[i] + c < best[j]) {
                best[j] = best[i] + c;
                from[j] = i;
            }
        }
    }
    if (best[K - 1] >= inf) return false;
    std::vector<int> cuts;
    for (int j = K - 1; j > 0; j = from[j]) cuts.push_back(j);
    std::reverse(cuts.begin(), cuts.end());
    if ((int)cuts.size() > kStMaxPhases) return false;

    // groups: the root of every supernode's group, then columns, matrices and tiles phase by phase
    std::vector<int32_t> groot(S, -1), phase(S, -1), gcols(S, 0), gcol_off(S, 0);
    std::vector<int64_t> gm_off(S, 0);
    for (int s = 0; s < S; ++s) {
        int k = 0;
        while (full[s] > thr[cuts[k]]) ++k;
        phase[s] = k;
    }
    for (int s = S - 1; s >= 0; --s) {  // parents first
        const int p = sn[s].parent;
        groot[s] = (p >= 0 && phase[p] == phase[s]) ? groot[p] : s;
    }
    out.sn.assign(S, StSn());
    for (int s = 0; s < S; ++s) {
        StSn &x = out.sn[s];
        x.pos = gcols[groot[s]];
        x.root = groot[s] == s;
        gcols[groot[s]] += sn[s].ncol;
    }
    const int np = (int)cuts.size();
    std::vector<std::vector<int32_t>> groups(np);
    for (int s = 0; s < S; ++s)
        if (groot[s] == s) groups[phase[s]].push_back(s);
    out.col.assign(m, -1);
    std::vector<int32_t> colpos(m, -1);  // column -> place in the column list
    int32_t coff = 0;
    int64_t moff = 0;
    for (int k = 0; k < np; ++k) {
        StPhase p{};
        p.c0 = coff;
        for (const int32_t g : groups[k]) {
            gcol_off[g] = coff;
            gm_off[g] = moff;
            const int n = gcols[g], r = sn[g].nrow - sn[g].ncol;
            moff += (int64_t)(n + r) * ld_of(n);
            coff += n;
            p.nmax = std::max(p.nmax, n);
            p.vmax = std::max(p.vmax, n + r);
            out.entries += 0.5 * n * (n + 1.0) + (double)n * r;
            out.nb_sum += r;
        }
        p.cn = coff - p.c0;
        p.big = !poses && k == np - 1 && groups[k].size() == 1 && p.nmax > kStBigTop;
        out.ph.push_back(p);
    }
    if (moff >= (int64_t)1 << 40) return false;
    out.m_size = moff + 256;
    for (int s = 0; s < S; ++s) {
        const int g = groot[s];
        StSn &x = out.sn[s];
        x.m_off = gm_off[g];
        x.n = gcols[g];
        x.ld = ld_of(x.n);
        for (int c = 0; c < sn[s].ncol; ++c) {
            out.col[gcol_off[g] + x.pos + c] = sn[s].first + c;
            colpos[sn[s].first + c] = gcol_off[g] + x.pos + c;
        }
    }
    // update entries per column, each sent from its group straight to the
    // column (groups in phase and column order: a fixed order of the sums)
    std::vector<int32_t> cnt(m + 1, 0);
    auto each_entry = [&](auto &&f) {
        for (int k = 0; k < np; ++k)
            for (const int32_t g : groups[k]) {
                const int r = sn[g].nrow - sn[g].ncol;
                for (int i = 0; i < r; ++i) f(colpos[sym.rows[sn[g].rows_off + i]], (int32_t)(sn[g].uvec_off + i));
            }
    };
    each_entry([&](int c, int32_t) { ++cnt[c]; });
    out.gptr.assign(m + 1, 0);
    for (int c = 0; c < m; ++c) out.gptr[c + 1] = out.gptr[c] + (cnt[c] + 3) / 4;
    out.gidx.assign((size_t)std::max(out.gptr[m], 1) * 4, -1);
    {
        std::vector<int32_t> fill(m);
        for (int c = 0; c < m; ++c) fill[c] = 4 * out.gptr[c];
        each_entry([&](int c, int32_t u) { out.gidx[fill[c]++] = u; });
    }
    // tiles
    for (int k = 0; k < np; ++k) {
        StPhase &p = out.ph[k];
        // columns of M per work item: as many as leave four CTAs per SM and
        // fit shared memory (two fronts and a block of that many columns)
        p.rc = kStInvCols;
        for (int s = 0; s < S; ++s)
            if (phase[s] == k) p.front = std::max(p.front, (int32_t)sn[s].nrow);
        while (p.rc > 2 && (p.cn / p.rc < 4 * sms || (int64_t)(2 * p.front + kDiagBlock) * p.rc * (fp64 ? 8 : 4) > 200 * 1024))
            p.rc /= 2;
        p.i0 = (int32_t)out.items.size() / 2;
        for (int s = 0; s < S; ++s) {
            if (phase[s] != k) continue;
            for (int c0 = 0; c0 < sn[s].ncol; c0 += p.rc) {
                out.items.push_back(s);
                out.items.push_back(c0);
            }
        }
        p.in = (int32_t)out.items.size() / 2 - p.i0;
        if (p.big) {
            const int32_t g = groups[k][0];
            out.big_n = gcols[g];
            out.big_off = gm_off[g];
            out.big_col = gcol_off[g];
            out.top_gptr.assign(out.big_n + 1, 0);
            for (int c = 0; c < out.big_n; ++c) {
                for (int q = 4 * out.gptr[p.c0 + c]; q < 4 * out.gptr[p.c0 + c + 1]; ++q)
                    if (out.gidx[q] >= 0) out.top_gidx.push_back(out.gidx[q]);
                out.top_gptr[c + 1] = (int32_t)out.top_gidx.size();
            }
            if (out.top_gidx.empty()) out.top_gidx.push_back(0);
            continue;
        }
        int64_t rows = 0;
        for (const int32_t g : groups[k]) rows += gcols[g] + sn[g].nrow - sn[g].ncol;
        // 512 threads where groups are large: the vectors' loads and the rows
        // per thread, a CTA's serial part, are a quarter (level-7 sphere 277 ->
        // 235 us per iteration, FP64 sphere level 3 46 -> 37)
        p.ntf = p.nmax > kStLargeCols ? kStThreadsLarge : kStThreads;
        p.ntb = p.vmax > kStLargeRows ? kStThreadsLarge : kStThreads;
        auto step = [&](int rw) { return p.ntf / p.G * rw; };
        int per;
        if (fp64) {
            // Bound by FP64 issue, so the work has to come in shares small
            // enough to even out over the schedulers: 8 lanes per row and 8
            // rows per CTA of 64 threads (one row per lane of 128-thread CTAs
            // left one scheduler in four without rows: bar 259 -> 224 us per
            // iteration, level-6 sphere 200 -> 167, 2,562 vertices 41 -> 40;
            // with 4 or 2 lanes per row 229 and 232).
            p.RW = 1;
            p.G = 32;
            if (p.nmax <= kStLargeCols) {
                p.ntf = kStThreadsSmall;
                p.G = 8;
            }
            per = step(1);
        } else {
            // lane groups of 8 for groups of few columns; as many rows per
            // lane group as leave four warps per scheduler
            p.G = p.nmax <= 128 ? 8 : 32;
            p.RW = 4;
            while (p.RW > 1 && rows / (32 / p.G * p.RW) < 4 * 4 * sms) p.RW /= 2;
            per = step(p.RW) * (int)std::min<int64_t>(8, std::max<int64_t>(1, rows / ((int64_t)step(p.RW) * 4 * sms)));
        }
        p.TC = fp64 ? 32 : 64;
        while (p.TC > (fp64 ? 4 : 8) && (int64_t)p.cn / p.TC * p.ntb < (int64_t)(fp64 ? 4 : 2) * kStThreads * sms) p.TC /= 2;
        if (poses) per = p.TC = 32;
        auto tile = [&](int32_t g, int first, int count) {
            StTile t{};
            t.m_off = gm_off[g];
            t.n = gcols[g];
            t.r = sn[g].nrow - sn[g].ncol;
            t.ld = ld_of(t.n);
            t.first = first;
            t.count = count;
            t.col_off = gcol_off[g];
            t.row_off = sn[g].rows_off;
            t.u_off = (int32_t)sn[g].uvec_off;
            const int32_t c0 = out.col[t.col_off];  // columns of a group ascend
            t.base = out.col[t.col_off + t.n - 1] - c0 == t.n - 1 ? c0 : -1;
            out.tiles.push_back(t);
        };
        p.f0 = (int32_t)out.tiles.size();
        for (const int32_t g : groups[k]) {
            const int tot = gcols[g] + sn[g].nrow - sn[g].ncol;
            for (int r0 = 0; r0 < tot; r0 += per) tile(g, r0, std::min(per, tot - r0));
        }
        p.fn = (int32_t)out.tiles.size() - p.f0;
        p.b0 = (int32_t)out.tiles.size();
        for (const int32_t g : groups[k])
            for (int c0 = 0; c0 < gcols[g]; c0 += p.TC) tile(g, c0, std::min((int)p.TC, gcols[g] - c0));
        p.bn = (int32_t)out.tiles.size() - p.b0;
    }
    out.ok = true;
    return true;
}

}  // namespace arapgpu
