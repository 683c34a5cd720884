// Launch shapes of the dense-phase plan (csrc/arap_strata.h) on the host: every
// phase's (threads, lanes, rows) and column tile is one that the kernels'
// dispatch (StKernels in csrc/arap_kernels.cu) has an instance of, for sheets of
// any size and for a mesh of random triangles, whose separators are so wide that
// FP64 plans end in a lone group of more than kStBigTop columns too.
#include <algorithm>
#include <cstdio>
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

static bool one_of(int x, std::initializer_list<int> set) { return std::find(set.begin(), set.end(), x) != set.end(); }

static int check(int V, const std::vector<int32_t> &faces, bool fp64_big) {
    Topology topo;
    std::string err;
    REQUIRE(build_topology(V, (int)faces.size() / 3, faces.data(), topo, err));
    std::vector<uint8_t> fixed(V, 0);
    for (int k = 0; k < 5; ++k) fixed[k] = 1;
    Symbolic s;
    bool singular;
    REQUIRE(build_symbolic(topo, fixed, s, err, singular));
    for (const StrataKind kind : {kStFp32, kStFp64, kStPoses}) {
        Strata p;
        REQUIRE(build_strata(s, kind, 152, p));
        bool big = false;
        for (const StPhase &q : p.ph) {
            REQUIRE(one_of(q.rc, {2, 4, 8}));
            if (q.big) {
                REQUIRE(kind != kStPoses && &q == &p.ph.back() && q.nmax > kStBigTop);
                big = true;
                continue;
            }
            if (kind == kStPoses) continue;  // one shape (k_bstrata)
            REQUIRE(one_of(q.ntb, {kStThreads, kStThreadsLarge}));
            if (kind == kStFp64) {
                REQUIRE((q.ntf == kStThreadsSmall && q.G == 8 && q.RW == 1) ||
                        (q.ntf == kStThreadsLarge && q.G == 32 && q.RW == 1));
                REQUIRE(one_of(q.TC, {4, 8, 16, 32}));
            } else {
                REQUIRE(one_of(q.ntf, {kStThreads, kStThreadsLarge}) && one_of(q.G, {8, 32}) && one_of(q.RW, {1, 2, 4}));
                REQUIRE(one_of(q.TC, {8, 16, 32, 64}));
            }
        }
        if (kind == kStFp64) REQUIRE(big == fp64_big);
    }
    return 0;
}

int main() {
    for (const int n : {4, 9, 17, 33, 70, 140, 260}) {
        std::vector<int32_t> f;
        for (int i = 0; i + 1 < n; ++i)
            for (int j = 0; j + 1 < n; ++j) {
                const int a = i * n + j, b = a + n, c = b + 1, d = a + 1;
                f.insert(f.end(), {a, b, c, a, c, d});
            }
        if (check(n * n, f, false)) return 1;
    }
    std::mt19937 rng(11);
    const int V = 3400;
    std::vector<int32_t> f;
    while ((int)f.size() < 9 * V) {
        const int32_t a = rng() % V, b = rng() % V, c = rng() % V;
        if (a != b && b != c && a != c) f.insert(f.end(), {a, b, c});
    }
    if (check(V, f, true)) return 1;
    std::printf("ok\n");
    return 0;
}
