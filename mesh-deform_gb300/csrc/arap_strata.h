// arap_strata.h -- the triangular solves of a request or of a pose batch in a few
// dense phases.
//
// The elimination tree is cut into strata of rooted subtrees ("groups"), each
// group's columns holding at most a few hundred to a few thousand columns.
// Per group the factorisation leaves one dense row-major matrix
//
//     M = [  X ]   X = inv(L_gg), n x n lower triangular
//         [ -W ]   W = L(rows below the group, group) X, r x n
//
// so a forward sweep is one product per stratum, [y; u] = M f (u goes to the
// columns above), and a backward sweep one transposed product,
// x = M^T [y; x_below]. No task waits for another inside a stratum; strata
// follow each other as launches. A sweep over a tree of 13 levels takes 3 to 7
// such phases instead of a chain of 13 dependent tasks.
#pragma once

#include <cstdint>
#include <vector>

namespace arapgpu {

struct Symbolic;

// One CTA's share of a phase: rows (forward) or columns (backward)
// [first, first + count) of a group's matrix. Everything a CTA needs comes
// with one 48-byte load.
struct StTile {
    int64_t m_off;    // the group's matrix, (n + r) rows of ld
    int32_t n, r, ld;
    int32_t first, count;
    int32_t col_off;  // the group's columns in the column list
    int32_t row_off;  // its rows below, in the symbolic row list
    int32_t u_off;    // its update vector
    int32_t base;     // its first column where its columns are consecutive, else -1
    int32_t pad;
};

// Per supernode: its group's matrix and its first column's place in it
struct StSn {
    int64_t m_off;
    int32_t ld, n, pos, root;  // root: 1 at the group's root
};

constexpr int kStMaxPhases = 16;
constexpr int kStMaxCols = 4096;   // most columns of a group
constexpr int kStThreads = 128;     // CTAs of the phases' kernels,
constexpr int kStThreadsLarge = 512;  // where groups are large,
constexpr int kStThreadsSmall = 64;   // and of the FP64 forward product where they are not
constexpr int kStBigTop = 1024;    // a lone last group with more columns runs the tiled top products
constexpr int kStLargeCols = 256, kStLargeRows = 400;  // columns / rows from which a group is large
constexpr int kStInvCols = 8;      // most columns of M one CTA of the inversion forms (8, 4 or 2)

struct StPhase {
    int32_t f0, fn, b0, bn;   // tiles of the forward / backward product
    int32_t G, RW, TC;        // lanes per row group, rows per group; columns per backward tile
    int32_t ntf, ntb;         // threads per CTA of the forward / backward product
    int32_t c0, cn;           // its columns in the column list
    int32_t nmax, vmax;       // largest n and n + r
    int32_t i0, in;           // its work items of the inversion
    int32_t front, rc;        // its largest front, columns of M per item
    int32_t big;              // the tiled top products run this phase
};

struct Strata {
    bool ok = false;
    std::vector<StPhase> ph;
    std::vector<StTile> tiles;
    std::vector<StSn> sn;
    std::vector<int32_t> col;    // columns (device indices) group by group
    std::vector<int32_t> gptr;   // per column-list entry: its update entries, in quads
    std::vector<int32_t> gidx;   // update-vector entries, padded with -1 to quads
    std::vector<int32_t> items;  // inversion: supernode, first column
    std::vector<int32_t> top_gptr;  // the big top's entries as the tiled products take them
    std::vector<int64_t> top_gidx;
    int64_t m_size = 0, big_off = 0;
    int32_t big_n = 0, big_col = 0;
    double entries = 0.0, nb_sum = 0.0;  // matrix entries of one sweep, update rows
};

// What the phases solve: one request in FP32 or FP64, or many poses in FP32
// (a plan that does not depend on how many: a pose's result is the same in
// any batch).
enum StrataKind { kStFp32 = 0, kStFp64 = 1, kStPoses = 2 };

// Cuts the tree for a device with `sms` SMs; false (and out.ok false) when
// some front does not fit the phases' kernels.
bool build_strata(const Symbolic &sym, StrataKind kind, int sms, Strata &out);

}  // namespace arapgpu
