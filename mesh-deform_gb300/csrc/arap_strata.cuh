// arap_strata.cuh -- kernels of the dense-phase triangular solves
// (arap_strata.h): forward and backward products of one stratum's groups, the
// gather of a stratum's right-hand sides, and the groups' matrices from the
// factor. Included by arap_kernels.cu.

// 16 bytes of T
template <typename T> struct StPack;
template <> struct StPack<float> {
    static constexpr int E = 4;
    float v[4];
    __device__ __forceinline__ void load(const float *p) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
    __device__ __forceinline__ void lds(const float *p) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
};
template <> struct StPack<double> {
    static constexpr int E = 2;
    double v[2];
    __device__ __forceinline__ void load(const double *p) {
        const double2 q = __ldg(reinterpret_cast<const double2 *>(p));
        v[0] = q.x; v[1] = q.y;
    }
    __device__ __forceinline__ void lds(const double *p) {
        const double2 q = *reinterpret_cast<const double2 *>(p);
        v[0] = q.x; v[1] = q.y;
    }
};

__device__ __forceinline__ StTile st_tile(const StTile *p) {
    const int4 *q = reinterpret_cast<const int4 *>(p);
    const int4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    StTile t;
    t.m_off = (int64_t)(unsigned)a.x | ((int64_t)a.y << 32);
    t.n = a.z; t.r = a.w;
    t.ld = b.x; t.first = b.y; t.count = b.z; t.col_off = b.w;
    t.row_off = c.x; t.u_off = c.y;
    t.base = c.z;
    t.pad = 0;
    return t;
}

// b[k] += the update entries of column k, for a stratum's columns, as a launch
// of its own: four threads per column, each an index quad at a time (its
// entries' loads in flight together), so that no thread runs a long chain of
// additions. 2.8 us on the bar's second stratum (10,538 columns); gathered
// inside the forward product instead, once per row tile, that product took
// 10.3 us against 7 (and in FP64 60% of its additions).
template <typename T>
__global__ void __launch_bounds__(kStThreads)
k_strata_gather(int c0, int cn, const int32_t *__restrict__ gcol, const int32_t *__restrict__ gptr,
                const int32_t *__restrict__ gidx, const Vec4<T> *uvec, Vec4<T> *b) {
    pdl_trigger();
    const int c = (blockIdx.x * kStThreads + threadIdx.x) >> 2, j = threadIdx.x & 3;
    int q0 = 0, q1 = 0, k = 0;
    int4 id{-1, -1, -1, -1};
    const int4 *gq = reinterpret_cast<const int4 *>(gidx);
    if (c < cn) {
        k = gcol[c0 + c];
        q0 = gptr[c0 + c] + j;
        q1 = gptr[c0 + c + 1];
        if (q0 < q1) id = __ldg(gq + q0);
    }
    pdl_wait();
    const Vec4<T> zero{(T)0, (T)0, (T)0, (T)0};
    Vec4<T> v = (j == 0 && c < cn) ? ldcg4(b + k) : zero;
    for (int q = q0; q < q1; q += 4) {
        if (q > q0) id = __ldg(gq + q);
        const Vec4<T> u0 = ldcg4(uvec + id.x);
        const Vec4<T> u1 = id.y >= 0 ? ldcg4(uvec + id.y) : zero;
        const Vec4<T> u2 = id.z >= 0 ? ldcg4(uvec + id.z) : zero;
        const Vec4<T> u3 = id.w >= 0 ? ldcg4(uvec + id.w) : zero;
        v.x += (u0.x + u1.x) + (u2.x + u3.x);
        v.y += (u0.y + u1.y) + (u2.y + u3.y);
        v.z += (u0.z + u1.z) + (u2.z + u3.z);
    }
#pragma unroll
    for (int off = 1; off <= 2; off <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
        v.z += __shfl_xor_sync(0xffffffffu, v.z, off);
    }
    if (j == 0 && c < cn) b[k] = v;
}

// Forward product of a stratum: M f for the rows of a tile, X's rows into y
// and -W's into the update vectors. A group of G lanes takes RW
// rows at a time, each lane 16 bytes of every row per step (consecutive lanes
// consecutive columns), with f as three arrays in shared memory so that a
// lane's four (two) columns come with one 16-byte load per component. A CTA's
// first loads of M (which only the factorisation writes) are issued before it
// waits for the kernel before it.
// FP32: bound by the launch's latency chain (tile, vector, product, store),
// not by L2: the bar's first stratum, 12 MB in 6.7 us. Four loads in flight
// per lane and 1,024 threads per SM beat eight and 512 (bar 164 -> 145 us per
// iteration). FP64: bound by FP64 issue (about 64 clocks per warp instruction
// and scheduler): tiles of 8 rows, so that the schedulers' shares even out.
template <typename T, int NT, int G, int RW>
__global__ void __launch_bounds__(NT, 1024 / NT)
k_strata_fwd(int ldf, const StTile *__restrict__ tiles, const T *__restrict__ Mall,
             const int32_t *__restrict__ gcol, const Vec4<T> *__restrict__ b, Vec4<T> *__restrict__ y,
             Vec4<T> *__restrict__ uvec) {
    extern __shared__ __align__(128) unsigned char st_raw[];
    constexpr int E = StPack<T>::E;
    constexpr int NB = 4 / RW;  // steps of one batch of loads: four 16-byte loads in flight per lane
    constexpr int kRows = NT / G * RW;
    T *fx = reinterpret_cast<T *>(st_raw), *fy = fx + ldf, *fz = fy + ldf;
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, l = tid % G, grp = tid / G;
    const StTile d = st_tile(tiles + blockIdx.x);
    const T *M = Mall + d.m_off;
    const int rend = d.first + d.count;
    // X is lower triangular: a warp's columns end at its last row's
    auto cols_to = [&](int last) {
        const int nc = last > d.n ? d.n : last;
        return (nc + G * E - 1) / (G * E) * (G * E);
    };
    const int ncol = rend > d.n ? d.n : rend, fspan = cols_to(rend);
    int span = cols_to(min(rend, d.first + (grp | (32 / G - 1)) * RW + RW));
    // column c of the group: consecutive ones in the first phase (whole subtrees)
    auto column = [&](int c) { return d.base >= 0 ? d.base + c : gcol[d.col_off + c]; };
    StPack<T> m[NB][RW];
    auto load = [&](int row, int c) {
#pragma unroll
        for (int k = 0; k < NB; ++k)
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const int cc = c + k * G * E;
                if (cc < d.ld && cc < span && row + i < rend) m[k][i].load(M + (int64_t)(row + i) * d.ld + cc);
                else
#pragma unroll
                    for (int e = 0; e < E; ++e) m[k][i].v[e] = (T)0;
            }
    };
    int row = d.first + grp * RW;
    load(row, l * E);
    // the places of f before the wait, f after it
    constexpr int kPre = 2;
    int at[kPre];
#pragma unroll
    for (int i = 0; i < kPre; ++i) at[i] = tid + i * NT < ncol ? column(tid + i * NT) : -1;
    pdl_wait();
    auto put = [&](int c, int k) {
        const Vec4<T> v = k >= 0 ? ldcg4(b + k) : Vec4<T>{(T)0, (T)0, (T)0, (T)0};
        fx[c] = v.x;
        fy[c] = v.y;
        fz[c] = v.z;
    };
#pragma unroll
    for (int i = 0; i < kPre; ++i)
        if (tid + i * NT < fspan) put(tid + i * NT, at[i]);
    for (int c = tid + kPre * NT; c < fspan; c += NT) put(c, c < ncol ? column(c) : -1);
    __syncthreads();
    for (int r0 = d.first; r0 < rend; r0 += kRows) {
        row = r0 + grp * RW;
        span = cols_to(min(rend, r0 + (grp | (32 / G - 1)) * RW + RW));
        constexpr int H = st_held<RW * 4, G>();
        // the value(s) this lane will hold after the reduction go to one row
        const int orow = row + (st_base<RW * 4, G>(lane) >> 2);
        const int ocol = orow < rend && orow < d.n ? column(orow) : 0;
        T acc[RW * 4];
#pragma unroll
        for (int i = 0; i < RW * 4; ++i) acc[i] = (T)0;
        for (int c = l * E; c < span; c += NB * G * E) {
            if (r0 > d.first || c >= NB * G * E) load(row, c);
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const int cc = c + k * G * E;
                if (cc >= span) break;
                StPack<T> px, py, pz;
                px.lds(fx + cc);
                py.lds(fy + cc);
                pz.lds(fz + cc);
#pragma unroll
                for (int i = 0; i < RW; ++i)
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        acc[4 * i] += m[k][i].v[e] * px.v[e];
                        acc[4 * i + 1] += m[k][i].v[e] * py.v[e];
                        acc[4 * i + 2] += m[k][i].v[e] * pz.v[e];
                    }
            }
        }
        const bool dup = st_reduce<RW * 4, G>(acc, lane);
        const int base = st_base<RW * 4, G>(lane);
        if (!dup && orow < rend) {
            T *dst = reinterpret_cast<T *>(orow < d.n ? y + ocol : uvec + d.u_off + (orow - d.n));
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const int comp = (base + j) & 3;
                if (comp < 3) dst[comp] = acc[j];
            }
        }
    }
}

// Backward product of a stratum: x = M^T v for TC columns of a group, v = y on
// its own rows and x on the rows below it (solved by the launches before).
// 16 bytes of a row per thread, TC / E threads per row, the rows dealt to the
// thread groups in turn; their sums meet in shared memory in a fixed order.
// Bound as the forward product; 64 columns per tile where that leaves two
// CTAs per SM (16 bars 318 -> 305 us per iteration against 32), fewer for
// small strata.
// x goes to the solution and the positions (mode 0: pc64 = x, 1: pc64 += x).
template <typename T, int NT, int TC>
__global__ void __launch_bounds__(NT, 1024 / NT)
k_strata_bwd(int vmax, const StTile *__restrict__ tiles, const T *__restrict__ Mall,
             const int32_t *__restrict__ gcol, const int32_t *__restrict__ rows, const Vec4<T> *__restrict__ y,
             Vec4<T> *sol, Vec4<double> *__restrict__ pc64, int mode) {
    extern __shared__ __align__(128) unsigned char st_raw[];
    constexpr int E = StPack<T>::E, QC = TC / E, NS = NT / QC, U = 8;
    Vec4<T> *v = reinterpret_cast<Vec4<T> *>(st_raw);
    T *red = reinterpret_cast<T *>(v + vmax);  // NS x (TC columns x 4)
    pdl_trigger();
    const int tid = threadIdx.x, q = tid % QC, s = tid / QC;
    const StTile d = st_tile(tiles + blockIdx.x);
    const T *M = Mall + d.m_off + (int64_t)d.first * d.ld + d.first + q * E;
    const int nrow = d.n + d.r - d.first;  // X is lower triangular: rows from the tile's first column on
    const bool in = d.first + q * E < d.ld;
    StPack<T> m[U];
    auto load = [&](int r) {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            if (in && r + i * NS < nrow) m[i].load(M + (int64_t)(r + i * NS) * d.ld);
            else
#pragma unroll
                for (int e = 0; e < E; ++e) m[i].v[e] = (T)0;
        }
    };
    load(s);
    // the vector's places before the wait, the vector after it
    auto column = [&](int c) { return d.base >= 0 ? d.base + c : gcol[d.col_off + c]; };
    constexpr int kPre = 4;
    int at[kPre];
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
        const int r = tid + i * NT, g = d.first + r;
        at[i] = r < nrow ? (g < d.n ? column(g) : rows[d.row_off + g - d.n]) : 0;
    }
    pdl_wait();
    // kSh threads per output value, each every kSh-th partial sum, kOut
    // values per thread; the outputs' places and positions are loaded
    // ahead of the product
    constexpr int kSh = 4 * TC < NT ? NT / (4 * TC) : 1;
    constexpr int kOut = 4 * TC > NT ? 4 * TC / NT : 1;
    const int h = tid % kSh;
    int ok[kOut];
    double before[kOut];
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
        const int o = tid / kSh + j * NT, oc = o >> 2, comp = o & 3;
        ok[j] = h == 0 && comp < 3 && oc < d.count ? column(d.first + oc) : -1;
        before[j] = ok[j] >= 0 && mode != 0 ? __ldcg(reinterpret_cast<const double *>(pc64 + ok[j]) + comp) : 0.0;
    }
    auto put = [&](int r, int k) {
        v[r] = ldcg4((d.first + r < d.n ? y : (const Vec4<T> *)sol) + k);
    };
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
        const int r = tid + i * NT;
        if (r < nrow) put(r, at[i]);
    }
    for (int r = tid + kPre * NT; r < nrow; r += NT) {
        const int g = d.first + r;
        put(r, g < d.n ? column(g) : rows[d.row_off + g - d.n]);
    }
    __syncthreads();
    T acc[E][3];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e][0] = acc[e][1] = acc[e][2] = (T)0;
    for (int r = s; r < nrow; r += U * NS) {
        if (r != s) load(r);
#pragma unroll
        for (int i = 0; i < U; ++i) {
            if (r + i * NS >= nrow) break;
            const Vec4<T> x = v[r + i * NS];
#pragma unroll
            for (int e = 0; e < E; ++e) {
                acc[e][0] += m[i].v[e] * x.x;
                acc[e][1] += m[i].v[e] * x.y;
                acc[e][2] += m[i].v[e] * x.z;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
        for (int c = 0; c < 3; ++c) red[(s * TC + q * E + e) * 4 + c] = acc[e][c];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
        const int o = tid / kSh + j * NT, comp = o & 3;
        T sum = (T)0;
#pragma unroll 8
        for (int i = h; i < NS; i += kSh) sum += red[i * TC * 4 + o];
#pragma unroll
        for (int off = 1; off < kSh; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (ok[j] >= 0) {
            reinterpret_cast<T *>(sol + ok[j])[comp] = sum;
            reinterpret_cast<double *>(pc64 + ok[j])[comp] = mode == 0 ? (double)sum : before[j] + (double)sum;
        }
    }
}

// RC columns [c0, c0 + RC) of supernode j's columns of its group's M: forward
// substitution L_gg Y = E (E the identity columns) along j's ancestors in the
// group, block column by block column of 32: Y_b = inv(L_bb) F_b with the
// factorisation's inverted diagonal blocks, then the rows below lose L Y_b;
// a supernode's rows below its columns go into its parent's front. The Y are
// X's rows; past the group's root, F is -W. Zeros of M (above the diagonal,
// and between subtrees that do not meet) are never written: they are cleared
// once when the matrices are laid out.
// The block that holds the columns starts from the identity: its Y are columns
// of inv(L_bb), and their rows above c0 are zero (half the FP64 work of groups
// with few columns: set-up of the bar in FP64 3.41 -> 2.83 ms).
// Bound by FP64 issue (FP64 form) or by the chain of blocks; a phase's columns
// per CTA are cut until it has four CTAs per SM. In FP32 more CTAs on an SM
// are worth more than loads ahead (bar's set-up 2.42 against 2.48 ms). The strata are independent:
// their launches overlap (`first` waits for the factor, the others only
// before they end).
template <typename T, int RC>
__global__ void __launch_bounds__(kStThreads, sizeof(T) == 8 ? 6 : 8)
k_strata_inverse(const int32_t *__restrict__ items, const SnInfo *__restrict__ sn, const StSn *__restrict__ ssn,
                 const int32_t *__restrict__ relind, const T *__restrict__ Lval, const T *__restrict__ Dinv,
                 int front, int first, T *__restrict__ Mall) {
    extern __shared__ __align__(128) unsigned char st_raw[];
    constexpr bool kAhead = sizeof(T) == 8;
    T *F = reinterpret_cast<T *>(st_raw);  // [row][RC], the current supernode's front
    T *G = F + (size_t)front * RC;         // its parent's
    T *Y = G + (size_t)front * RC;         // [row][RC], the current block's solution
    const int tid = threadIdx.x;
    const int j = items[2 * blockIdx.x], c0 = items[2 * blockIdx.x + 1];
    SnInfo dn = sn[j];
    const StSn gj = ssn[j];
    const int w = min(RC, dn.ncol - c0);
    T *M = Mall + gj.m_off + gj.pos + c0;  // the block's first column
    for (int q = tid; q < dn.nrow * RC; q += kStThreads) F[q] = q / RC == c0 + q % RC ? (T)1 : (T)0;
    if (first) pdl_wait();
    pdl_trigger();
    __syncthreads();
    int node = j, jb = c0 / NB;
    bool start = true;
    for (;;) {
        const int n = dn.nrow, nc = dn.ncol, pos = ssn[node].pos;
        const T *P = Lval + dn.panel_off;
        for (; jb * NB < nc; ++jb) {
            const int j0 = jb * NB, wb = min(NB, nc - j0);
            const int kb = start ? c0 - j0 : 0;  // the solution's rows above are zero
            const T *D = Dinv + dn.dinv_off + (int64_t)jb * NB * NB;  // D[k * NB + r] = inv(L_bb)(r, k)
            // FP64: the row of L below the block that this thread takes first is
            // loaded ahead of the block's solution
            T l[NB];
            auto load = [&](int i) {
                const T *Li = P + (int64_t)j0 * n + i;
#pragma unroll
                for (int k = 0; k < NB; ++k) l[k] = k >= kb && k < wb ? Li[(int64_t)k * n] : (T)0;
            };
            const int i0 = j0 + wb + tid;
            if (kAhead && i0 < n) load(i0);
            for (int o = tid; o < NB * RC; o += kStThreads) {
                const int r = o % NB, c = o / NB;
                T s = (T)0;
                if (start) {  // F is the identity's columns
                    if (c < w) s = D[(kb + c) * NB + r];
                } else {
                    T dk[NB];
#pragma unroll
                    for (int k = 0; k < NB; ++k) dk[k] = D[k * NB + r];
#pragma unroll
                    for (int k = 0; k < NB; ++k)
                        if (k < wb) s += dk[k] * F[(j0 + k) * RC + c];
                }
                Y[r * RC + c] = s;
                if (r < wb && c < w) M[(int64_t)(pos + j0 + r) * gj.ld + c] = s;
            }
            start = false;
            __syncthreads();
            for (int i = i0; i < n; i += kStThreads) {
                T acc[RC];
#pragma unroll
                for (int c = 0; c < RC; ++c) acc[c] = F[i * RC + c];
                if constexpr (kAhead) {
                    if (i != i0) load(i);
#pragma unroll
                    for (int k0 = 0; k0 < NB; k0 += 4) {
                        if (k0 + 4 <= kb || k0 >= wb) continue;
#pragma unroll
                        for (int k = k0; k < k0 + 4; ++k)
#pragma unroll
                            for (int c = 0; c < RC; ++c) acc[c] -= l[k] * Y[k * RC + c];
                    }
                } else {
                    const T *Li = P + (int64_t)j0 * n + i;
#pragma unroll 8
                    for (int k = kb; k < wb; ++k) {
                        const T lk = Li[(int64_t)k * n];
#pragma unroll
                        for (int c = 0; c < RC; ++c) acc[c] -= lk * Y[k * RC + c];
                    }
                }
#pragma unroll
                for (int c = 0; c < RC; ++c) F[i * RC + c] = acc[c];
            }
            __syncthreads();
        }
        const int nb = n - nc;
        if (ssn[node].root) {
            for (int q = tid; q < nb * RC; q += kStThreads)
                if (q % RC < w) M[(int64_t)(gj.n + q / RC) * gj.ld + q % RC] = F[nc * RC + q];
            break;
        }
        const int32_t *ri = relind + dn.relind_off;
        node = dn.parent;
        dn = sn[node];
        for (int q = tid; q < dn.nrow * RC; q += kStThreads) G[q] = (T)0;
        __syncthreads();
        for (int q = tid; q < nb * RC; q += kStThreads) G[ri[q / RC] * RC + q % RC] = F[nc * RC + q];
        __syncthreads();
        T *t = F;
        F = G;
        G = t;
        jb = 0;
    }
    if (!first) pdl_wait();
}
