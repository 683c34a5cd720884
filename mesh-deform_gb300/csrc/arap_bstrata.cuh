// arap_bstrata.cuh -- the dense-phase triangular solves (arap_strata.h) for
// many poses: a stratum's product with all poses' right-hand sides, a matrix
// product [rows] x [K] x [poses x 3] per group in FP32. Included by
// arap_batch.cu.

constexpr int kBsThreads = 128, kBsK = 16;
constexpr int kBsRows = 32, kBsPoses = kStPoseTile, kBsRing = 4;  // tile, shared-memory buffers
// floats of a chunk of M in shared memory (forward rows padded to 20)
constexpr int bs_m_floats() { return kBsRows * (kBsK + 4); }

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

// b(k, p) += the update entries of column k, for a stratum's columns (as
// k_strata_gather); thread = (column, pose), so every load is coalesced over
// the poses.
__global__ void __launch_bounds__(256)
k_bstrata_gather(int c0, int cn, int P, const int32_t *__restrict__ gcol, const int32_t *__restrict__ gptr,
                 const int32_t *__restrict__ gidx, const Vec4<float> *uvec, Vec4<float> *b) {
    pdl_wait();
    pdl_trigger();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= (int64_t)cn * P) return;
    const int c = (int)(t / P), p = (int)(t % P);
    const int q0 = gptr[c0 + c], q1 = gptr[c0 + c + 1];
    if (q0 == q1) return;
    Vec4<float> *dst = b + (int64_t)gcol[c0 + c] * P + p;
    Vec4<float> v = ldcg4(dst);
    const Vec4<float> zero{0.f, 0.f, 0.f, 0.f};
    for (int q = q0; q < q1; ++q) {
        const int4 id = __ldg(reinterpret_cast<const int4 *>(gidx) + q);
        const Vec4<float> u0 = ldcg4(uvec + (int64_t)id.x * P + p);
        const Vec4<float> u1 = id.y >= 0 ? ldcg4(uvec + (int64_t)id.y * P + p) : zero;
        const Vec4<float> u2 = id.z >= 0 ? ldcg4(uvec + (int64_t)id.z * P + p) : zero;
        const Vec4<float> u3 = id.w >= 0 ? ldcg4(uvec + (int64_t)id.w * P + p) : zero;
        v.x += (u0.x + u1.x) + (u2.x + u3.x);
        v.y += (u0.y + u1.y) + (u2.y + u3.y);
        v.z += (u0.z + u1.z) + (u2.z + u3.z);
    }
    *dst = v;
}

// One 32 x 32 tile of a group's product: BWD false, rows [first, first +
// count) of M f, X's rows into `out` (y) and -W's into uvec; BWD true, columns
// of M^T v, v = y on the group's rows and x (`below`) on the rows below, into
// `out` (the solution; null where no stratum below reads it) and added to the
// positions. 128 threads as 8 row groups
// x 16 pose groups, each 4 rows x 2 poses (x, y, z of every pose in one
// 16-byte load); K in chunks of 16 through a ring of four shared-memory
// buffers filled by cp.async (two left a chunk waiting for its loads: 0.95 us
// per chunk). Every sum runs over K in order, so a pose's result does not
// depend on the batch. Bound by FP32 issue and shared-memory reads (24 FMAs
// for 3 16-byte loads a thread and column); tiles of 64 rows or poses, with
// fewer loads per FMA, need 130 to 250 registers and were slower (256 poses of
// the level-5 sphere: 106 / 137 us per sweep with 64 x 32, 111 / 162 with
// 64 x 64, 101 / 129 with this tile; the persistent supernodal sweeps with the
// tensor-core top before: 171 / 221).
template <bool BWD>
__global__ void __launch_bounds__(kBsThreads)
k_bstrata(int P, const StTile *__restrict__ tiles, const float *__restrict__ Mall, const int32_t *__restrict__ gcol,
          const int32_t *__restrict__ rows, const Vec4<float> *__restrict__ own, const Vec4<float> *below,
          Vec4<float> *out, Vec4<float> *__restrict__ uvec, Vec4<double> *__restrict__ pc64) {
    constexpr int TR = kBsRows, TP = kBsPoses, NS = kBsRing, KC = kBsK, RT = TR / 8, PT = TP / 16;
    constexpr int NF = KC * TP / kBsThreads, NM = KC * TR / 4 / kBsThreads;
    constexpr int LDM = BWD ? TR : KC + 4;       // forward: M's rows, backward: M's columns
    constexpr int MS = bs_m_floats();
    extern __shared__ __align__(128) unsigned char bs_raw[];
    Vec4<float> *Fs = reinterpret_cast<Vec4<float> *>(bs_raw);          // [NS][KC][TP]
    float *Ms = reinterpret_cast<float *>(Fs + NS * KC * TP);            // [NS][MS]
    int *idx = reinterpret_cast<int *>(Ms + NS * MS);                    // source row of every k (< 0: ~k of `below`)
    const StTile d = tiles[blockIdx.x];
    const float *M = Mall + d.m_off;
    const int tid = threadIdx.x, p0 = blockIdx.y * TP;
    const int rend = d.first + d.count;
    // forward: X is lower triangular, columns end at the tile's last row;
    // backward: rows start at the tile's first column
    const int K = BWD ? d.n + d.r - d.first : (rend > d.n ? d.n : rend);
    auto column = [&](int c) { return d.base >= 0 ? d.base + c : gcol[d.col_off + c]; };
    for (int k = tid; k < K; k += kBsThreads) {
        const int r = BWD ? d.first + k : k;
        idx[k] = r < d.n ? column(r) : ~rows[d.row_off + r - d.n];
    }
    pdl_wait();  // the vectors of the kernels before (an overlapped launch)
    pdl_trigger();
    __syncthreads();
    const int nk = (K + KC - 1) / KC;
    auto issue = [&](int c) {
        if (c < nk) {
            const int k0 = c * KC, buf = c % NS;
#pragma unroll
            for (int j = 0; j < NF; ++j) {
                const int e = tid + j * kBsThreads, k = e / TP, p = e % TP;
                const bool ok = k0 + k < K && p0 + p < P;
                const int s = ok ? idx[k0 + k] : 0;
                const Vec4<float> *src =
                    (!BWD || s >= 0 ? own + (int64_t)s * P : below + (int64_t)~s * P) + (ok ? p0 + p : 0);
                cp_async16(Fs + (buf * KC + k) * TP + p, src, ok);
            }
#pragma unroll
            for (int j = 0; j < NM; ++j) {
                const int e = tid + j * kBsThreads;
                if (BWD) {
                    const int cq = e % (TR / 4), k = e / (TR / 4);
                    const bool ok = k0 + k < K && d.first + 4 * cq < d.ld;
                    cp_async16(Ms + buf * MS + k * LDM + 4 * cq,
                               M + (ok ? (int64_t)(d.first + k0 + k) * d.ld + d.first + 4 * cq : 0), ok);
                } else {
                    const int kq = e % (KC / 4), row = e / (KC / 4);
                    const bool ok = row < d.count && k0 + 4 * kq < d.ld;
                    cp_async16(Ms + buf * MS + row * LDM + 4 * kq,
                               M + (ok ? (int64_t)(d.first + row) * d.ld + k0 + 4 * kq : 0), ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // forward: thread row i is rg + 8 i (two row groups of a warp then read
    // different banks), backward: column rg RT + i
    const int pg = tid & 15, rg = tid >> 4;
    auto row_of = [&](int i) { return BWD ? rg * RT + i : rg + 8 * i; };
    float acc[RT][PT][3];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < PT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = 0.f;
    for (int c = 0; c < NS - 1; ++c) issue(c);
    for (int c = 0; c < nk; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();  // chunk c is in place; the buffer issued next has no readers left
        issue(c + NS - 1);
        const Vec4<float> *F = Fs + (c % NS) * KC * TP + pg;
        const float *Mb = Ms + (c % NS) * MS;
#pragma unroll
        for (int k4 = 0; k4 < KC; k4 += 4) {
            float m[4][RT];
            if (BWD) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int i = 0; i < RT; i += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(Mb + (k4 + k) * LDM + rg * RT + i);
                        m[k][i] = v.x; m[k][i + 1] = v.y; m[k][i + 2] = v.z; m[k][i + 3] = v.w;
                    }
            } else {
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const float4 v = *reinterpret_cast<const float4 *>(Mb + (rg + 8 * i) * LDM + k4);
                    m[0][i] = v.x; m[1][i] = v.y; m[2][i] = v.z; m[3][i] = v.w;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int j = 0; j < PT; ++j) {
                    const Vec4<float> f = F[(k4 + k) * TP + 16 * j];
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        acc[i][j][0] += m[k][i] * f.x;
                        acc[i][j][1] += m[k][i] * f.y;
                        acc[i][j][2] += m[k][i] * f.z;
                    }
                }
        }
    }
    // two rows at a time: backward, their positions' loads ahead of the stores
#pragma unroll
    for (int i0 = 0; i0 < RT; i0 += 2) {
        int at[2];  // row of `out` (or of uvec, < 0: ~row)
        Vec4<double> v[2][PT];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int o = row_of(i0 + i), r = d.first + o;
            const bool in = o < d.count;
            at[i] = !in ? 0 : BWD || r < d.n ? column(r) : ~(d.u_off + (r - d.n));
            if (BWD)
#pragma unroll
                for (int j = 0; j < PT; ++j) {
                    const int p = p0 + pg + 16 * j;
                    if (in && p < P) v[i][j] = pc64[(int64_t)at[i] * P + p];
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (row_of(i0 + i) >= d.count) continue;
            Vec4<float> *dst = at[i] >= 0 ? out + (int64_t)at[i] * P : uvec + (int64_t)~at[i] * P;
#pragma unroll
            for (int j = 0; j < PT; ++j) {
                const int p = p0 + pg + 16 * j;
                if (p >= P) continue;
                const float *x = acc[i0 + i][j];
                if (!BWD || out) dst[p] = {x[0], x[1], x[2], 0.f};
                if (BWD) {
                    Vec4<double> q = v[i][j];
                    q.x += dev::to_double(x[0]);
                    q.y += dev::to_double(x[1]);
                    q.z += dev::to_double(x[2]);
                    pc64[(int64_t)at[i] * P + p] = q;
                }
            }
        }
    }
}
