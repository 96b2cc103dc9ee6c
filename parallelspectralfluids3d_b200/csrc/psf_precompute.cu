// Per-domain precompute kernels (include/psf_precompute.h): the operator
// product of the eigen-solve and the advection tensor build, FP64 throughout.
//
//   psf_csr_cheb     one warp per row of a CSR matrix, 16-byte gathers of the
//                    block's rows, fused with the Chebyshev three-term
//                    recurrence (out = alpha A Y + beta Y + gamma X)
//   psf_wedge_w      W[e][k][j] = sum_g q_e[g][k] Phi[g_e][j] with
//                    q_e[g][k] = sum_f S_e[f][g] Phi[f_e][k] over the
//                    (at most 8) faces the edge's terms name: the wedge
//                    matrices of a batch of modes, one warp per edge.  S_e is
//                    antisymmetric, so W[e][k][j] = -W[e][j][k] and only the
//                    columns j > k of a mode are made
//   psf_wedge_gemm   partial[s][a][c] = sum_{e in split s} Psi[e][a] W[e][c]:
//                    a 64 x 128 x 16 FP64 tile GEMM on mma.sync with a
//                    three-stage cp.async pipeline, split along the edges
//   psf_wedge_reduce C[k][a][j] = (1/lambda_k) sum_s partial[s][a][(k, j)] and
//                    C[j][a][k] = -(1/lambda_j) of the same sum, splits summed
//                    in a fixed order (deterministic)
//
// The reference builds the same tensor with dense E x N matrices per mode
// (Solver/SolverImpl/psfsolver.cpp:431-551); here the 12 wedge terms of every
// voxel are gathered per edge into an antisymmetric matrix over the faces
// its terms name, so W_k is generated on the fly from Phi and never held for
// more than a batch of modes.  (The reference's edge slots pair one term in
// twelve with a face that does not touch the edge, so an edge can name five
// faces; eight slots cover any four terms.)

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>

#include "psf_internal.h"
#include "psf_precompute.h"

namespace {

using psf::cuda_fail;
using psf::fail;

// ------------------------------------------------------------- CSR x block
// Warp w of the grid takes rows w, w + warps, ...; the row's non-zeros are
// staged in the warp's shared slots (broadcast reads), and lane l owns the
// double2 columns l, l + 32, ... of the block.
__global__ void __launch_bounds__(256) psf_csr_cheb(long long n_rows, int m2, long long ld2,
                                                    const int32_t *__restrict__ row_ptr,
                                                    const int32_t *__restrict__ col_idx,
                                                    const double *__restrict__ vals, const double2 *__restrict__ Y,
                                                    const double2 *__restrict__ X, double2 *__restrict__ out,
                                                    double alpha, double beta, double gamma)
{
    __shared__ int32_t scol[8][32];
    __shared__ double sval[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nwarps = (long long)gridDim.x * 8;
    for (long long row = (long long)blockIdx.x * 8 + warp; row < n_rows; row += nwarps) {
        const int b = __ldg(row_ptr + row), e = __ldg(row_ptr + row + 1);
        for (int c0 = 0; c0 < m2; c0 += 32) {
            const int c = c0 + lane;
            double2 acc = make_double2(0.0, 0.0);
            for (int p0 = b; p0 < e; p0 += 32) {
                const int cnt = min(32, e - p0);
                __syncwarp();
                if (lane < cnt) {
                    scol[warp][lane] = __ldg(col_idx + p0 + lane);
                    sval[warp][lane] = __ldg(vals + p0 + lane);
                }
                __syncwarp();
                if (c < m2) {
                    int q = 0;
                    for (; q + 4 <= cnt; q += 4) {
                        const double2 y0 = __ldg(Y + (size_t)scol[warp][q] * ld2 + c);
                        const double2 y1 = __ldg(Y + (size_t)scol[warp][q + 1] * ld2 + c);
                        const double2 y2 = __ldg(Y + (size_t)scol[warp][q + 2] * ld2 + c);
                        const double2 y3 = __ldg(Y + (size_t)scol[warp][q + 3] * ld2 + c);
                        const double v0 = sval[warp][q], v1 = sval[warp][q + 1];
                        const double v2 = sval[warp][q + 2], v3 = sval[warp][q + 3];
                        acc.x = fma(v0, y0.x, acc.x);
                        acc.y = fma(v0, y0.y, acc.y);
                        acc.x = fma(v1, y1.x, acc.x);
                        acc.y = fma(v1, y1.y, acc.y);
                        acc.x = fma(v2, y2.x, acc.x);
                        acc.y = fma(v2, y2.y, acc.y);
                        acc.x = fma(v3, y3.x, acc.x);
                        acc.y = fma(v3, y3.y, acc.y);
                    }
                    for (; q < cnt; ++q) {
                        const double2 y = __ldg(Y + (size_t)scol[warp][q] * ld2 + c);
                        const double v = sval[warp][q];
                        acc.x = fma(v, y.x, acc.x);
                        acc.y = fma(v, y.y, acc.y);
                    }
                }
            }
            if (c < m2) {
                double2 r = make_double2(alpha * acc.x, alpha * acc.y);
                if (beta != 0.0) {
                    const double2 y = __ldg(Y + (size_t)row * ld2 + c);
                    r.x = fma(beta, y.x, r.x);
                    r.y = fma(beta, y.y, r.y);
                }
                if (gamma != 0.0) {
                    const double2 x = __ldg(X + (size_t)row * ld2 + c);
                    r.x = fma(gamma, x.x, r.x);
                    r.y = fma(gamma, x.y, r.y);
                }
                out[(size_t)row * ld2 + c] = r;
            }
        }
    }
}

// ------------------------------------------------------------ wedge terms
constexpr int WEDGE_KB_MAX = 64;  // modes per W batch (shared-memory q table)
constexpr int SLOTS = PSF_WEDGE_SLOTS;

// Columns of a batch of modes k0 .. k0 + kb: mode k has the columns j from
// first_of(k) (k + 1 rounded down to even, for 16-byte accesses) to N rounded
// up to even, one mode after the other.
__host__ __device__ __forceinline__ int first_of(int k) { return (k + 1) & ~1; }
__host__ __device__ __forceinline__ long long columns_before(int N, int k0, int k)
{
    // sum over k0 <= i < k of (N2 - first_of(i)); first_of sums to m (m + 1) / 2 rounded per parity
    const long long N2 = (N + 1) & ~1;
    const long long f1 = (long long)(k / 2) * ((k + 1) / 2), f0 = (long long)(k0 / 2) * ((k0 + 1) / 2);
    return (long long)(k - k0) * N2 - 2 * (f1 - f0);
}

// One warp per edge: q_e[g][kk] in shared memory (used slots compacted to
// the front), then the edge's W rows.  Slots holding the zero row are
// skipped; the test is warp-uniform.  Rows e >= n_edges (padding up to whole
// GEMM chunks) are written as zeros.  Bound by the stores: 0.18 ms for the
// 0.72 GB of two batches at 16^3, N = 128 (0.28 ms with all columns).
__global__ void __launch_bounds__(256) psf_wedge_w(long long n_edges, long long n_rows, int N, int ldn, long long ldc,
                                                   int k0, int kb, const int32_t *__restrict__ edge_faces,
                                                   const double *__restrict__ edge_S,
                                                   const double *__restrict__ phi, long long zero_row,
                                                   double *__restrict__ W)
{
    __shared__ double qs[8][SLOTS][WEDGE_KB_MAX];
    __shared__ int32_t fs[8][SLOTS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nwarps = (long long)gridDim.x * 8;
    const int n2 = (N + 1) / 2;
    for (long long e = (long long)blockIdx.x * 8 + warp; e < n_rows; e += nwarps) {
        double2 *We = reinterpret_cast<double2 *>(W + (size_t)e * ldc);
        if (e >= n_edges) {
            for (long long i = lane; i < ldc / 2; i += 32) We[i] = make_double2(0.0, 0.0);
            continue;
        }
        __syncwarp();
        int f[SLOTS];
#pragma unroll
        for (int g = 0; g < SLOTS; ++g) f[g] = __ldg(edge_faces + (size_t)SLOTS * e + g);
        for (int kk = lane; kk < kb; kk += 32) {
            double pk[SLOTS];
#pragma unroll
            for (int h = 0; h < SLOTS; ++h)
                pk[h] = f[h] == zero_row ? 0.0 : __ldg(phi + (size_t)f[h] * ldn + k0 + kk);
            int u = 0;
#pragma unroll
            for (int g = 0; g < SLOTS; ++g) {
                if (f[g] == zero_row) continue;
                double q = 0.0;
#pragma unroll
                for (int h = 0; h < SLOTS; ++h) q = fma(__ldg(edge_S + ((size_t)SLOTS * e + h) * SLOTS + g), pk[h], q);
                qs[warp][u++][kk] = q;
            }
        }
        int used = 0;
#pragma unroll
        for (int g = 0; g < SLOTS; ++g)
            if (f[g] != zero_row) {
                if (lane == 0) fs[warp][used] = f[g];
                ++used;
            }
        __syncwarp();
        for (int c2 = first_of(k0) / 2; c2 < n2; c2 += 32) {
            const int j2 = c2 + lane;
            double2 p[SLOTS];
#pragma unroll
            for (int g = 0; g < SLOTS; ++g)
                if (g < used && j2 < n2)
                    p[g] = __ldg(reinterpret_cast<const double2 *>(phi + (size_t)fs[warp][g] * ldn) + j2);
            // Modes with a column in this run; `at` is the place of mode k's column pair 0.
            const int kend = min(kb, 2 * min(c2 + 32, n2) - k0);
            double2 *at = We - first_of(k0) / 2;
            for (int kk = 0; kk < kend; ++kk) {
                const int first2 = first_of(k0 + kk) / 2;
                double2 w = make_double2(0.0, 0.0);
#pragma unroll
                for (int g = 0; g < SLOTS; ++g)
                    if (g < used) {
                        const double q = qs[warp][g][kk];
                        w.x = fma(q, p[g].x, w.x);
                        w.y = fma(q, p[g].y, w.y);
                    }
                if (j2 >= first2 && j2 < n2) at[j2] = w;
                at += n2 - first_of(k0 + kk + 1) / 2;
            }
        }
    }
}

// ---------------------------------------------------------- FP64 tile GEMM
constexpr int GB_M = 64, GB_N = 128, GB_K = 16, GB_STAGES = 3, GB_THREADS = 128;
constexpr int GB_PA = GB_M + 4, GB_PB = GB_N + 4;  // row pitches: 32 bytes beyond a bank cycle
constexpr int GB_SMEM = GB_STAGES * GB_K * (GB_PA + GB_PB) * 8;
constexpr int GB_PER_SM = 2;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int src_bytes)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], const double (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// partial[split][a][c] over the edge chunks of split `blockIdx.z`: A = psi
// [n_edges][ldn] (rows beyond n_edges read as zero), B = W [rows][ldc].  A
// warp owns 64 rows x 32 columns as 4 x 4 tiles of 16 x 8.  Rows and columns
// of a tile are assigned so that a lane's fragments are neighbours in shared
// memory: fragment row g (g + 8) is row 2g (2g + 1) of the 16, and column n of
// an even (odd) tile is column 2n (2n + 1) of a pair's 16; every fragment load
// is then 16 bytes and free of bank conflicts.
//
// Bound by the FP64 units: mma.sync m16n8k8 runs at 37.1 TFLOP/s on registers
// alone, an 8 x 8 outer product of FMAs (the form this replaces) at 31.0.
// Half of the columns are left out by antisymmetry, 64-row tiles follow N more
// closely than 128-row ones (ldn is the padded size), and two blocks per SM
// cover each other's barriers.  16^3 box, N = 128 (11,280 edges): 0.77 ms in
// two batches against 2.69 ms; the whole tensor 0.96 against 2.97 ms, 20^3,
// N = 256: 12.9 against 37.2 ms, 11 x 17 x 13, N = 25: 0.06 against 0.36 ms.
__global__ void __launch_bounds__(GB_THREADS, GB_PER_SM) psf_wedge_gemm(long long n_edges, int ldn, long long ldc,
                                                                        long long chunks_per_split,
                                                                        long long n_chunks,
                                                                        const double *__restrict__ psi,
                                                                        const double *__restrict__ W,
                                                                        double *__restrict__ partial)
{
    extern __shared__ __align__(16) double gsm[];
    double *As = gsm;                             // [STAGES][K][PA]
    double *Bs = gsm + GB_STAGES * GB_K * GB_PA;  // [STAGES][K][PB]
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wn = (tid >> 5) * 32;
    const int a0 = blockIdx.y * GB_M;
    const long long c0 = (long long)blockIdx.x * GB_N;
    const long long ch0 = (long long)blockIdx.z * chunks_per_split;
    const long long ch1 = min(n_chunks, ch0 + chunks_per_split);
    const int nk = (int)max(0ll, ch1 - ch0);

    auto load_stage = [&](int kt, int slot) {
        const long long e0 = (ch0 + kt) * GB_K;
        double *sa = As + slot * GB_K * GB_PA, *sb = Bs + slot * GB_K * GB_PB;
#pragma unroll
        for (int r = 0; r < GB_K * GB_M / 2 / GB_THREADS; ++r) {
            const int q = tid + GB_THREADS * r, row = q / (GB_M / 2), piece = q % (GB_M / 2);
            const bool ok = e0 + row < n_edges;
            cp_async16(sa + row * GB_PA + 2 * piece, ok ? psi + (size_t)(e0 + row) * ldn + a0 + 2 * piece : psi,
                       ok ? 16 : 0);
        }
#pragma unroll
        for (int r = 0; r < GB_K * GB_N / 2 / GB_THREADS; ++r) {
            const int q = tid + GB_THREADS * r, row = q / (GB_N / 2), piece = q % (GB_N / 2);
            cp_async16(sb + row * GB_PB + 2 * piece, W + (size_t)(e0 + row) * ldc + c0 + 2 * piece, 16);
        }
    };

    double acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;

#pragma unroll
    for (int s = 0; s < GB_STAGES - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_async_commit();
    }
    int slot = 0;
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<GB_STAGES - 2>();
        __syncthreads();
        const int nxt = kt + GB_STAGES - 1;
        if (nxt < nk) load_stage(nxt, slot == 0 ? GB_STAGES - 1 : slot - 1);
        cp_async_commit();
        const double *A = As + slot * GB_K * GB_PA + 2 * g;
        const double *B = Bs + slot * GB_K * GB_PB + wn + 2 * g;
        slot = slot + 1 == GB_STAGES ? 0 : slot + 1;
#pragma unroll
        for (int k8 = 0; k8 < GB_K; k8 += 8) {
            double a[4][4], b[4][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = k8 + 4 * h + t;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double2 v = *reinterpret_cast<const double2 *>(A + k * GB_PA + 16 * i);
                    a[i][2 * h] = v.x;
                    a[i][2 * h + 1] = v.y;
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const double2 v = *reinterpret_cast<const double2 *>(B + k * GB_PB + 16 * j);
                    b[2 * j][h] = v.x;
                    b[2 * j + 1][h] = v.y;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_f64(acc[i][j], a[i], b[j]);
        }
    }
    cp_async_wait<0>();

    double *P = partial + ((size_t)blockIdx.z * gridDim.y * GB_M + a0) * ldc + c0 + wn + 4 * t;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            double *row = P + (size_t)(16 * i + 2 * g + r) * ldc;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const double *even = acc[i][2 * j] + 2 * r, *odd = acc[i][2 * j + 1] + 2 * r;
                *reinterpret_cast<double2 *>(row + 16 * j) = make_double2(even[0], odd[0]);
                *reinterpret_cast<double2 *>(row + 16 * j + 2) = make_double2(even[1], odd[1]);
            }
        }
}

// A warp sums one row a of one mode k at a time, lanes along j.
__global__ void __launch_bounds__(256) psf_wedge_reduce(int N, int rows, long long ldc, int k0, int kb, int splits,
                                                        const double *__restrict__ partial,
                                                        const double *__restrict__ lam, double *__restrict__ C)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * 8;
    const size_t split_stride = (size_t)rows * ldc;
    for (long long t = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); t < (long long)kb * N; t += nwarps) {
        const int kk = (int)(t / N), a = (int)(t % N), k = k0 + kk;
        const double *src = partial + (size_t)a * ldc + columns_before(N, k0, k) - first_of(k);
        const double lk = lam[k];
        double *row = C + ((size_t)k * N + a) * N;
        if (lane == 0) row[k] = 0.0;
        for (int j = k + 1 + lane; j < N; j += 32) {
            double s = 0.0;
            for (int p = 0; p < splits; ++p) s += __ldcs(src + p * split_stride + j);
            row[j] = s / lk;
            C[((size_t)j * N + a) * N + k] = -s / lam[j];
        }
    }
}

// Work split of one W batch.  The grid is (column tiles, row tiles, edge
// splits); the splits are chosen so that the last of its waves over
// GB_PER_SM blocks per SM is well filled, against the cost of more partial
// sums: a chunk of a full wave takes about 2.4 us, a block's start and end
// about eight chunks, a partial sum is written and read once at about 5 TB/s.
struct WedgePlan {
    long long n_chunks, rows, ldc, row_tiles, col_tiles, splits, chunks_per_split;
    size_t w_bytes, partial_bytes;
};

// What the workspace of batches of k_batch modes may take: W with all ldn columns
// of a mode and its partial sums over so many splits that 128 x 128 tiles of them
// come to about two per SM, which is what it took before half of the columns were
// left out: N = 512 in batches of 8 modes (5,000 edges) would take 258 MB instead
// of 214 otherwise.  Fewer splits cost up to 13 % there (16^3, N = 512: 60.5 against
// 53.6 ms, with all columns 149 ms); up to N = 256 in batches of 64 modes the bound
// changes nothing.
size_t workspace_bound(const psf_wedge_desc *d, int k_batch)
{
    const long long chunks = (d->n_edges + GB_K - 1) / GB_K, ldc = (long long)k_batch * d->ldn;
    const long long tiles = (long long)(d->ldn / 128) * (ldc / 128);
    long long splits = std::max(1ll, std::min({(2ll * 148 + tiles - 1) / tiles, 64ll, std::max(1ll, chunks)}));
    const long long per = std::max(1ll, (chunks + splits - 1) / splits);
    splits = std::max(1ll, (chunks + per - 1) / per);
    return (size_t)(chunks * GB_K + splits * d->ldn) * ldc * sizeof(double);
}

WedgePlan plan_of(const psf_wedge_desc *d, int k_batch, int k0)
{
    const int kb = std::min(k_batch, d->n_modes - k0);
    WedgePlan p{};
    p.n_chunks = (d->n_edges + GB_K - 1) / GB_K;
    p.rows = p.n_chunks * GB_K;
    p.col_tiles = std::max(1ll, (columns_before(d->n_modes, k0, k0 + kb) + GB_N - 1) / GB_N);
    p.ldc = p.col_tiles * GB_N;
    p.row_tiles = (d->n_modes + GB_M - 1) / GB_M;
    const long long tiles = p.row_tiles * p.col_tiles, slots = 148ll * GB_PER_SM;
    p.w_bytes = (size_t)p.rows * p.ldc * sizeof(double);
    // The partial sums follow the W of the first batch, the largest.
    const long long ldc0 = (columns_before(d->n_modes, 0, k_batch) + GB_N - 1) / GB_N * GB_N;
    const size_t split_bytes = (size_t)p.row_tiles * GB_M * p.ldc * sizeof(double);
    const long long most = (long long)((workspace_bound(d, k_batch) - (size_t)p.rows * ldc0 * sizeof(double)) / split_bytes);
    double best = 1e300;
    p.splits = p.chunks_per_split = 1;
    for (long long s = 1; s <= std::min(64ll, std::max(1ll, p.n_chunks)); ++s) {
        const long long per = std::max(1ll, (p.n_chunks + s - 1) / s);
        const long long used = std::max(1ll, (p.n_chunks + per - 1) / per);
        const double cost = (double)((tiles * used + slots - 1) / slots) * (double)(per + 8) * 2.4 +
                            (double)used * (double)(tiles * GB_M * GB_N * 16) / 5e6;
        if (cost < best && used <= std::max(1ll, most)) {
            best = cost;
            p.splits = used;
            p.chunks_per_split = per;
        }
    }
    p.partial_bytes = (size_t)p.splits * split_bytes;
    return p;
}

// Workspace layout: W of the largest batch (the first) at offset 0, then the
// partial sums, sized for the batch that needs most.
struct Workspace {
    size_t w_bytes, partial_bytes;
};

Workspace workspace_of(const psf_wedge_desc *d, int kb)
{
    Workspace ws{0, 0};
    for (int k0 = 0; k0 < d->n_modes; k0 += kb) {
        const WedgePlan q = plan_of(d, kb, k0);
        ws.w_bytes = std::max(ws.w_bytes, q.w_bytes);
        ws.partial_bytes = std::max(ws.partial_bytes, q.partial_bytes);
    }
    return ws;
}

int check_desc(const psf_wedge_desc *d, int kb)
{
    if (!d) return fail(PSF_ERR_INVALID, "null wedge descriptor");
    if (d->n_edges < 0 || d->n_modes < 1 || d->ldn < d->n_modes || d->ldn % 128 != 0)
        return fail(PSF_ERR_INVALID, "wedge descriptor: n_modes >= 1 and ldn a multiple of 128 >= n_modes");
    if (kb < 1 || kb > d->n_modes || kb > WEDGE_KB_MAX)
        return fail(PSF_ERR_INVALID, "k_batch must be in [1, min(n_modes, 64)]");
    if (d->n_edges > 0 && (!d->edge_faces || !d->edge_S || !d->psi))
        return fail(PSF_ERR_INVALID, "null wedge array");
    if (!d->phi || !d->eigenvalues) return fail(PSF_ERR_INVALID, "null phi or eigenvalues");
    if (d->phi_zero_row < 0) return fail(PSF_ERR_INVALID, "phi_zero_row must be a row of phi");
    return PSF_OK;
}

}  // namespace

extern "C" int psf_pre_csr_cheb(int64_t n_rows, int64_t n_cols, int32_t m, int64_t ld, const int32_t *row_ptr,
                                const int32_t *col_idx, const double *vals, const double *Y, const double *X,
                                double *out, double alpha, double beta, double gamma, void *stream)
{
    if (n_rows < 0 || n_cols < 0 || m < 0 || ld < m || (ld & 1))
        return fail(PSF_ERR_INVALID, "psf_pre_csr_cheb: need 0 <= m <= ld, ld even");
    if (beta != 0.0 && n_rows != n_cols)
        return fail(PSF_ERR_INVALID, "psf_pre_csr_cheb: beta != 0 needs a square matrix");
    if (n_rows == 0 || m == 0) return PSF_OK;
    if (!row_ptr || !col_idx || !vals || !Y || !out || (gamma != 0.0 && !X))
        return fail(PSF_ERR_INVALID, "psf_pre_csr_cheb: null array");
    if ((reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(out) |
         (gamma != 0.0 ? reinterpret_cast<uintptr_t>(X) : 0)) & 15)
        return fail(PSF_ERR_INVALID, "psf_pre_csr_cheb: blocks must be 16-byte aligned");
    if (out == Y || (gamma != 0.0 && out == X))
        return fail(PSF_ERR_INVALID, "psf_pre_csr_cheb: out aliases an input");
    const long long blocks = std::min<long long>((n_rows + 7) / 8, 148ll * 16);
    psf_csr_cheb<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        n_rows, (m + 1) / 2, ld / 2, row_ptr, col_idx, vals, reinterpret_cast<const double2 *>(Y),
        reinterpret_cast<const double2 *>(X), reinterpret_cast<double2 *>(out), alpha, beta, gamma);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_csr_cheb launch");
}

extern "C" int psf_pre_advection_workspace(const psf_wedge_desc *d, int32_t k_batch, int64_t *bytes)
{
    int rc = check_desc(d, k_batch);
    if (rc != PSF_OK) return rc;
    if (!bytes) return fail(PSF_ERR_INVALID, "null output");
    const Workspace ws = workspace_of(d, k_batch);
    *bytes = (int64_t)(ws.w_bytes + ws.partial_bytes);
    return PSF_OK;
}

extern "C" int psf_pre_advection_tensor(const psf_wedge_desc *d, int32_t k_batch, void *workspace,
                                        int64_t workspace_bytes, double *C, void *stream)
{
    int rc = check_desc(d, k_batch);
    if (rc != PSF_OK) return rc;
    if (!C || !workspace) return fail(PSF_ERR_INVALID, "null tensor or workspace");
    const Workspace ws = workspace_of(d, k_batch);
    if (workspace_bytes < 0 || (size_t)workspace_bytes < ws.w_bytes + ws.partial_bytes)
        return fail(PSF_ERR_INVALID, "workspace smaller than psf_pre_advection_workspace");
    if ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(d->psi) |
         reinterpret_cast<uintptr_t>(d->phi)) & 15)
        return fail(PSF_ERR_INVALID, "workspace, psi and phi must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *W = static_cast<double *>(workspace);
    double *partial = reinterpret_cast<double *>(static_cast<char *>(workspace) + ws.w_bytes);
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev >= 64 || !configured[dev]) {
        e = cudaFuncSetAttribute(psf_wedge_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, GB_SMEM);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(psf_wedge_gemm)");
        if (dev < 64) configured[dev] = true;
    }
    const int N = d->n_modes;
    for (int k0 = 0; k0 < N; k0 += k_batch) {
        const int kb = std::min(k_batch, N - k0);
        const WedgePlan q = plan_of(d, k_batch, k0);
        const long long wblocks = std::max(1ll, std::min<long long>((q.rows + 7) / 8, 148ll * 16));
        psf_wedge_w<<<(unsigned)wblocks, 256, 0, st>>>(d->n_edges, q.rows, N, d->ldn, q.ldc, k0, kb, d->edge_faces,
                                                       d->edge_S, d->phi, d->phi_zero_row, W);
        if (q.n_chunks > 0) {
            const dim3 grid((unsigned)q.col_tiles, (unsigned)q.row_tiles, (unsigned)q.splits);
            psf_wedge_gemm<<<grid, GB_THREADS, GB_SMEM, st>>>(d->n_edges, d->ldn, q.ldc, q.chunks_per_split,
                                                             q.n_chunks, d->psi, W, partial);
        } else {
            e = cudaMemsetAsync(partial, 0, q.partial_bytes, st);
            if (e != cudaSuccess) return cuda_fail(e, "clearing the partial sums");
        }
        const long long rblocks = std::min<long long>(((long long)kb * N + 7) / 8, 148ll * 8);
        psf_wedge_reduce<<<(unsigned)rblocks, 256, 0, st>>>(N, (int)(q.row_tiles * GB_M), q.ldc, k0, kb, (int)q.splits,
                                                           partial, d->eigenvalues, C);
        e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "advection tensor launch");
    }
    return PSF_OK;
}
