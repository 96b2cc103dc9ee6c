// Batched spectral-fluid step on the 5th-generation tensor cores (sm_100a).
//
// Many instances ("slots") share one domain basis; a batch may hold several
// bases.  For the slots of one basis the two dense products of a step are
// GEMMs with the slots' coefficient vectors as the narrow operand:
//
//   contraction     Y[(k,a), b] = sum_j C[k][a][j] W[j][b]     (M = N*N, K = N)
//                   dw[k][b]    = sum_a w[a][b] Y[(k,a), b]     (epilogue, FP64)
//   reconstruction  U[f, b]     = sum_i Phi[f][i] W[i][b]       (M = F_act, K = N)
//
// C, Phi and W are stored as BF16 hi + lo pairs (x = hi + lo with both parts
// rounded to nearest) and each product is compensated:
// A_hi B_hi + A_hi B_lo + A_lo B_hi, accumulated in FP32 in TMEM.  Slots with
// fewer modes than the basis are zero-padded, which is exact: their W rows
// beyond N_b are zero, and dw_k for k >= N_b is ignored.
//
// psf_batch_step_tc is one persistent kernel over the tiles of every basis:
// warp 0 streams 128-row A tiles and the W tile through a TMA ring of
// shared-memory stages (128-byte swizzle, no multicast), warp 1 issues the
// tcgen05.mma chain for a tile into one of two TMEM accumulators, warps 2-9
// drain the other accumulator (tcgen05.ld) and run the epilogue, so loads,
// MMAs and epilogue overlap.  In the default (fused) step one cooperative
// launch runs the contraction, the FP64 state update of every slot and the
// reconstruction, separated by bounded grid barriers; the tracer
// (psf_batch_trace, the same interpolant as the single-instance path)
// completes the step.  Unfused launches (one GEMM each, plus
// psf_batch_state) serve autotuning and per-phase profiling.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "psf_b200.h"
#include "psf_batch_internal.h"
#include "psf_device.cuh"
#include "psf_internal.h"
#include "psf_sm100.cuh"

namespace psf {

using namespace sm100;

constexpr int TRACE_BLOCK = 128;

template <int BN_MAX>
struct GemmCfg {
    static constexpr int STAGES = BN_MAX == 64 ? 4 : (BN_MAX == 128 ? 3 : 2);
    static constexpr int A_BYTES = 2 * 128 * 128;  // hi + lo: 128 rows x 64 BF16
    static constexpr int B_BYTES = 2 * BN_MAX * 128;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int TMEM_COLS = 2 * BN_MAX;   // two accumulators
    static constexpr int BAR_BYTES = 256;
    static constexpr int SMEM = STAGES * STAGE_BYTES + BAR_BYTES + 1024;  // + alignment slack
};

// Work unit t of a launch: contraction units first, then reconstruction units.
// MODE 0 launches only contraction units, MODE 1 only reconstruction units,
// MODE 2 (fused) both, so the unit kind is known at compile time except there.
template <int MODE>
__device__ __forceinline__ const GemmGroup &unit_group(const StepArgs &a, int t, bool &recon, int *local)
{
    recon = MODE == 1 ? true : (MODE == 0 ? false : t >= a.c_tiles);
    int base = recon ? a.n_groups : 0;
    int u = recon ? t - a.c_tiles : t;
    int g = 0;
    while (g + 1 < a.n_groups && u >= a.g[base + g].tiles) {
        u -= a.g[base + g].tiles;
        ++g;
    }
    *local = u;
    return a.g[base + g];
}

// Work unit -> (outer index, row tile, K range [kc0, kc1)).
struct Unit {
    int outer, inner, ks, kc0, kc1;
};

__device__ __forceinline__ Unit decode_unit(const GemmGroup &G, int lt)
{
    Unit u;
    const int per_outer = G.m_inner * G.ksplit;
    u.outer = lt / per_outer;
    const int rem = lt - u.outer * per_outer;
    u.inner = rem / G.ksplit;
    u.ks = rem - u.inner * G.ksplit;
    u.kc0 = u.ks * G.kc_per;
    u.kc1 = min(G.k_chunks, u.kc0 + G.kc_per);
    return u;
}

// 32 values per lane -> lane l holds the sum over the warp of value l.
__device__ __forceinline__ float warp_reduce_scatter32f(float (&v)[32], int lane)
{
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool upper = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const float send = upper ? v[i] : v[i + s];
            const float keep = upper ? v[i + s] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    return v[0];
}

__device__ __forceinline__ double warp_allsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void epilogue_bar() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// Grid-wide barrier of a cooperative launch: arrive, then wait (bounded) until
// `target` arrivals were counted.  Called by one thread per CTA after a CTA
// barrier, as the cooperative-groups grid sync does.
__device__ __forceinline__ bool grid_sync(unsigned int *bar, unsigned int target, int *err)
{
    __threadfence();
    atomicAdd(bar, 1u);
    const unsigned long long t0 = globaltimer();
    for (;;) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if (v >= target) break;
        if (globaltimer() - t0 > PSF_WAIT_LIMIT_NS) {
            record_error(err, ERR_GRID_SYNC);
            return false;
        }
        __nanosleep(64);
    }
    __threadfence();
    return true;
}

__device__ __forceinline__ void split_bf16(double x, __nv_bfloat16 *hi, __nv_bfloat16 *lo)
{
    const __nv_bfloat16 h = __float2bfloat16_rn((float)x);
    *hi = h;
    *lo = __float2bfloat16_rn((float)(x - (double)__bfloat162float(h)));
}

// FP64 update of one slot by the epilogue threads of a CTA, in the
// reference's order (psfsolver.cpp:37-59), then the new state's FP32 copy and
// BF16 hi/lo split.  Energy sums: per warp (shuffles), then the warps in
// fixed order, so the result does not depend on timing.
__device__ void state_update_cta(const GroupDev *__restrict__ groups, SlotDev &s, int et, double *red)
{
    const int lane = et & 31, ew = et >> 5;
    if (!s.active) return;  // uniform over the threads
    if (s.target != 0ull && s.step >= s.target) {
        if (et == 0) s.stepped = 0;
        return;
    }
    const GroupDev &G = groups[s.group];
    const int b = s.slot, N = s.n_modes, parts = G.nparts;
    double *w = G.w + (size_t)b * G.N;
    double e1 = 0.0, e2 = 0.0;
    for (int i = et; i < N; i += EPI_THREADS) {
        double dw = 0.0;
        const double *dp = G.dwpart + (size_t)i * parts * G.cap + b;
        for (int p = 0; p < parts; ++p) dw += dp[(size_t)p * G.cap];
        const double wi = w[i];
        const double w1 = wi + s.dt * dw;
        w[i] = w1;
        e1 += wi * wi;
        e2 += w1 * w1;
    }
    e1 = warp_allsum(e1);
    e2 = warp_allsum(e2);
    if (lane == 0) {
        red[ew] = e1;
        red[EPI_WARPS + ew] = e2;
    }
    epilogue_bar();
    e1 = e2 = 0.0;
#pragma unroll
    for (int i = 0; i < EPI_WARPS; ++i) {
        e1 += red[i];
        e2 += red[EPI_WARPS + i];
    }
    const double scale = (s.flags & PSF_FLAG_RENORM) ? sqrt(e1 / e2) : 1.0;
    const int stepped = e1 > (double)s.fast_above ? STEPPED_FAST : STEPPED;
    __nv_bfloat16 *Whi = reinterpret_cast<__nv_bfloat16 *>(G.W) + (size_t)b * G.Nj;
    __nv_bfloat16 *Wlo = Whi + (size_t)G.bn * G.Nj;
    for (int i = et; i < N; i += EPI_THREADS) {
        double v = w[i] * scale;
        v *= exp(s.visc_signed * G.lam[i] * s.dt);
        if (s.flags & PSF_FLAG_FORCING) v += s.dt * G.force[(size_t)b * G.N + i];
        w[i] = v;
        G.wf[(size_t)b * G.N + i] = (float)v;
        split_bf16(v, Whi + i, Wlo + i);
    }
    epilogue_bar();  // red[] is reused by the next slot
    if (et == 0) {
        s.step += 1ull;
        s.stepped = stepped;
    }
}

// One launch of the tensor-core step.  Warp 0: TMA producer; warp 1: MMA
// issuer; warps 2-9: TMEM epilogue, two per lane quarter, which take every other
// 32 columns.  Unfused launches run their contraction
// or reconstruction units.  A fused launch (cooperative) is one whole step of
// the coefficient pipeline: the epilogue warps first update every slot's
// state from the contraction partials of the previous launch (FP64, one CTA
// per slot), a grid barrier makes the new coefficients visible, and then
// one sweep runs the reconstruction of the new state together with the
// contraction that the next step's update will use (both need only the new
// coefficients).  During the update the producer already loads the first
// tiles of C and Phi, which do not depend on the state, and issues their
// coefficient (W) loads once the barrier has passed.
template <int BN_MAX, int MODE>
__global__ void __launch_bounds__(GEMM_THREADS, 1) psf_batch_step_tc(const __grid_constant__ StepArgs args)
{
    using Cfg = GemmCfg<BN_MAX>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char *smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t *full = bars;
    uint64_t *empty = bars + STAGES;
    uint64_t *acc_full = bars + 2 * STAGES;
    uint64_t *acc_empty = acc_full + 2;
    uint64_t *wready = acc_empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(wready + 1);
    double *red = reinterpret_cast<double *>(wready + 2);  // 2 EPI_WARPS doubles (from byte 8 (2 STAGES + 6))

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *err = args.err;
    const int total = args.c_tiles + args.r_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], EPI_THREADS);
        }
        mbar_init(wready, 1);
        mbar_fence_init();
        for (int g = 0; g < 2 * args.n_groups; ++g) {
            tma_prefetch_desc(&args.g[g].tmA);
            tma_prefetch_desc(&args.g[g].tmB);
        }
    }
    if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------------------------------------------- TMA producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            uint32_t last_parity[STAGES];
            bool issued[STAGES];
            for (int s = 0; s < STAGES; ++s) issued[s] = false;
            // Stages whose W load waits for the state update (in this launch or
            // in the kernel before): their C or Phi tiles load meanwhile.
            int pend_stage[STAGES], pend_kc[STAGES], pend_t[STAGES];
            int npend = 0;
            bool w_ok = false;
            bool ok = true;
            auto flush = [&]() -> bool {
                if (MODE == 2) {
                    if (!mbar_wait(wready, 0u, err, ERR_WAIT_STATE)) return false;
                } else {
                    grid_dependency_wait();
                    launch_dependents();
                }
                for (int i = 0; i < npend; ++i) {
                    bool rc;
                    int lt;
                    const GemmGroup &G = unit_group<MODE>(args, pend_t[i], rc, &lt);
                    unsigned char *sB = smem + pend_stage[i] * Cfg::STAGE_BYTES + Cfg::A_BYTES;
                    tma_load_3d(sB, &G.tmB, &full[pend_stage[i]], pend_kc[i] * 64, 0, 0);
                }
                npend = 0;
                w_ok = true;
                return true;
            };
            for (int t = blockIdx.x; ok && t < total; t += gridDim.x) {
                bool recon;
                int lt;
                const GemmGroup &G = unit_group<MODE>(args, t, recon, &lt);
                const Unit un = decode_unit(G, lt);
                for (int kc = un.kc0; kc < un.kc1; ++kc) {
                    if (!mbar_wait(&empty[stage], phase ^ 1u, err, ERR_WAIT_EMPTY)) {
                        ok = false;
                        break;
                    }
                    unsigned char *sA = smem + stage * Cfg::STAGE_BYTES;
                    unsigned char *sB = sA + Cfg::A_BYTES;
                    mbar_arrive_expect_tx(&full[stage], G.tx_bytes);
                    tma_load_4d(sA, &G.tmA, &full[stage], kc * 64, un.inner * 128, 0, un.outer);
                    if (!w_ok) {
                        pend_stage[npend] = stage;
                        pend_kc[npend] = kc;
                        pend_t[npend] = t;
                        ++npend;
                    } else {
                        tma_load_3d(sB, &G.tmB, &full[stage], kc * 64, 0, 0);
                    }
                    issued[stage] = true;
                    last_parity[stage] = phase;
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                    if (npend == STAGES && !flush()) {
                        ok = false;
                        break;
                    }
                }
            }
            if (ok && npend > 0) ok = flush();
            // After an error, copies may still be in flight that no one
            // consumes: wait (bounded) for them before the CTA exits.
            if (*(volatile int *)err != 0)
                for (int s = 0; s < STAGES; ++s)
                    if (issued[s]) mbar_wait(&full[s], last_parity[s], err, ERR_WAIT_DRAIN);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int abuf = 0;
            uint32_t aphase = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < total; t += gridDim.x) {
                bool recon;
                int lt;
                const GemmGroup &G = unit_group<MODE>(args, t, recon, &lt);
                const Unit un = decode_unit(G, lt);
                if (!mbar_wait(&acc_empty[abuf], aphase ^ 1u, err, ERR_WAIT_ACC_EMPTY)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(abuf * BN_MAX);
                const uint32_t idesc = idesc_bf16_f32(128, G.bn);
                for (int kc = un.kc0; kc < un.kc1; ++kc) {
                    if (!mbar_wait(&full[stage], phase, err, ERR_WAIT_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = smem_u32(smem + stage * Cfg::STAGE_BYTES);
                    const uint32_t b0 = a0 + Cfg::A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint64_t ah = desc_kmajor_sw128(a0 + kk * 32);
                        const uint64_t al = desc_kmajor_sw128(a0 + 128 * 128 + kk * 32);
                        const uint64_t bh = desc_kmajor_sw128(b0 + kk * 32);
                        const uint64_t bl = desc_kmajor_sw128(b0 + (uint32_t)G.bn * 128u + kk * 32);
                        mma_bf16(d, ah, bh, idesc, (kc != un.kc0 || kk != 0) ? 1u : 0u);
                        mma_bf16(d, ah, bl, idesc, 1u);
                        mma_bf16(d, al, bh, idesc, 1u);
                    }
                    mma_commit(&empty[stage]);
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                mma_commit(&acc_full[abuf]);
                if (++abuf == 2) {
                    abuf = 0;
                    aphase ^= 1u;
                }
            }
        }
    } else {
        // -------------------------------------------------------- epilogue
        const int q = warp & 3;   // TMEM lanes 32q .. 32q+31 belong to this warp
        const int first = 32 * ((warp - 2) >> 2);  // and columns first + 64 i .. + 32
        const int row = q * 32 + lane;
        int abuf = 0;
        uint32_t aphase = 0;
        if (MODE != 2) grid_dependency_wait();
        if (MODE == 2) {
            // Every slot's state update (one CTA per slot), then a grid
            // barrier before any coefficient (W) load of the sweep.
            const int et = threadIdx.x - 64;
            for (int s = blockIdx.x; s < args.n_slots; s += gridDim.x)
                state_update_cta(args.groups, args.slots[s], et, red);
            // The new coefficients are read next by TMA (the async proxy).
            asm volatile("fence.proxy.async.global;" ::: "memory");
            epilogue_bar();
            if (threadIdx.x == 64) {
                if (grid_sync(args.grid_bar, gridDim.x, err)) mbar_arrive(wready);
            }
            epilogue_bar();
            // The epilogue reads other CTAs' new state (wf) below with
            // ordinary (L1-cached) loads: order them after the barrier.
            __threadfence();
        }
        for (int t = blockIdx.x; t < total; t += gridDim.x) {
            bool recon;
            int lt;
            const GemmGroup &G = unit_group<MODE>(args, t, recon, &lt);
            const Unit un = decode_unit(G, lt);
            const int outer = un.outer, inner = un.inner;
            // Two epilogue warps per lane quarter instead of one took the
            // contraction of 513 slots from 77.6 to 60 us and of 64 slots of
            // N = 384 from 52 to 45 us: with one, a CTA's last tiles waited
            // for the epilogue.
            // Contraction: the state values of this warp's rows for its first
            // slots are loaded while the accumulator is still being computed,
            // those of a later chunk one chunk ahead of its use.
            float wa[32];
            const int a_row = inner * 128 + row;
            const bool arow = !recon && a_row < G.n_rows;
            auto load_w = [&](int c0) {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const int b = c0 + c;
                    wa[c] = (arow && b < G.cap) ? G.wf[(size_t)b * G.ldw + a_row] : 0.f;
                }
            };
            if (!recon && first < G.bn) load_w(first);
            bool ok = mbar_wait(&acc_full[abuf], aphase, err, ERR_WAIT_ACC_FULL);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(abuf * BN_MAX);
            if (!recon) {
                // dw partial of mode k = outer over this warp's 32 rows a:
                // sum_a w[a][b] Y[a][b] for every slot b, in FP32.
                for (int c0 = first; c0 < G.bn; c0 += 64) {
                    float y[32];
                    tmem_ld32(tbase + (uint32_t)c0, y);
#pragma unroll
                    for (int c = 0; c < 32; ++c) y[c] *= wa[c];
                    if (c0 + 64 < G.bn) load_w(c0 + 64);
                    const float s = warp_reduce_scatter32f(y, lane);
                    const int b = c0 + lane;
                    if (b < G.cap)
                        G.dwpart[((size_t)outer * G.nparts + (inner * G.ksplit + un.ks) * 4 + q) * G.cap + b] =
                            (double)s;
                }
            } else {
                // Face velocities of this warp's 32 rows, scattered into the
                // field of every slot that stepped (a face lands in one place,
                // or in the pairs of its two voxels): the tracer reads no
                // others, so an empty or finished slot costs no stores.  The
                // stores bound this launch once the slots outnumber the modes
                // (FACE_FIELD_DENSITY has the figures).
                const long long f = (long long)inner * 128 + row;
                const bool frow = f < G.n_rows;
                const int32_t d0 = frow ? __ldg(G.field_dst + 2 * f) : -1;
                const int32_t d1 = frow ? __ldg(G.field_dst + 2 * f + 1) : -1;
                const size_t step = (size_t)G.field_floats;
                const bool twice = __any_sync(0xffffffffu, d1 >= 0);
                for (int c0 = first; c0 < G.bn; c0 += 64) {
                    const int bl = c0 + lane;
                    const unsigned stepped =
                        __ballot_sync(0xffffffffu, bl < G.cap && G.slot_of[bl].stepped != 0);
                    float y[32];
                    tmem_ld32(tbase + (uint32_t)c0, y);
                    auto put = [&](int32_t place) {
                        float *p = G.field + (size_t)c0 * step + max(place, 0);
                        if (stepped == 0xffffffffu) {
#pragma unroll
                            for (int c = 0; c < 32; ++c, p += step)
                                if (place >= 0) *p = y[c];
                        } else {
#pragma unroll
                            for (int c = 0; c < 32; ++c, p += step)
                                if (place >= 0 && ((stepped >> c) & 1u)) *p = y[c];
                        }
                    };
                    if (stepped) {
                        put(d0);
                        if (twice) put(d1);
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[abuf]);
            if (++abuf == 2) {
                abuf = 0;
                aphase ^= 1u;
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ------------------------------------------------------------ state update
// FP64 update of one slot in the reference's order (psfsolver.cpp:37-59),
// then the new state's BF16 hi/lo split for the next products.
__global__ void __launch_bounds__(256) psf_batch_state(const GroupDev *__restrict__ groups,
                                                       SlotDev *__restrict__ slots)
{
    __shared__ double red[8];
    __shared__ double wnew[PSF_MAX_MODES];
    launch_dependents();  // the reconstruction, which waits for this grid's end before it reads
    SlotDev &s = slots[blockIdx.x];
    if (!s.active) return;
    if (s.target != 0ull && s.step >= s.target) {
        if (threadIdx.x == 0) s.stepped = 0;
        return;
    }
    const GroupDev &G = groups[s.group];
    const int b = s.slot, N = s.n_modes, parts = G.nparts;
    double *w = G.w + (size_t)b * G.N;
    double e1 = 0.0, e2 = 0.0;
    for (int i = threadIdx.x; i < N; i += 256) {
        double dw = 0.0;
        const double *dp = G.dwpart + (size_t)i * parts * G.cap + b;
        for (int p = 0; p < parts; ++p) dw += dp[(size_t)p * G.cap];
        const double wi = w[i];
        const double w1 = wi + s.dt * dw;
        wnew[i] = w1;
        e1 += wi * wi;
        e2 += w1 * w1;
    }
    e1 = block_sum_256(e1, red);
    e2 = block_sum_256(e2, red);
    const double scale = (s.flags & PSF_FLAG_RENORM) ? sqrt(e1 / e2) : 1.0;
    const int stepped = e1 > (double)s.fast_above ? STEPPED_FAST : STEPPED;
    __nv_bfloat16 *Whi = reinterpret_cast<__nv_bfloat16 *>(G.W) + (size_t)b * G.Nj;
    __nv_bfloat16 *Wlo = Whi + (size_t)G.bn * G.Nj;
    for (int i = threadIdx.x; i < N; i += 256) {
        double v = wnew[i] * scale;
        v *= exp(s.visc_signed * G.lam[i] * s.dt);
        if (s.flags & PSF_FLAG_FORCING) v += s.dt * G.force[(size_t)b * G.N + i];
        w[i] = v;
        G.wf[(size_t)b * G.N + i] = (float)v;
        split_bf16(v, Whi + i, Wlo + i);
    }
    if (threadIdx.x == 0) {
        s.step += 1ull;
        s.stepped = stepped;
    }
}

// BF16 split of one slot's current state (after it was set from the host).
__global__ void psf_batch_pack(const GroupDev *__restrict__ groups, const SlotDev *__restrict__ slots, int sg)
{
    const SlotDev &s = slots[sg];
    const GroupDev &G = groups[s.group];
    __nv_bfloat16 *Whi = reinterpret_cast<__nv_bfloat16 *>(G.W) + (size_t)s.slot * G.Nj;
    __nv_bfloat16 *Wlo = Whi + (size_t)G.bn * G.Nj;
    for (int i = threadIdx.x; i < G.Nj; i += blockDim.x) {
        const double v = (s.active && i < s.n_modes) ? G.w[(size_t)s.slot * G.N + i] : 0.0;
        split_bf16(v, Whi + i, Wlo + i);
        if (i < G.N) G.wf[(size_t)s.slot * G.N + i] = (float)v;
    }
}

// ----------------------------------------------------------------- read-back
__global__ void psf_batch_gather_states(const ReadJob *__restrict__ jobs, double *__restrict__ w_out)
{
    const ReadJob &j = jobs[blockIdx.x];
    for (int i = threadIdx.x; i < j.n_w; i += blockDim.x) w_out[j.w_at + i] = j.w[i];
}

// A grid row per slot.  A slot by itself is a launch of a few microseconds that
// moves a few hundred KB; together they run at the memory's rate.
__global__ void psf_batch_unorder(const ReadJob *__restrict__ jobs, const float4 *__restrict__ pool,
                                  const int32_t *__restrict__ perm, float4 *__restrict__ stage)
{
    const ReadJob &j = jobs[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < j.n_parts; i += gridDim.x * blockDim.x)
        stage[j.stage + perm[j.poff + i]] = pool[j.poff + i];
}

// ------------------------------------------------------------------ tracer
// Every occupied slot's particles form one index space through the prefix
// sums of the slots' particle counts; a warp takes 32 neighbouring indices at a
// time, and a thread finds its particle's slot by a walk or a binary search in
// shared memory.  Slots that did not advance this step (step limit reached) are
// skipped.
//
// With pairs a warp puts aside the particles whose stages leave their first
// half-cell or whose life is over, and takes 32 of them at once: otherwise one
// such lane holds the other 31 for up to three more gathers.  Slots whose flow
// carries most particles out of their half-cell (FAST_STEP) go straight through
// after the others, and so do all where no thread has two particles (65,536 on
// 16^3 16.7 against 18.2 us a step; 131,072, beyond the grid, 19.6 either way).  16 x 262,144
// particles on the 32^3 box with a sphere, RK4: 107 against 126 us at 0.03 voxel
// per step, 136 against 141 at 0.12, 96 against 98 at 0.001; RK1 70 either way.
// Where faces are stored once (few particles per voxel) a warp's particles lie
// in many half-cells from the start and the first gather is most of the work:
// 276 against 268 us at 513 x 16,384 particles and 0.001 voxel per step, 319
// against 332 at 0.03; there, and with off-centre domains in the batch, every
// particle goes straight through.  So it does in the single-instance tracer
// too, which has two or three particles per thread: 17.5 us per step against
// 20.2 with the lists (32^3, 262,144), 75 against 80 (48^3, 1,048,576).
struct TraceSlot {
    const GroupDev *G = nullptr;
    const float *field = nullptr;
    size_t base = 0;  // the slot's first particle in its group's pool, less `first`
    TraceParams tp = {};
    uint64_t step = 0;
    bool live = false;

    __device__ __forceinline__ void load(const GroupDev *__restrict__ groups, const SlotDev &s, long long first)
    {
        live = s.stepped != 0;
        G = groups + s.group;
        base = (size_t)s.poff - (size_t)first;
        tp.dt = (float)s.dt;
        tp.lifetime = s.lifetime;
        tp.rk4 = s.rk4;
        tp.seed = s.seed;
        step = s.step - 1ull;
        field = G->field + (size_t)s.slot * (size_t)G->field_floats;
    }

    template <class Box>
    __device__ __forceinline__ void advance(size_t idx) const
    {
        using Ptr = typename Box::Ptr;
        G->parts[idx] = advance_particle<Box>(G->parts[idx], G->grid, reinterpret_cast<Ptr>(field), tp, step, G->perm, idx);
    }
};

// A particle put aside: its slot and its index in it.
__device__ __noinline__ void trace_later(const GroupDev *__restrict__ groups, const SlotDev &s, uint32_t at)
{
    TraceSlot t;
    t.load(groups, s, 0);
    t.advance<CentredBox<PairField>>(t.base + at);
}

// Slot of particle gi, searched from slot `from` on (-1: the first).
__device__ __forceinline__ int slot_of_particle(const long long *pre, int n_slots, int from, long long gi)
{
    int lo = from < 0 ? 0 : from;
    int walk = 0;
    while (pre[lo + 1] <= gi && walk < 8) {
        ++lo;
        ++walk;
    }
    if (pre[lo + 1] <= gi) {  // far away: binary search, pre[lo] <= gi < pre[hi]
        int hi = n_slots;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (pre[mid] <= gi)
                lo = mid;
            else
                hi = mid;
        }
    }
    return lo;
}

// The particles of slots that stepped in one of the ways from `least` on, each
// straight through.  In fast slots hardly one stays in its half-cell, and trying it
// there first cost up to 37 % (16 x 262,144, RK4, 0.9 voxel per step: 376 against 275
// us).  A function of its own: inlined, its registers cost the slow slots' loop 5 %.
__device__ __noinline__ void trace_straight(const GroupDev *__restrict__ groups, const SlotDev *__restrict__ slots,
                                            const long long *pre, int n_slots, long long total, int least)
{
    int cur = -1;
    TraceSlot t;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x; gi < total; gi += stride) {
        if (cur < 0 || gi >= pre[cur + 1]) {
            cur = slot_of_particle(pre, n_slots, cur, gi);
            t.load(groups, slots[cur], pre[cur]);
            t.live = slots[cur].stepped >= least;
        }
        if (t.live) t.advance<CentredBox<PairField>>(t.base + (size_t)gi);
    }
}

template <bool ALL_CENTRED, bool FACES>
__global__ void __launch_bounds__(TRACE_BLOCK, 5) psf_batch_trace(const GroupDev *__restrict__ groups,
                                                          const SlotDev *__restrict__ slots,
                                                          const long long *__restrict__ prefix, int n_slots)
{
    constexpr bool ASIDE = ALL_CENTRED && !FACES;
    __shared__ long long pre[BATCH_MAX_ALL_SLOTS + 1];
    __shared__ int32_t aside_slot[ASIDE ? TRACE_BLOCK / 32 : 1][64];
    __shared__ uint32_t aside_at[ASIDE ? TRACE_BLOCK / 32 : 1][64];
    __shared__ int any_fast;  // kept here, not in a register, until the end
    bool fast = false;
    for (int i = threadIdx.x; i <= n_slots; i += blockDim.x) {
        const int kind = ASIDE ? slots[min(i, n_slots - 1)].stepped : 0;
        pre[i] = prefix[i];
        fast |= kind == STEPPED_FAST;
    }
    if (ASIDE)
        any_fast = __syncthreads_or(fast);  // every thread writes, and reads what it wrote
    else
        __syncthreads();
    launch_dependents();  // the next step's contraction, which waits for this grid's end
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *as = aside_slot[ASIDE ? warp : 0];
    uint32_t *aa = aside_at[ASIDE ? warp : 0];
    const long long total = pre[n_slots];
    const long long stride = (long long)gridDim.x * blockDim.x;
    if constexpr (ASIDE) {
        if (total <= stride) {  // no second particle to put with those put aside
            trace_straight(groups, slots, pre, n_slots, total, STEPPED);
            return;
        }
    }
    // Parameters of the slot the thread is in, reloaded only when it changes.
    int cur = -1, waiting = 0;
    TraceSlot t;
    for (long long at = (long long)blockIdx.x * blockDim.x + warp * 32; at < total; at += stride) {
        const long long gi = at + lane;
        bool aside = false;
        if (gi < total) {
            if (cur < 0 || gi >= pre[cur + 1]) {
                cur = slot_of_particle(pre, n_slots, cur, gi);
                t.load(groups, slots[cur], pre[cur]);
                if (ASIDE) t.live = slots[cur].stepped == STEPPED;
            }
            if (t.live) {
                const size_t idx = t.base + (size_t)gi;
                if constexpr (ASIDE) {
                    float4 p = t.G->parts[idx];
                    aside = !advance_inside<PairField>(p, t.G->grid, reinterpret_cast<const float2 *>(t.field), t.tp);
                    if (!aside) t.G->parts[idx] = p;
                } else if constexpr (FACES) {
                    t.advance<CentredBox<FaceField>>(idx);
                } else if (t.G->grid.centered) {
                    t.advance<CentredBox<PairField>>(idx);
                } else {
                    t.advance<AnyBox>(idx);
                }
            }
        }
        if constexpr (ASIDE) {
            const unsigned m = __ballot_sync(0xffffffffu, aside);
            if (aside) {
                const int k = waiting + __popc(m & ((1u << lane) - 1u));
                as[k] = cur;
                aa[k] = (uint32_t)(gi - pre[cur]);
            }
            waiting += __popc(m);
            if (waiting >= 32) {
                __syncwarp();
                waiting -= 32;
                trace_later(groups, slots[as[waiting + lane]], aa[waiting + lane]);
                __syncwarp();
            }
        }
    }
    if constexpr (ASIDE) {
        __syncwarp();
        if (lane < waiting) trace_later(groups, slots[as[lane]], aa[lane]);
        if (any_fast) trace_straight(groups, slots, pre, n_slots, total, STEPPED_FAST);
    }
}

// A flow mixes its particles, and a warp's gathers then touch up to 32 lines
// each: after 4,000 steps at 0.03 voxel per step the tracer takes 143 instead of
// 111 us (16 x 262,144 on 32^3) and 86 instead of 53 (64 x 16,384 on 64 x 32 x
// 32).  Every so many steps the particles are put back in brick order, in place
// and with no memory of their own, in two launches:
//   1. A block takes a window of neighbouring particles, looks at 512 of them,
//      and sorts the window if more than a fifth of the neighbours lie in
//      different bricks (and more than 2.5 times as many as in a sorted slot).
//   2. In slots where that happened the windows, up to 128 at a time, deal their
//      sorted particles out: block i takes the i-th part of every window, sorts
//      the union and writes it to the same places, so that each part becomes a
//      run of neighbours of the whole slot (columnsort's first steps).
// The sort is one counting pass over the keys' range in the block, cut into at
// most 8,192 buckets; it need not be exact.  Results do not depend on the order:
// the caller's index goes with each particle.  A slot that has reached its steps
// is left alone, as another stream may be reading it.
// Bound by memory: 80 bytes a particle where both launches work, every 64 steps.
// Steps 2,048 to 3,584 with it and without: 124 against 156 us (16 x 262,144,
// 0.03 voxel per step), 46 against 54 (16 x 65,536, 0.01), 83 against 110 (64 x
// 16,384, 0.03), 68 against 72 (the same, 0.001), 25.3 against 25.7 (16 x
// 16,384, 0.001), 17.2 against 18.8 (64 x 1,000 on 16^3, 0.03).  Every 32 steps
// or 128, and thresholds of a tenth or two fifths, are within 2 % of this.
constexpr int ORDER_BLOCK = 512;
constexpr int ORDER_ITEMS = 8;                        // particles of a thread
constexpr int ORDER_MOST = ORDER_BLOCK * ORDER_ITEMS; // of a block
constexpr int ORDER_GROUP = 128;                      // windows dealt out together
constexpr int ORDER_WINDOW = ORDER_MOST - ORDER_GROUP;
constexpr int ORDER_BUCKETS = 8192;
constexpr int ORDER_SMEM = ORDER_MOST * (16 + 4) + ORDER_BUCKETS * 4;

template <bool DEAL>
__global__ void __launch_bounds__(ORDER_BLOCK, 2) psf_batch_reorder(const GroupDev *__restrict__ groups, SlotDev *slots,
                                                                    const long long *__restrict__ prefix, int n_slots,
                                                                    int round)
{
    extern __shared__ __align__(16) unsigned char order_smem[];
    float4 *sp = reinterpret_cast<float4 *>(order_smem);
    int32_t *si = reinterpret_cast<int32_t *>(sp + ORDER_MOST);
    uint32_t *count = reinterpret_cast<uint32_t *>(si + ORDER_MOST);
    __shared__ uint32_t lowest, highest, sums[ORDER_BLOCK / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Slot s has the blocks from prefix[s] / ORDER_WINDOW + s on, enough for its windows.
    int lo = 0, hi = n_slots;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] / ORDER_WINDOW + mid <= (long long)blockIdx.x)
            lo = mid;
        else
            hi = mid;
    }
    SlotDev &s = slots[lo];
    const long long n = prefix[lo + 1] - prefix[lo];
    const long long windows = (n + ORDER_WINDOW - 1) / ORDER_WINDOW;
    const long long v = (long long)blockIdx.x - (prefix[lo] / ORDER_WINDOW + lo);
    if (v >= windows || !s.stepped || (s.target && s.step >= s.target)) return;
    if (DEAL && (windows == 1 || s.mixed != round)) return;
    const GroupDev &G = groups[s.group];
    const long long w = ((n + windows - 1) / windows + 31) / 32 * 32;  // <= ORDER_WINDOW
    // The block's particles: of `m` windows from `first` on, places [o, o + len) each.
    long long first = v, m = 1, o = 0, len = w;
    if (DEAL) {
        first = v / ORDER_GROUP * ORDER_GROUP;
        m = min((long long)ORDER_GROUP, windows - first);
        const long long part = (w + m - 1) / m;
        o = (v - first) * part;
        len = min(part, w - o);
    }
    const long long end = min(n, (first + m) * w) - first * w;
    if (end <= 0 || len <= 0) return;
    const int T = (int)(end / w * len + max(0ll, min(len, end % w - o)));  // only the last windows can be short
    const size_t base = (size_t)s.poff + (size_t)(first * w + o);
    const Bricks bricks = bricks_of(G.grid);
    if (!DEAL) {
        // Neighbours in different bricks, in 512 of the window's particles.
        const int i = max(0, (T - ORDER_BLOCK) / 2) + tid;
        const uint32_t k = i < T ? bricks.key(G.grid, G.parts[base + i]) >> BRICK_BITS : 0u;
        const uint32_t k1 = __shfl_down_sync(0xffffffffu, k, 1);
        const int apart = __syncthreads_count(lane < 31 && i + 1 < T && k != k1);
        const int pairs = min(T, ORDER_BLOCK) * 31 / 32;
        const float sorted = (float)((double)bricks.nx * bricks.ny * bricks.nz / (double)n);
        if ((float)apart <= fmaxf(0.2f, 2.5f * sorted) * (float)pairs) return;
        if (tid == 0) s.mixed = round;
    }
    if (tid == 0) {
        lowest = 0xffffffffu;
        highest = 0u;
    }
    for (int i = tid; i < ORDER_BUCKETS; i += ORDER_BLOCK) count[i] = 0u;
    __syncthreads();
    float4 p[ORDER_ITEMS];
    int32_t id[ORDER_ITEMS];
    uint32_t key[ORDER_ITEMS];
    uint32_t kmin = 0xffffffffu, kmax = 0u;
#pragma unroll
    for (int q = 0; q < ORDER_ITEMS; ++q) {
        const int r = q * ORDER_BLOCK + tid;
        if (r < T) {
            const size_t at = base + (DEAL ? (size_t)(r / (int)len) * (size_t)w + (size_t)(r % (int)len) : (size_t)r);
            p[q] = G.parts[at];
            id[q] = G.perm[at];
            key[q] = bricks.key(G.grid, p[q]);
            kmin = min(kmin, key[q]);
            kmax = max(kmax, key[q]);
        }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) {
        atomicMin(&lowest, kmin);
        atomicMax(&highest, kmax);
    }
    __syncthreads();
    // Bucket of a key: never falls as the key grows.
    const uint32_t low = lowest, range = highest - low;
    const bool exact = range < (uint32_t)ORDER_BUCKETS;
    const float scale = (float)ORDER_BUCKETS / ((float)range + 1.0f);
    uint32_t rank[ORDER_ITEMS];
#pragma unroll
    for (int q = 0; q < ORDER_ITEMS; ++q) {
        if (q * ORDER_BLOCK + tid < T) {
            const uint32_t d = key[q] - low;
            key[q] = exact ? d : min((uint32_t)(ORDER_BUCKETS - 1), (uint32_t)((float)d * scale));
            rank[q] = atomicAdd(&count[key[q]], 1u);
        }
    }
    __syncthreads();
    // Exclusive sums over the buckets, 16 neighbours per thread.
    constexpr int PER = ORDER_BUCKETS / ORDER_BLOCK;
    uint32_t mine[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        mine[q] = count[tid * PER + q];
        sum += mine[q];
    }
    uint32_t upto = sum;
#pragma unroll
    for (int dlt = 1; dlt < 32; dlt <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, upto, dlt);
        if (lane >= dlt) upto += t;
    }
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    uint32_t before = upto - sum;
    for (int q = 0; q < warp; ++q) before += sums[q];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        count[tid * PER + q] = before;
        before += mine[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ORDER_ITEMS; ++q) {
        if (q * ORDER_BLOCK + tid < T) {
            const uint32_t to = count[key[q]] + rank[q];
            sp[to] = p[q];
            si[to] = id[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ORDER_ITEMS; ++q) {
        const int r = q * ORDER_BLOCK + tid;
        if (r < T) {
            const size_t at = base + (DEAL ? (size_t)(r / (int)len) * (size_t)w + (size_t)(r % (int)len) : (size_t)r);
            G.parts[at] = sp[r];
            G.perm[at] = si[r];
        }
    }
}

// --------------------------------------------------------------- launchers
int batch_gemm_smem_bytes(int bn_max)
{
    switch (bn_max) {
    case 64: return GemmCfg<64>::SMEM;
    case 128: return GemmCfg<128>::SMEM;
    case 256: return GemmCfg<256>::SMEM;
    default: return -1;
    }
}

template <int BN, int MODE>
static int launch_tc_t(const StepArgs &args, int grid, cudaStream_t st, bool after_kernel)
{
    // The shared-memory limit is a per-device attribute of the kernel.
    static unsigned long long configured = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured & bit)) {
        e = cudaFuncSetAttribute(psf_batch_step_tc<BN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 GemmCfg<BN>::SMEM);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(psf_batch_step_tc)");
        configured |= bit;
    }
    PdlLaunch L((unsigned)grid, GEMM_THREADS, st, after_kernel && MODE != 2, GemmCfg<BN>::SMEM);
    if (MODE == 2) {
        L.attr[0].id = cudaLaunchAttributeCooperative;
        L.attr[0].val.cooperative = 1;
        L.cfg.numAttrs = 1;
    }
    e = cudaLaunchKernelEx(&L.cfg, psf_batch_step_tc<BN, MODE>, args);
    if (e != cudaSuccess) return cuda_fail(e, "psf_batch_step_tc launch");
    return PSF_OK;
}

template <int MODE>
static int launch_tc_mode(const StepArgs &args, int bn_max, int grid, cudaStream_t st, bool after_kernel)
{
    switch (bn_max) {
    case 64: return launch_tc_t<64, MODE>(args, grid, st, after_kernel);
    case 128: return launch_tc_t<128, MODE>(args, grid, st, after_kernel);
    case 256: return launch_tc_t<256, MODE>(args, grid, st, after_kernel);
    }
    return fail(PSF_ERR_UNSUPPORTED, "GEMM variant must have 64, 128 or 256 columns");
}

int launch_batch_step_tc(const StepArgs &args, int bn_max, int grid, cudaStream_t st, bool after_kernel)
{
    const int total = args.c_tiles + args.r_tiles;
    if (total <= 0 && !args.fused) return PSF_OK;
    if (!args.fused) grid = std::min(grid, total);
    grid = std::max(1, grid);
    for (int g = 0; g < 2 * args.n_groups; ++g) {
        const bool used = g < args.n_groups ? args.c_tiles > 0 : args.r_tiles > 0;
        if (used && (args.g[g].bn > bn_max || args.g[g].bn % 16 != 0 || args.g[g].bn < 16))
            return fail(PSF_ERR_INVALID, "GEMM group N tile does not fit the kernel variant");
    }
    if (args.fused) return launch_tc_mode<2>(args, bn_max, grid, st, after_kernel);
    if (args.r_tiles == 0) return launch_tc_mode<0>(args, bn_max, grid, st, after_kernel);
    if (args.c_tiles == 0) return launch_tc_mode<1>(args, bn_max, grid, st, after_kernel);
    return fail(PSF_ERR_INVALID, "an unfused launch runs either contraction or reconstruction units");
}

// Largest persistent grid a cooperative launch of the variant can hold.
int max_fused_grid(int bn_max, int num_sms)
{
    int per_sm = 0;
    cudaError_t e = cudaSuccess;
    switch (bn_max) {
    case 64:
        cudaFuncSetAttribute(psf_batch_step_tc<64, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg<64>::SMEM);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, psf_batch_step_tc<64, 2>, GEMM_THREADS,
                                                          GemmCfg<64>::SMEM);
        break;
    case 128:
        cudaFuncSetAttribute(psf_batch_step_tc<128, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             GemmCfg<128>::SMEM);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, psf_batch_step_tc<128, 2>, GEMM_THREADS,
                                                          GemmCfg<128>::SMEM);
        break;
    default:
        cudaFuncSetAttribute(psf_batch_step_tc<256, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             GemmCfg<256>::SMEM);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, psf_batch_step_tc<256, 2>, GEMM_THREADS,
                                                          GemmCfg<256>::SMEM);
        break;
    }
    if (e != cudaSuccess) return 0;
    return per_sm * num_sms;
}

int launch_batch_state(const GroupDev *groups, SlotDev *slots, int n_slots, cudaStream_t st)
{
    if (n_slots <= 0) return PSF_OK;
    psf_batch_state<<<n_slots, 256, 0, st>>>(groups, slots);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_batch_state launch");
}

int launch_batch_pack(const GroupDev *groups, const SlotDev *slots, int slot_global, cudaStream_t st)
{
    psf_batch_pack<<<1, 256, 0, st>>>(groups, slots, slot_global);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_batch_pack launch");
}

int launch_batch_gather_states(const ReadJob *jobs, int n, double *w_out, cudaStream_t st)
{
    if (n <= 0) return PSF_OK;
    psf_batch_gather_states<<<n, 128, 0, st>>>(jobs, w_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_batch_gather_states launch");
}

int launch_batch_unorder(const ReadJob *jobs, int n, int max_parts, const float4 *pool, const int32_t *perm,
                         float4 *stage, cudaStream_t st)
{
    if (n <= 0 || max_parts <= 0) return PSF_OK;
    const dim3 grid((unsigned)std::min(256, (max_parts + 255) / 256), (unsigned)n);
    psf_batch_unorder<<<grid, 256, 0, st>>>(jobs, pool, perm, stage);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_batch_unorder launch");
}

int batch_trace_grid(int num_sms, bool faces)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, faces ? psf_batch_trace<true, true> : psf_batch_trace<true, false>, TRACE_BLOCK, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 4;
    return num_sms * per_sm;
}

int launch_batch_trace(const GroupDev *groups, const SlotDev *slots, const long long *prefix, int n_slots, int grid,
                       bool all_centred, bool faces, cudaStream_t st)
{
    if (n_slots < 1 || n_slots > BATCH_MAX_ALL_SLOTS) return fail(PSF_ERR_INVALID, "slot count out of range");
    auto kernel = faces         ? psf_batch_trace<true, true>
                  : all_centred ? psf_batch_trace<true, false>
                                : psf_batch_trace<false, false>;
    kernel<<<grid, TRACE_BLOCK, 0, st>>>(groups, slots, prefix, n_slots);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PSF_OK : cuda_fail(e, "psf_batch_trace launch");
}

// ------------------------------------------------------------ host helpers
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_tensor_map(CUtensorMap *map, void *base, int rank, const uint64_t *dims, const uint64_t *strides_bytes,
                      const uint32_t *box)
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p)
            return fail(PSF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    cuuint64_t d[5];
    cuuint64_t s[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; ++i) {
        d[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) s[i] = strides_bytes[i];
    }
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, base, d, s, bx, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(PSF_ERR_CUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
    return PSF_OK;
}

void split_bf16_host(double x, uint16_t *hi, uint16_t *lo)
{
    const __nv_bfloat16 h = __float2bfloat16_rn((float)x);
    const __nv_bfloat16 l = __float2bfloat16_rn((float)(x - (double)__bfloat162float(h)));
    std::memcpy(hi, &h, 2);
    std::memcpy(lo, &l, 2);
}

int prepare_batch_reorder()
{
    for (int deal = 0; deal < 2; ++deal) {
        auto kernel = deal ? psf_batch_reorder<true> : psf_batch_reorder<false>;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ORDER_SMEM);
        if (e != cudaSuccess) return cuda_fail(e, "psf_batch_reorder shared memory");
    }
    return PSF_OK;
}

int launch_batch_reorder(const GroupDev *groups, SlotDev *slots, const long long *prefix, int n_slots, long long total,
                         int round, cudaStream_t st)
{
    const long long blocks = total / ORDER_WINDOW + n_slots;
    for (int deal = 0; deal < 2; ++deal) {
        auto kernel = deal ? psf_batch_reorder<true> : psf_batch_reorder<false>;
        kernel<<<(unsigned)blocks, ORDER_BLOCK, ORDER_SMEM, st>>>(groups, slots, prefix, n_slots, round);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "psf_batch_reorder launch");
    }
    return PSF_OK;
}

}  // namespace psf
