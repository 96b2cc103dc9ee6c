// Internal types of the batched engine (include/psf_batch.h), shared by the
// kernels (psf_batch.cu) and the C ABI implementation (psf_batch_api.cpp).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "psf_internal.h"

namespace psf {

constexpr int BATCH_MAX_GROUPS = 6;   // distinct bases in one batch
constexpr int BATCH_MAX_SLOTS = 256;  // instance slots per basis (one MMA N tile)
constexpr int BATCH_MAX_ALL_SLOTS = BATCH_MAX_GROUPS * BATCH_MAX_SLOTS;
constexpr int EPI_WARPS = 8;          // epilogue: two warps per TMEM lane quarter
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int GEMM_THREADS = 64 + EPI_THREADS;  // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int GEMM_MAX_KSPLIT = 4;

// One basis inside a GEMM launch: A operand (C or Phi) and B operand (the
// slots' coefficient vectors), both BF16 hi/lo pairs, K-major, 128-byte
// swizzled by TMA.
struct SlotDev;

struct alignas(64) GemmGroup {
    CUtensorMap tmA;        // 4D (k inner 64, rows 128, hi/lo 2, outer 1)
    CUtensorMap tmB;        // 3D (k inner 64, bn rows, hi/lo 2)
    int tiles;              // work units of this basis: 128-row tiles x K splits
    int m_inner;            // row tiles per outer index (contraction: a-tiles per mode k)
    int k_chunks;           // K / 64
    int ksplit;             // K ranges per row tile (each writes its own partial sums)
    int kc_per;             // K chunks per range
    int bn;                 // MMA N: slots rounded up to 16
    uint32_t tx_bytes;      // bytes one pipeline stage receives
    int cap;                // slots in use (columns)
    int n_rows;             // valid rows: N (contraction) or F_act (reconstruction)
    int ldw;                // row stride of w (= the basis' N)
    const float *wf;        // contraction: FP32 copy of the state [cap][ldw]
    double *dwpart;         // contraction: partials [k][nparts (a-tile, K range, warp)][slot]
    int nparts;             // contraction: partials per (slot, k)
    long long n_faces;
    const int32_t *field_dst;  // reconstruction: [n_rows][2] places of a face in a slot's field (-1: none)
    float *field;           // reconstruction: the slots' face fields, FaceField or PairField (psf_device.cuh)
    long long field_floats; // floats per slot in field
    const SlotDev *slot_of; // reconstruction: the group's slots (column b is slot_of[b]); fields are
                            // written only for slots that stepped (the tracer reads no others)
};

struct GroupDev;

// Arguments of one tensor-core launch: contraction units [0, c_tiles) over
// g[0 .. n_groups), reconstruction units over g[n_groups .. 2 n_groups).
// A fused launch (cooperative) runs the state update between the two.
struct StepArgs {
    GemmGroup g[2 * BATCH_MAX_GROUPS];
    int n_groups;
    int c_tiles;
    int r_tiles;
    int fused;
    int *err;                 // device error word (bounded waits)
    unsigned int *grid_bar;   // grid barrier counter, zeroed before each fused launch
    const GroupDev *groups;   // state update of a fused launch
    SlotDev *slots;
    int n_slots;
};

// SlotDev::stepped, else 0: the slot advanced, and with it a flow that carries most
// particles out of their half-cell in an RK4 step.
constexpr int STEPPED = 1, STEPPED_FAST = 2;

// Per-slot parameters and counters, in device memory.
struct SlotDev {
    int active;
    int n_modes;
    int rk4;
    int group;
    int slot;
    unsigned int flags;
    double dt;
    double visc_signed;
    float lifetime;
    float fast_above;         // |w|^2 above which the slot's flow is fast (FAST_STEP)
    unsigned long long seed;
    unsigned long long step;  // steps taken since the slot was set (device counter)
    long long n_particles;
    long long poff;           // first particle of the slot in the particle pool
    unsigned long long target;  // stop after this many steps (0: no limit)
    int stepped;              // STEPPED or STEPPED_FAST if the slot advanced in the current step (set by the state kernel)
    int mixed;                // round of launch_batch_reorder in which the slot was out of order
};

// Per-basis device view used by the state kernel and the tracer.
struct GroupDev {
    GridDev grid;
    int N, Nj, cap, bn, a_tiles, slot_base;
    int nparts;           // contraction partials per mode: a_tiles x ksplit x 4
    long long n_faces, pmax;
    double *w;            // [cap][N]
    float *wf;            // [cap][N] FP32 copy of w (contraction epilogue)
    double *force;        // [cap][N]
    const double *lam;    // [N]
    double *dwpart;       // see GemmGroup
    uint16_t *W;          // BF16 [2][bn][Nj]
    float *field;         // [cap][field_floats] face field of each slot
    long long field_floats;
    long long V;
    float4 *parts;        // particle pool (all slots of the batch)
    int32_t *perm;        // caller index of each pooled particle
};


// Launchers (psf_batch.cu).  `bn_max` selects the kernel variant (64, 128 or
// 256 MMA columns per accumulator); `grid` the number of persistent CTAs.
int batch_gemm_smem_bytes(int bn_max);
// `after_kernel`: the launch directly follows a kernel in the stream and may
// start during that kernel's tail (programmatic dependent launch).
int launch_batch_step_tc(const StepArgs &args, int bn_max, int grid, cudaStream_t st, bool after_kernel = false);
int max_fused_grid(int bn_max, int num_sms);
int launch_batch_state(const GroupDev *groups, SlotDev *slots, int n_slots, cudaStream_t st);
// prefix[s] = particles of slots 0..s-1 (occupied slots only); n_slots + 1 entries.
int launch_batch_trace(const GroupDev *groups, const SlotDev *slots, const long long *prefix, int n_slots, int grid,
                       bool all_centred, bool faces, cudaStream_t st);
// Put the particles of slots that go on stepping back in brick order where the
// flow has mixed them.  `round` differs from call to call; `total` is prefix[n_slots].
// prepare_batch_reorder loads the kernels on the current device, so that no step waits for it.
int prepare_batch_reorder();
int launch_batch_reorder(const GroupDev *groups, SlotDev *slots, const long long *prefix, int n_slots, long long total,
                         int round, cudaStream_t st);
// One slot of a grouped read-back: its state row, its particles in the pool and
// where both go in the staging buffers.
struct ReadJob {
    const double *w;
    long long poff, stage;  // first particle in the pool and in the staging buffer
    int n_w, w_at;          // state values (0: not wanted) and their place
    int n_parts;            // particles in this group of jobs (0: none)
};

// Gather the jobs' states into `w_out`, and their particles, in the caller's
// order, into `stage`.
int launch_batch_gather_states(const ReadJob *jobs, int n, double *w_out, cudaStream_t st);
int launch_batch_unorder(const ReadJob *jobs, int n, int max_parts, const float4 *pool, const int32_t *perm,
                         float4 *stage, cudaStream_t st);
int launch_batch_pack(const GroupDev *groups, const SlotDev *slots, int slot_global, cudaStream_t st);
int batch_trace_grid(int num_sms, bool faces);

// Host helpers.
int encode_tensor_map(CUtensorMap *map, void *base, int rank, const uint64_t *dims, const uint64_t *strides_bytes,
                      const uint32_t *box);
void split_bf16_host(double x, uint16_t *hi, uint16_t *lo);

}  // namespace psf

// Entry points of psf_batch_api.cpp used by the serving engine
// (psf_engine.cpp); not part of the C ABI.
struct psf_batch;
struct psf_instance_desc;
namespace psf {
// psf_batch_set_instances without the closing synchronisation: the copies,
// orderings and the priming contraction stay queued on the batch's stream.
// Host rows the copies read are kept until the next psf_batch_sync.
int batch_place_async(psf_batch *B, int32_t n, const int32_t *basis, const int32_t *slot,
                      const psf_instance_desc *const *inst, int32_t *status);
// Second stream and pinned buffers for batch_read_frozen (once, before use).
int batch_prepare_reads(psf_batch *B);
// State and caller-order particles of occupied slots that the work queued on
// the batch's stream does not step (their step target is reached), read on a
// second stream while that work runs.  The caller-order scatter runs on the
// host.
int batch_read_frozen(psf_batch *B, int32_t n, const int32_t *basis, const int32_t *slot, double *const *w,
                      float *const *xyzw);
}  // namespace psf
