// Particle density volume and its ray-marched image: the compute part of the
// reference's PSFSolverGPU::drawParticles (Solver/SolverImpl/psfsolvergpu.cpp:876-1022)
// as CUDA kernels writing device buffers, with no graphics API.
//
//   psf_vol_clear      zeroes what the last frame left (Texture3D::clearImage)
//   psf_vol_histogram  particle -> cell counts; a warp merges equal cells
//                      (__match_any_sync) before one atomic per distinct cell
//   psf_vol_density    counts / 1e6 -> FP16 density (volume.comp) in the counts'
//                      place, and one bit for every texel that is not zero
//   psf_vol_occupancy  one bit per trilinear cell: any of its 8 texels not zero
//   psf_vol_unpack     the density as res^3 FP16 values, for reading back
//   psf_vol_render     a lane carries one ray at a time: ray/AABB slab test,
//                      march with trilinear clamp-to-border samples, shadow ray
//                      toward the light, front-to-back emission/absorption
//                      (volume.frag); cells without density are stepped over
//
// A volume is one array of 4-byte words, R + 2 slices of R + 2 rows of R + 1
// words, and the bits.  Word c of the row of texels (y, z), row y + 1 of slice
// z + 1, holds the texels (c - 1, c) as two FP16 values; the outer rows and
// slices are the zero border.  While particles are counted, word c of that row
// holds the count of texel c.  So a sample of the march is four loads with no
// border tests, and a volume takes 4.3 bytes per texel (571 MB at R = 512; the
// counts and an FP16 array beside them would be 805 MB).
//
// The density (68 MB at R = 256) stays L2-resident while a frame is rendered.
// Arithmetic is round-to-nearest FP32 through explicit intrinsics
// in a fixed order (no contraction), so results equal a plain C restatement
// bit for bit.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <string>

#include "psf_device.cuh"
#include "psf_internal.h"
#include "psf_volume.h"

namespace {

constexpr float VOL_ZDIR = -1.792590986919304f;          // -1 / tan(45.0 / 2.0), radians as in volume.frag
constexpr float VOL_SHADOW_THRESH = 6.907755278982137f;  // -log(0.001) / 1.0

struct Box {
    float mn[3], mx[3], ext[3];
    int R;
};

struct View {
    float view[16];
    float cam[3], light[3];
    float mn[3], mx[3];
    int W, H, R;
};

// Words from a row to the next and from a slice to the next.
__host__ __device__ __forceinline__ uint32_t row_pitch(int R) { return (uint32_t)R + 1u; }
__host__ __device__ __forceinline__ uint32_t slice_pitch(int R) { return ((uint32_t)R + 1u) * ((uint32_t)R + 2u); }
// First word of the row of texels (y, z).
__host__ __device__ __forceinline__ uint32_t row_at(int R, uint32_t y, uint32_t z)
{
    return (z + 1u) * slice_pitch(R) + (y + 1u) * row_pitch(R);
}
uint32_t row_words_of(int R) { return (uint32_t)(R + 31) / 32; }       // bit words of a row of texels
uint32_t cell_words_of(int R) { return (uint32_t)(R + 1 + 31) / 32; }  // ... and of cells

// The kernels of a splat start during the tail of the one before (programmatic
// dependent launch): 11 us for all four at R = 64 with 1,000 particles.

// Zeroes the words that hold density: those of a texel with its bit set and of the
// texel after it.  A warp takes a row.
__global__ void __launch_bounds__(256) psf_vol_clear(uint32_t *__restrict__ words,
                                                     const uint32_t *__restrict__ texel_bits, int R, int row_words,
                                                     uint32_t *__restrict__ occupied)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *occupied = 0u;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    psf::launch_dependents();
    for (uint32_t row = warp; row < (uint32_t)R * (uint32_t)R; row += nwarps) {
        const uint32_t mine = lane < row_words ? texel_bits[(size_t)row * row_words + lane] : 0u;
        if (!__any_sync(0xffffffffu, mine != 0u)) continue;
        uint32_t *w = words + row_at(R, row % (uint32_t)R, row / (uint32_t)R);
        uint32_t carry = 0;
        for (int k = 0; k * 32 <= R; ++k) {
            const uint32_t m = k < row_words ? __shfl_sync(0xffffffffu, mine, k) : 0u;
            const uint32_t held = m | (m << 1) | carry;
            carry = m >> 31;
            const int c = k * 32 + lane;
            if (c <= R && ((held >> lane) & 1u)) w[c] = 0u;
        }
    }
}

// Grid-stride over groups of 32 particles so every lane takes part in the match.
__global__ void psf_vol_histogram(const float4 *__restrict__ p, long long n, Box b, int *__restrict__ words)
{
    psf::grid_dependency_wait();
    psf::launch_dependents();
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long base = warp * 32; base < n; base += nwarps * 32) {
        const long long i = base + lane;
        int key = -1;
        if (i < n) {
            const float4 q = p[i];
            const float c[3] = {q.x, q.y, q.z};
            uint32_t at[3];
            bool ok = true;
            for (int a = 0; a < 3; ++a) {
                const float t = __fdiv_rn(__fsub_rn(c[a], b.mn[a]), b.ext[a]);
                const float f = floorf(__fmul_rn(t, (float)b.R));
                if (!(f >= 0.0f) || f >= (float)b.R) ok = false;
                at[a] = ok ? (uint32_t)f : 0u;
            }
            if (ok) key = (int)(row_at(b.R, at[1], at[2]) + at[0]);
        }
        const unsigned same = __match_any_sync(0xffffffffu, key);
        if (key >= 0 && lane == __ffs(same) - 1) atomicAdd(words + key, __popc(same));
    }
}

// A warp takes a row of texels, four runs of 32 with their loads in flight.  A
// word is read and written by the same lane, so the density takes the place of
// the counts; words of empty cells are zero already and are not written.  Traffic
// bounds it: 4 B read per texel, and 4 B written here and in psf_vol_clear where
// there is density.  Splat of 2 M particles over 256^3 82 us, of 100,000 56 (with
// counts, FP16 array and pairs apart 103 and 62; counts and FP16 array 84 and 56).
__global__ void __launch_bounds__(256) psf_vol_density(uint32_t *__restrict__ words, uint32_t *__restrict__ texel_bits,
                                                       int R, int row_words)
{
    psf::grid_dependency_wait();
    psf::launch_dependents();
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t row = warp; row < (uint32_t)R * (uint32_t)R; row += nwarps) {
        uint32_t *w = words + row_at(R, row % (uint32_t)R, row / (uint32_t)R);
        uint32_t before = 0;
        for (int w0 = 0; w0 < row_words; w0 += 4) {
            uint32_t h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = (w0 + k) * 32 + lane;
                h[k] = x < R ? w[x] : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = (w0 + k) * 32 + lane;
                const uint32_t d =
                    h[k] ? (uint32_t)__half_as_ushort(__float2half_rn(__fdiv_rn((float)(int)h[k], 1000000.0f))) : 0u;
                const uint32_t up = __shfl_up_sync(0xffffffffu, d, 1);
                const uint32_t pair = (lane == 0 ? before : up) | (d << 16);
                before = __shfl_sync(0xffffffffu, d, 31);
                if (x < R && pair) w[x] = pair;
                if (x == R - 1 && d) w[R] = d;
                const uint32_t bits = __ballot_sync(0xffffffffu, d != 0u);
                if (lane == 0 && w0 + k < row_words) texel_bits[(size_t)row * row_words + w0 + k] = bits;
            }
        }
    }
}

// Cell c of an axis (0 .. R) interpolates between texels c - 1 and c; texels
// -1 and R are the border (zero).  One thread writes the 32 cells of a word.  The
// occupied cells are counted for the ray march.
__global__ void __launch_bounds__(256) psf_vol_occupancy(const uint32_t *__restrict__ texel_bits, int R,
                                                         uint32_t row_words, uint32_t cell_words, uint32_t words,
                                                         uint32_t *__restrict__ cell_bits,
                                                         uint32_t *__restrict__ occupied)
{
    psf::grid_dependency_wait();
    uint32_t cells = 0;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < words; t += gridDim.x * blockDim.x) {
        const uint32_t w = t % cell_words, row = t / cell_words;
        const int cy = (int)(row % (uint32_t)(R + 1)), cz = (int)(row / (uint32_t)(R + 1));
        uint32_t here = 0, before = 0;
        for (int z = max(cz - 1, 0); z <= min(cz, R - 1); ++z)
            for (int y = max(cy - 1, 0); y <= min(cy, R - 1); ++y) {
                const uint32_t *b = texel_bits + ((size_t)z * R + y) * row_words;
                if (w < row_words) here |= b[w];
                if (w > 0) before |= b[w - 1];
            }
        const uint32_t bits = here | (here << 1) | (before >> 31);
        cell_bits[t] = bits;
        cells += (uint32_t)__popc(bits);
    }
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    cells = __reduce_add_sync(0xffffffffu, cells);
    if ((threadIdx.x & 31) == 0 && cells) atomicAdd(&sum, cells);
    __syncthreads();
    if (threadIdx.x == 0 && sum) atomicAdd(occupied, sum);
}

// Texels of the slices from z0 on.
__global__ void __launch_bounds__(256) psf_vol_unpack(const uint32_t *__restrict__ words, int R, uint32_t z0,
                                                      uint32_t texels, uint16_t *__restrict__ out)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= texels) return;
    const uint32_t row = t / (uint32_t)R, x = t % (uint32_t)R;
    out[t] = (uint16_t)(words[row_at(R, row % (uint32_t)R, z0 + row / (uint32_t)R) + x] >> 16);
}

__device__ __forceinline__ float lerp1(float a, float b, float t)
{
    return __fadd_rn(__fmul_rn(__fsub_rn(1.0f, t), a), __fmul_rn(t, b));
}

// floor(u) + 1 for -2^22 < u < 2^22 without the conversion unit: adding
// 1.5 * 2^23 rounded down leaves the floor in the low mantissa bits.
constexpr float FLOOR_MAGIC = 12582912.0f;
__device__ __forceinline__ uint32_t floor_cell(float u, float &fl)
{
    const float m = __fadd_rd(u, FLOOR_MAGIC);
    fl = __fsub_rn(m, FLOOR_MAGIC);
    return __float_as_uint(m) - (0x4B400000u - 1u);
}

// Texel coordinate of a position; cell -1 .. R - 1 of it is inside the border.
__device__ __forceinline__ float texel_coord(float p, float Rf) { return __fsub_rn(__fmul_rn(p, Rf), 0.5f); }
__device__ __forceinline__ bool in_border(float u, float v, float w, float Rf)
{
    return u >= -1.0f && u < Rf && v >= -1.0f && v < Rf && w >= -1.0f && w < Rf;
}

// Trilinear clamp-to-border sample: four 4-byte loads with no border tests.
__device__ __forceinline__ float sample(const __half2 *__restrict__ pairs, int R, float px, float py, float pz)
{
    const float Rf = (float)R;
    const float u = texel_coord(px, Rf), v = texel_coord(py, Rf), w = texel_coord(pz, Rf);
    if (!in_border(u, v, w, Rf)) return 0.0f;
    float fu, fv, fw;
    const uint32_t ux = floor_cell(u, fu), uy = floor_cell(v, fv), uz = floor_cell(w, fw);
    const float a = __fsub_rn(u, fu), b = __fsub_rn(v, fv), c = __fsub_rn(w, fw);
    const uint32_t row = row_pitch(R), slice = slice_pitch(R);
    const __half2 *at = pairs + (uz * slice + uy * row + ux);
    const float2 t00 = __half22float2(__ldg(at)), t10 = __half22float2(__ldg(at + row));
    const float2 t01 = __half22float2(__ldg(at + slice)), t11 = __half22float2(__ldg(at + slice + row));
    const float c00 = lerp1(t00.x, t00.y, a), c10 = lerp1(t10.x, t10.y, a);
    const float c01 = lerp1(t01.x, t01.y, a), c11 = lerp1(t11.x, t11.y, a);
    const float c0 = lerp1(c00, c10, b), c1 = lerp1(c01, c11, b);
    return lerp1(c0, c1, c);
}

// exp(-y) for y in [0, 1]: Taylor series to degree 12, Horner form.
__device__ __forceinline__ float exp_neg_unit(float y)
{
    const float x = -y;
    float r = 1.0f;
#pragma unroll
    for (int k = 12; k >= 1; --k) r = __fadd_rn(1.0f, __fmul_rn(__fdiv_rn(x, (float)k), r));
    return r;
}

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ float len3(float x, float y, float z)
{
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

// A warp works through rays in rounds.  In the first phase of a round every
// lane marches its own ray and puts each sample that has density, as a query
// (position, opacity), into a pool of the warp in shared memory; a lane whose
// ray is done takes the next pixel from a counter.  The march needs no shadow
// ray: where it stops depends on the opacities alone.  In the second phase the
// lanes take the pool's queries one by one and walk their shadow rays, and in
// the third each lane composites its ray's queries in their order.  So the
// shadow rays, nearly all of the work, keep every lane busy however the
// queries fall on the rays, and one long ray's shadow rays are walked by 32
// lanes.  Before a trilinear sample a walk looks at the cell's occupancy bit:
// a cell without density adds exactly zero and is stepped over.  A shadow ray
// that has left the volume and moves away from it ends there: its remaining
// samples are zero.  Every ray's and shadow ray's own operations and their
// order are those of a plain loop over the pixel, so the image is
// bit-identical to that.
//
// Measured (1 x B200, device time of the launch): 262,144 particles spread
// over 256^3, 1280 x 720: 1.90 ms, against 21.6 ms for a thread per pixel with
// the shadow loop inside the march (about one sample in eight has density, so
// nearly every step some lane of a warp walked 128 shadow steps while the
// others waited) and 3.1 ms for a lane that switches between its march and its
// shadow ray (long rays then walk thousands of samples alone).  2 M particles,
// normal cloud: 1.55 against 11.6 ms; 100,000 in 128^3, 640 x 360: 3.2 against
// 22.7 ms.  It is bound by issue (16.8 M particles, normal cloud:
// 76 % of the slots, 20.5 lanes per instruction) with the occupancy words and
// pairs in L1 and L2.  One
// occupancy look-up at a time took 2.7 ms at the first size (its load latency
// stood between any two steps); POOL = 512 or 8 blocks per SM changed nothing.
constexpr int RENDER_THREADS = 128;
constexpr int REFILL = 8;       // idle lanes before a warp takes new pixels
constexpr int AHEAD = 4;        // positions whose occupancy is looked up together (below)
constexpr int SKIP = 4;         // look-ups per pass ...
constexpr int WALKERS = 16;     // ... or until so few lanes have not reached density
constexpr int HANDS = 4;        // turns the pixels of an image are dealt out in, at least
constexpr int HOLD_LEAST = 4;   // rays a warp holds, at least
constexpr int POOL = 256;       // queries of a round
constexpr float SPARSE = 1e-3f;       // share of occupied cells below which not one ray in four meets density
constexpr float FILLED = 0.9f;        // ... above which nearly every sample has density
constexpr float SHORT_SHADOW = 8.0f;  // samples of a shadow ray that cost little beside the march

struct RayConst {
    float vox, step;
    float lview[3], ext[3];
};

__device__ __forceinline__ void render_consts(const View &V, RayConst &k)
{
    for (int a = 0; a < 3; ++a) k.ext[a] = __fsub_rn(V.mx[a], V.mn[a]);
    k.vox = __fmul_rn(__fmul_rn(__fdiv_rn(k.ext[0], (float)V.R), __fdiv_rn(k.ext[1], (float)V.R)),
                      __fdiv_rn(k.ext[2], (float)V.R));
    k.step = __fdiv_rn(k.ext[0], 256.0f);
    for (int i = 0; i < 3; ++i)
        k.lview[i] =
            __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(V.view[i], V.light[0]), __fmul_rn(V.view[4 + i], V.light[1])),
                                __fmul_rn(V.view[8 + i], V.light[2])),
                      __fmul_rn(V.view[12 + i], 1.0f));
}

// Entry point, step vector and length of pixel (px, py)'s ray.
__device__ void ray_setup(const View &V, const RayConst &k, int px, int py, float (&pos)[3], float (&sv)[3], float &rl)
{
    float r0 = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, __fadd_rn((float)px, 0.5f)), (float)V.W), 1.0f);
    const float r1 = __fsub_rn(__fdiv_rn(__fmul_rn(2.0f, __fadd_rn((float)py, 0.5f)), (float)V.H), 1.0f);
    r0 = __fmul_rn(r0, __fdiv_rn((float)V.W, (float)V.H));
    const float r2 = VOL_ZDIR;
    float d[3];
    for (int j = 0; j < 3; ++j) {
        const float *col = V.view + 4 * j;
        d[j] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r0, col[0]), __fmul_rn(r1, col[1])), __fmul_rn(r2, col[2])),
                         __fmul_rn(0.0f, col[3]));
    }
    float tmin[3], tmax[3];
    for (int a = 0; a < 3; ++a) {
        const float inv = __fdiv_rn(1.0f, d[a]);
        const float tt = __fmul_rn(inv, __fsub_rn(V.mx[a], V.cam[a]));
        const float tb = __fmul_rn(inv, __fsub_rn(V.mn[a], V.cam[a]));
        tmin[a] = fminf(tt, tb);
        tmax[a] = fmaxf(tt, tb);
    }
    const float t0 = fmaxf(0.0f, fmaxf(fmaxf(tmin[0], tmin[1]), fmaxf(tmin[0], tmin[2])));
    const float t1 = fminf(fminf(tmax[0], tmax[1]), fminf(tmax[0], tmax[2]));
    float ray[3];
    for (int a = 0; a < 3; ++a) {
        const float s0 = __fdiv_rn(__fsub_rn(__fadd_rn(V.cam[a], __fmul_rn(d[a], t0)), V.mn[a]), k.ext[a]);
        const float s1 = __fdiv_rn(__fsub_rn(__fadd_rn(V.cam[a], __fmul_rn(d[a], t1)), V.mn[a]), k.ext[a]);
        pos[a] = s0;
        ray[a] = __fsub_rn(s1, s0);
    }
    rl = len3(ray[0], ray[1], ray[2]);
    for (int a = 0; a < 3; ++a) sv[a] = __fdiv_rn(__fmul_rn(k.step, ray[a]), rl);
}

// A walk through the volume: position, step vector, steps left.
struct Walk {
    float q[3], v[3];
    int n;
    bool near;  // the last sample had density
};

__device__ __forceinline__ void step_on(Walk &w)
{
    w.q[0] = __fadd_rn(w.q[0], w.v[0]);
    w.q[1] = __fadd_rn(w.q[1], w.v[1]);
    w.q[2] = __fadd_rn(w.q[2], w.v[2]);
    --w.n;
}

struct Cells {
    const uint32_t *__restrict__ bits;
    uint32_t words;  // per row
    int R;
    bool no_skip;  // a voxel volume that underflows: an empty sample is 0 / 0, not zero
    bool runs;     // a sample with density is mostly followed by another
    // Whether the warp's walks (this lane has one if `walking`) all take their next
    // sample without a look ahead: where the last samples of all of them had density
    // the look would be in vain (2 M particles in 64^3, 1280 x 720, inside: 8.7 against
    // 13.6 ms).  Lane by lane it would cost, as the other lanes' look-ups take the time
    // anyway (one sample in eight with density: 2.2 -> 2.65 ms).  It is tried where
    // most cells are occupied, and up to R = 32, where a walk takes eight steps or more
    // in a cell (500,000 in a cloud in 16^3, 1280 x 720: 11.5 against 14.9 ms); in finer
    // and sparser volumes it cost up to 5 %.
    __device__ __forceinline__ bool straight(bool walking, const Walk &w) const
    {
        return no_skip || (runs && __all_sync(0xffffffffu, !walking || w.near));
    }
};

// Looks at the walk's next AHEAD positions, whose occupancy loads are in
// flight together, and moves to the first one with density (true) or past
// them.  `ended`: the walk is over; MARCH walks also end with their length,
// others where the position is outside the volume and the step leads away
// from it.
template <bool MARCH>
__device__ __forceinline__ bool look_ahead(const Cells &c, Walk &w, float &left, float dec, bool &ended)
{
    const float Rf = (float)c.R;
    const uint32_t R1 = (uint32_t)c.R + 1u;
    float q[3] = {w.q[0], w.q[1], w.q[2]};
    uint32_t word[AHEAD], bit[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
        const float u = texel_coord(q[0], Rf), v = texel_coord(q[1], Rf), x = texel_coord(q[2], Rf);
        float f;
        const uint32_t cx = floor_cell(u, f), cy = floor_cell(v, f), cz = floor_cell(x, f);
        word[j] = in_border(u, v, x, Rf) ? __ldg(c.bits + ((cz * R1 + cy) * c.words + (cx >> 5))) : 0u;
        bit[j] = cx;
        if (!MARCH && j == AHEAD - 1)
            ended = (u < -1.0f && w.v[0] <= 0.0f) || (u >= Rf && w.v[0] >= 0.0f) || (v < -1.0f && w.v[1] <= 0.0f) ||
                    (v >= Rf && w.v[1] >= 0.0f) || (x < -1.0f && w.v[2] <= 0.0f) || (x >= Rf && w.v[2] >= 0.0f);
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = __fadd_rn(q[a], w.v[a]);
    }
    bool found = false, over = false;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
        if (!found && !over) {
            if ((word[j] >> (bit[j] & 31u)) & 1u) {
                found = true;
            } else {
                step_on(w);
                if (MARCH) left = __fsub_rn(left, dec);
                over = !(w.n > 0 && (!MARCH || left > 0.0f));
            }
        }
    }
    ended = !found && (over || (!MARCH && ended));
    return found;
}

__global__ void __launch_bounds__(RENDER_THREADS) psf_vol_render(const __half2 *__restrict__ pairs,
                                                                 const uint32_t *__restrict__ cell_bits,
                                                                 uint32_t cell_words, View V, uint32_t tiles_x,
                                                                 uint32_t n_items, int hold, int hold_filled,
                                                                 uint32_t *__restrict__ next,
                                                                 const uint32_t *__restrict__ occupied,
                                                                 float4 *__restrict__ out)
{
    constexpr int WARPS = RENDER_THREADS / 32;
    __shared__ float pool_x[WARPS][POOL], pool_y[WARPS][POOL], pool_z[WARPS][POOL], pool_dens[WARPS][POOL];
    __shared__ uint16_t pool_link[WARPS][POOL];  // the next query of the same ray
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *qx = pool_x[warp], *qy = pool_y[warp], *qz = pool_z[warp], *qd = pool_dens[warp];
    uint16_t *link = pool_link[warp];
    const unsigned below = (1u << lane) - 1u;
    const int R = V.R;
    RayConst k;
    render_consts(V, k);
    const float share = (float)__ldg(occupied) / (float)((R + 1) * (R + 1) * (R + 1));
    const Cells cells{cell_bits, cell_words, R, !(k.vox > 0.0f), share > 0.5f || R <= 32};
    hold = share < SPARSE ? 32 : share > FILLED ? hold_filled : hold;

    Walk ray;
    ray.n = 0;
    ray.near = false;
    float left = 0.0f, trans = 1.0f;                           // the march: length left, transmittance so far
    float le0 = 0.0f, le1 = 0.0f, le2 = 0.0f, shown = 1.0f;    // composited so far
    uint32_t pixel = 0;
    bool live = false, more = true;
    for (;;) {
        // ---- march
        int count = 0, head = -1, tail = -1;
        for (;;) {
            const unsigned idle = __ballot_sync(0xffffffffu, !live && head < 0);
            unsigned marching = __ballot_sync(0xffffffffu, live);
            const int take = min(hold - 32, 0) + __popc(idle);  // lanes that get a pixel: at most `hold` rays in hand
            if (more && (take >= min(REFILL, hold) || (marching == 0u && take > 0))) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(next, (uint32_t)take);
                base = __shfl_sync(0xffffffffu, base, 0);
                more = base < n_items;
                const int rank = __popc(idle & below);
                const uint32_t item = base + (uint32_t)rank;
                if (((idle >> lane) & 1u) && rank < take && item < n_items) {
                    // 8 x 4 pixel tiles
                    const uint32_t tile = item >> 5, in = item & 31u;
                    const int px = (int)((tile % tiles_x) * 8u + (in & 7u));
                    const int py = (int)((tile / tiles_x) * 4u + (in >> 3));
                    if (px < V.W && py < V.H) {
                        ray_setup(V, k, px, py, ray.q, ray.v, left);
                        ray.n = 1024;
                        ray.near = false;
                        pixel = (uint32_t)py * (uint32_t)V.W + (uint32_t)px;
                        trans = shown = 1.0f;
                        le0 = le1 = le2 = 0.0f;
                        live = left > 0.0f;
                        if (!live) out[pixel] = make_float4(le0, le1, le2, shown);
                    }
                }
                continue;
            }
            if (marching == 0u || count > POOL - 32 || (count >= POOL / 4 && __popc(marching) < REFILL)) break;
            bool ended = false, dense = cells.straight(live, ray) && live;
#pragma unroll 1
            for (int j = 0; j < SKIP; ++j) {
                if (live && !ended && !dense) dense = look_ahead<true>(cells, ray, left, k.step, ended);
                if (__popc(__ballot_sync(0xffffffffu, live && !dense && !ended)) <= WALKERS) break;
            }
            bool query = false;
            float dens = 0.0f, at[3] = {0.0f, 0.0f, 0.0f};
            if (dense) {
                const float d = sample(pairs, R, ray.q[0], ray.q[1], ray.q[2]), s = __fdiv_rn(d, k.vox);
                ray.near = d > 0.0f;
                query = s > 0.001f;
                if (query) {
                    for (int a = 0; a < 3; ++a) at[a] = ray.q[a];
                    dens = clampf(__fmul_rn(s, k.step), 0.0f, 1.0f);
                    trans = __fmul_rn(trans, __fsub_rn(1.0f, dens));
                    ended = trans < 0.01f;
                    trans = clampf(trans, 0.0f, 1.0f);
                }
                if (!ended) {
                    step_on(ray);
                    left = __fsub_rn(left, k.step);
                    ended = !(left > 0.0f && ray.n > 0);
                }
            }
            const unsigned asks = __ballot_sync(0xffffffffu, query);
            if (query) {
                const int i = count + __popc(asks & below);
                qx[i] = at[0];
                qy[i] = at[1];
                qz[i] = at[2];
                qd[i] = dens;
                if (head < 0)
                    head = i;
                else
                    link[tail] = (uint16_t)i;
                tail = i;
            }
            count += __popc(asks);
            if (live && ended) {
                live = false;
                if (head < 0) out[pixel] = make_float4(le0, le1, le2, shown);
            }
        }
        if (count == 0) {
            if (!more && !__any_sync(0xffffffffu, live)) return;
            continue;
        }
        __syncwarp();
        // ---- shadow rays: a query's light takes the place of its x
        {
            Walk sh;
            float sd = 0.0f;
            int mine = -1, taken = 0;
            for (;;) {
                const unsigned idle = __ballot_sync(0xffffffffu, mine < 0);
                if (taken < count) {
                    if (mine < 0) {
                        const int i = taken + __popc(idle & below);
                        if (i < count) {
                            mine = i;
                            sh.q[0] = qx[i];
                            sh.q[1] = qy[i];
                            sh.q[2] = qz[i];
                            const float lx = __fsub_rn(k.lview[0], sh.q[0]), ly = __fsub_rn(k.lview[1], sh.q[1]),
                                        lz = __fsub_rn(k.lview[2], sh.q[2]);
                            const float ll = len3(lx, ly, lz);
                            sh.v[0] = __fdiv_rn(__fmul_rn(k.step, lx), ll);
                            sh.v[1] = __fdiv_rn(__fmul_rn(k.step, ly), ll);
                            sh.v[2] = __fdiv_rn(__fmul_rn(k.step, lz), ll);
                            sd = 0.0f;
                            sh.n = 129;
                            sh.near = true;
                            step_on(sh);  // 128 samples left, the first one step away
                        }
                    }
                    taken += __popc(idle);
                } else if (idle == 0xffffffffu) {
                    break;
                }
                bool ended = false, dense = cells.straight(mine >= 0, sh) && mine >= 0;
#pragma unroll 1
                for (int j = 0; j < SKIP; ++j) {
                    if (mine >= 0 && !ended && !dense) dense = look_ahead<false>(cells, sh, sd, 0.0f, ended);
                    if (__popc(__ballot_sync(0xffffffffu, mine >= 0 && !dense && !ended)) <= WALKERS) break;
                }
                if (dense) {
                    const float d = sample(pairs, R, sh.q[0], sh.q[1], sh.q[2]);
                    sh.near = d > 0.0f;
                    sd = __fadd_rn(sd, __fdiv_rn(d, k.vox));
                    step_on(sh);
                    ended = sd > VOL_SHADOW_THRESH || sh.n == 0;
                }
                if (ended) {
                    qx[mine] = exp_neg_unit(clampf(__fmul_rn(sd, k.step), 0.0f, 1.0f));
                    mine = -1;
                }
            }
        }
        __syncwarp();
        // ---- composite, front to back
        for (int i = head; i >= 0; i = i == tail ? -1 : (int)link[i]) {
            const float e = qx[i], dens = qd[i];
            const float sh0 = __fmul_rn(1.0f, e), sh1 = __fmul_rn(0.5f, e), sh2 = __fmul_rn(0.0f, e);
            le0 = __fadd_rn(le0, __fmul_rn(__fmul_rn(sh0, dens), shown));
            le1 = __fadd_rn(le1, __fmul_rn(__fmul_rn(sh1, dens), shown));
            le2 = __fadd_rn(le2, __fmul_rn(__fmul_rn(sh2, dens), shown));
            shown = __fmul_rn(shown, __fsub_rn(1.0f, dens));
            if (!(shown < 0.01f)) {
                le0 = clampf(le0, 0.0f, 1.0f);
                le1 = clampf(le1, 0.0f, 1.0f);
                le2 = clampf(le2, 0.0f, 1.0f);
                shown = clampf(shown, 0.0f, 1.0f);
            }
        }
        if (head >= 0 && !live) out[pixel] = make_float4(le0, le1, le2, shown);
        __syncwarp();
    }
}

}  // namespace

struct psf_volume {
    int device = 0;
    int sms = 148;
    int R = 256;
    cudaStream_t stream = nullptr;  // own stream (host splats and renders)
    uint32_t *words = nullptr;      // counts, then pairs of texels; the rest follows in the same allocation
    uint32_t *texel_bits = nullptr, *cell_bits = nullptr;  // occupancy of texels and of trilinear cells
    uint32_t *next = nullptr;       // the ray march's pixel counter
    uint32_t *occupied = nullptr;   // cells with their bit set
    uint16_t *texels = nullptr;     // slices of the density on their way to the host
    int texel_slices = 1;
    int render_blocks = 148 * 4;
    float4 *parts = nullptr;        // host-splat staging
    long long parts_cap = 0;
    float4 *img = nullptr;
    long long img_cap = 0;
    // last host splat (its particles stay in `parts`), for profiling
    const float4 *last_parts = nullptr;
    long long last_n = -1;
    Box last_box{};
    float last_mean = 0.0f;         // density of the last splat's particles, had they filled the box evenly
    bool have_density = false;
};

namespace {

int cuda_status(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return PSF_OK;
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return psf::fail(PSF_ERR_NOMEM, std::string(what) + ": out of device memory");
    }
    return psf::cuda_fail(e, what);
}

int make_box(const float *mn, const float *mx, int R, Box *b)
{
    for (int a = 0; a < 3; ++a) {
        if (!std::isfinite(mn[a]) || !std::isfinite(mx[a]) || !(mx[a] > mn[a]))
            return psf::fail(PSF_ERR_INVALID, "the box must have max > min on every axis");
        b->mn[a] = mn[a];
        b->mx[a] = mx[a];
        b->ext[a] = mx[a] - mn[a];
    }
    b->R = R;
    return PSF_OK;
}

float mean_density(const Box &b, long long n)
{
    return (float)((double)n * 1e-6 / ((double)b.ext[0] * b.ext[1] * b.ext[2]));
}

int launch_splat(psf_volume *v, const float4 *parts, long long n, const Box &b, cudaStream_t st)
{
    const uint32_t row_words = row_words_of(v->R), cell_words = cell_words_of(v->R);
    const uint32_t rows = (uint32_t)v->R * (uint32_t)v->R;
    const unsigned grid = (unsigned)std::min<long long>((rows + 7) / 8, (long long)v->sms * 8);
    psf_vol_clear<<<grid, 256, 0, st>>>(v->words, v->texel_bits, v->R, (int)row_words, v->occupied);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && n > 0) {
        const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, (long long)v->sms * 8);
        psf::PdlLaunch L(blocks, 256, st, /*after_kernel=*/true);
        e = cudaLaunchKernelEx(&L.cfg, psf_vol_histogram, parts, n, b, reinterpret_cast<int *>(v->words));
    }
    if (e == cudaSuccess) {
        psf::PdlLaunch L(grid, 256, st, /*after_kernel=*/true);
        e = cudaLaunchKernelEx(&L.cfg, psf_vol_density, v->words, v->texel_bits, (int)v->R, (int)row_words);
    }
    if (e == cudaSuccess) {
        const uint32_t owords = (uint32_t)(v->R + 1) * (uint32_t)(v->R + 1) * cell_words;
        const unsigned blocks = std::min((owords + 255) / 256, (unsigned)v->sms * 8);
        psf::PdlLaunch L(blocks, 256, st, /*after_kernel=*/true);
        e = cudaLaunchKernelEx(&L.cfg, psf_vol_occupancy, (const uint32_t *)v->texel_bits, (int)v->R, row_words,
                               cell_words, owords, v->cell_bits, v->occupied);
    }
    return cuda_status(e, "volume splat launch");
}

int check_view(const psf_volume_view *view)
{
    if (!view) return psf::fail(PSF_ERR_INVALID, "null view");
    if (view->width < 1 || view->height < 1 || (long long)view->width * view->height > (1ll << 28))
        return psf::fail(PSF_ERR_INVALID, "image size must be positive and at most 2^28 pixels");
    return PSF_OK;
}

int launch_render(psf_volume *v, const psf_volume_view *view, cudaStream_t st)
{
    View V;
    std::memcpy(V.view, view->view, sizeof(V.view));
    for (int a = 0; a < 3; ++a) {
        V.cam[a] = view->camera[a];
        V.light[a] = view->light[a];
        V.mn[a] = v->last_box.mn[a];
        V.mx[a] = v->last_box.mx[a];
    }
    V.W = view->width;
    V.H = view->height;
    V.R = v->R;
    const uint32_t tiles_x = (uint32_t)(V.W + 7) / 8, tiles_y = (uint32_t)(V.H + 3) / 4;
    const long long items = 32ll * tiles_x * tiles_y;
    const cudaError_t e = cudaMemsetAsync(v->next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return cuda_status(e, "cudaMemsetAsync");
    // Rays a warp holds: few enough that the pixels are dealt out over HANDS
    // turns of every warp.  With 32 in every warp of a 640 x 360 image the
    // warps that got the cloud's core ended long after the others: 5.7 ms
    // against 3.2 ms; 16 turns left too few lanes marching (4.3 to 5.3 ms
    // against 2.8 ms at 1280 x 720).
    // Where the march is the work and not the shadow rays, that leaves lanes idle.
    // So a warp holds 32 rays where hardly a cell is occupied (no particles, 640 x
    // 360: 0.43 ms against 1.05; 1,000 in 512^3, 320 x 200: 0.24 against 0.87), and
    // its share of the pixels where nearly all are and the mean density ends a shadow
    // ray within SHORT_SHADOW samples (2 M in 64^3, 320 x 200, inside: 1.0 against 1.6
    // ms; with longer shadow rays the small hands are better, 100,000 in 64^3, from
    // outside: 4.0 against 10 ms).
    const long long warps = (long long)v->render_blocks * (RENDER_THREADS / 32);
    auto held = [](long long rays) { return (int)std::max<long long>(HOLD_LEAST, std::min<long long>(32, rays)); };
    const int hold = held(items / (warps * HANDS));
    const bool opaque = v->last_mean * SHORT_SHADOW > VOL_SHADOW_THRESH;
    const int hold_filled = opaque ? held(items / warps) : hold;
    // Blocks for all pixels at once, if the chip holds so many: a 64 x 48 image in
    // warps of four rays is done in one turn.
    const long long need = (items + RENDER_THREADS / 32 * hold - 1) / (RENDER_THREADS / 32 * hold);
    psf_vol_render<<<(unsigned)std::min<long long>(need, v->render_blocks), RENDER_THREADS, 0, st>>>(
        reinterpret_cast<const __half2 *>(v->words), v->cell_bits, cell_words_of(v->R), V, tiles_x, (uint32_t)items, hold,
        hold_filled, v->next, v->occupied, v->img);
    return cuda_status(cudaGetLastError(), "volume render launch");
}

int ensure_image(psf_volume *v, long long pixels)
{
    if (pixels <= v->img_cap) return PSF_OK;
    cudaStreamSynchronize(v->stream);
    cudaFree(v->img);
    v->img = nullptr;
    v->img_cap = 0;
    const cudaError_t e = cudaMalloc(&v->img, (size_t)pixels * sizeof(float4));
    if (e != cudaSuccess) return cuda_status(e, "cudaMalloc");
    v->img_cap = pixels;
    return PSF_OK;
}

}  // namespace

extern "C" {

int psf_volume_create(int device, int32_t res, psf_volume **out)
{
    if (!out) return psf::fail(PSF_ERR_INVALID, "null output");
    *out = nullptr;
    if (res < 2 || res > PSF_VOLUME_MAX_RES) return psf::fail(PSF_ERR_UNSUPPORTED, "res must be in [2, 512]");
    const cudaError_t es = cudaSetDevice(device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    auto *v = new (std::nothrow) psf_volume();
    if (!v) return psf::fail(PSF_ERR_NOMEM, "host allocation failed");
    v->device = device;
    v->R = res;
    cudaDeviceGetAttribute(&v->sms, cudaDevAttrMultiProcessorCount, device);
    cudaError_t e = cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking);
    const size_t words = (size_t)(res + 2) * slice_pitch(res);
    const size_t tw = (size_t)res * res * row_words_of(res), cw = (size_t)(res + 1) * (res + 1) * cell_words_of(res);
    // Half of the density at a time crosses to the host, or 16 MB.
    v->texel_slices = (int)std::max<size_t>(1, std::min<size_t>((res + 1) / 2, (8u << 20) / ((size_t)res * res)));
    const size_t staging = (size_t)v->texel_slices * res * res;
    if (e == cudaSuccess) e = cudaMalloc(&v->words, (words + tw + cw + 2) * sizeof(uint32_t) + staging * sizeof(uint16_t));
    if (e == cudaSuccess) {
        v->texel_bits = v->words + words;
        v->cell_bits = v->texel_bits + tw;
        v->next = v->cell_bits + cw;
        v->occupied = v->next + 1;
        v->texels = reinterpret_cast<uint16_t *>(v->occupied + 1);
        e = cudaMemsetAsync(v->words, 0, (words + tw + cw + 2) * sizeof(uint32_t), v->stream);
    }
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, psf_vol_render, RENDER_THREADS, 0);
    if (e == cudaSuccess) v->render_blocks = v->sms * std::max(1, per_sm);
    if (e == cudaSuccess) e = cudaStreamSynchronize(v->stream);
    if (e != cudaSuccess) {
        psf_volume_destroy(v);
        return cuda_status(e, "volume buffers");
    }
    *out = v;
    return PSF_OK;
}

int psf_volume_destroy(psf_volume *v)
{
    if (!v) return psf::fail(PSF_ERR_INVALID, "null volume");
    cudaSetDevice(v->device);
    if (v->stream) cudaStreamSynchronize(v->stream);
    cudaFree(v->words);
    cudaFree(v->parts);
    cudaFree(v->img);
    if (v->stream) cudaStreamDestroy(v->stream);
    delete v;
    return PSF_OK;
}

int psf_volume_splat(psf_volume *v, const float *particles, int64_t n, const float aabb_min[3],
                     const float aabb_max[3])
{
    if (!v || !aabb_min || !aabb_max || n < 0 || (n > 0 && !particles))
        return psf::fail(PSF_ERR_INVALID, "null argument or negative count");
    Box b;
    int rc = make_box(aabb_min, aabb_max, v->R, &b);
    if (rc != PSF_OK) return rc;
    const cudaError_t es = cudaSetDevice(v->device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    if (n > v->parts_cap) {
        cudaStreamSynchronize(v->stream);
        cudaFree(v->parts);
        v->parts = nullptr;
        v->parts_cap = 0;
        const cudaError_t e = cudaMalloc(&v->parts, (size_t)n * sizeof(float4));
        if (e != cudaSuccess) return cuda_status(e, "cudaMalloc");
        v->parts_cap = n;
    }
    if (n > 0) {
        const cudaError_t e = cudaMemcpyAsync(v->parts, particles, (size_t)n * sizeof(float4), cudaMemcpyHostToDevice,
                                              v->stream);
        if (e != cudaSuccess) return cuda_status(e, "cudaMemcpyAsync");
    }
    rc = launch_splat(v, v->parts, n, b, v->stream);
    if (rc != PSF_OK) return rc;
    const cudaError_t e = cudaStreamSynchronize(v->stream);
    if (e != cudaSuccess) return cuda_status(e, "volume splat");
    v->last_parts = v->parts;
    v->last_n = n;
    v->last_box = b;
    v->last_mean = mean_density(b, n);
    v->have_density = true;
    return PSF_OK;
}

int psf_volume_splat_context(psf_volume *v, psf_ctx *ctx)
{
    if (!v || !ctx) return psf::fail(PSF_ERR_INVALID, "null argument");
    psf::ContextParticles cp;
    int rc = psf::context_particles(ctx, &cp);
    if (rc != PSF_OK) return rc;
    if (cp.device != v->device) return psf::fail(PSF_ERR_INVALID, "the context lives on another device");
    if (cp.n > 0 && !cp.parts) return psf::fail(PSF_ERR_STATE, "the context has no particles");
    Box b;
    rc = make_box(cp.mn, cp.mx, v->R, &b);
    if (rc != PSF_OK) return rc;
    const cudaError_t es = cudaSetDevice(v->device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    // Runs on the context's stream, after its queued steps.
    rc = launch_splat(v, cp.parts, cp.n, b, cp.stream);
    if (rc != PSF_OK) return rc;
    const cudaError_t e = cudaStreamSynchronize(cp.stream);
    if (e != cudaSuccess) return cuda_status(e, "volume splat");
    // The context owns its particles; profiling needs a host splat.
    v->last_parts = nullptr;
    v->last_n = -1;
    v->last_box = b;
    v->last_mean = mean_density(b, cp.n);
    v->have_density = true;
    return PSF_OK;
}

int psf_volume_get_density(psf_volume *v, uint16_t *density, int64_t count)
{
    if (!v || !density) return psf::fail(PSF_ERR_INVALID, "null argument");
    const long long cells = (long long)v->R * v->R * v->R;
    if (count < cells) return psf::fail(PSF_ERR_INVALID, "output smaller than res^3");
    const cudaError_t es = cudaSetDevice(v->device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    const size_t slice = (size_t)v->R * v->R;
    cudaError_t e = cudaSuccess;
    for (int z = 0; z < v->R && e == cudaSuccess; z += v->texel_slices) {
        const uint32_t texels = (uint32_t)(slice * std::min(v->texel_slices, v->R - z));
        psf_vol_unpack<<<(texels + 255) / 256, 256, 0, v->stream>>>(v->words, v->R, (uint32_t)z, texels, v->texels);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(density + slice * z, v->texels, texels * sizeof(uint16_t), cudaMemcpyDeviceToHost, v->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(v->stream);
    return cuda_status(e, "density read-back");
}

int psf_volume_render(psf_volume *v, const psf_volume_view *view, float *rgba, int64_t count)
{
    if (!v || !rgba) return psf::fail(PSF_ERR_INVALID, "null argument");
    int rc = check_view(view);
    if (rc != PSF_OK) return rc;
    if (!v->have_density) return psf::fail(PSF_ERR_STATE, "no density yet: splat particles first");
    const long long pixels = (long long)view->width * view->height;
    if (count < 4 * pixels) return psf::fail(PSF_ERR_INVALID, "output smaller than width * height * 4");
    const cudaError_t es = cudaSetDevice(v->device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    if ((rc = ensure_image(v, pixels)) != PSF_OK) return rc;
    if ((rc = launch_render(v, view, v->stream)) != PSF_OK) return rc;
    cudaError_t e = cudaMemcpyAsync(rgba, v->img, (size_t)pixels * sizeof(float4), cudaMemcpyDeviceToHost, v->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(v->stream);
    return cuda_status(e, "image read-back");
}

int psf_volume_profile(psf_volume *v, const psf_volume_view *view, int32_t iters, double *splat_ms,
                       double *render_ms)
{
    if (!v || !splat_ms || !render_ms || iters < 1) return psf::fail(PSF_ERR_INVALID, "null argument or iters < 1");
    int rc = check_view(view);
    if (rc != PSF_OK) return rc;
    if (!v->have_density || v->last_n < 0)
        return psf::fail(PSF_ERR_STATE, "profiling re-splats the particles of the last psf_volume_splat");
    const cudaError_t es = cudaSetDevice(v->device);
    if (es != cudaSuccess) return psf::cuda_fail(es, "cudaSetDevice");
    if ((rc = ensure_image(v, (long long)view->width * view->height)) != PSF_OK) return rc;
    cudaEvent_t ev[3];
    for (int i = 0; i < 3; ++i) {
        const cudaError_t e = cudaEventCreate(&ev[i]);
        if (e != cudaSuccess) {
            for (int k = 0; k < i; ++k) cudaEventDestroy(ev[k]);
            return psf::cuda_fail(e, "cudaEventCreate");
        }
    }
    cudaStream_t st = v->stream;
    rc = launch_splat(v, v->last_parts, v->last_n, v->last_box, st);  // warm-up
    if (rc == PSF_OK) rc = launch_render(v, view, st);
    cudaEventRecord(ev[0], st);
    for (int k = 0; k < iters && rc == PSF_OK; ++k) rc = launch_splat(v, v->last_parts, v->last_n, v->last_box, st);
    cudaEventRecord(ev[1], st);
    for (int k = 0; k < iters && rc == PSF_OK; ++k) rc = launch_render(v, view, st);
    cudaEventRecord(ev[2], st);
    const cudaError_t e = cudaEventSynchronize(ev[2]);
    if (rc == PSF_OK && e != cudaSuccess) rc = psf::cuda_fail(e, "cudaEventSynchronize");
    if (rc == PSF_OK) {
        float a = 0.0f, b = 0.0f;
        cudaEventElapsedTime(&a, ev[0], ev[1]);
        cudaEventElapsedTime(&b, ev[1], ev[2]);
        *splat_ms = (double)a / iters;
        *render_ms = (double)b / iters;
    }
    for (int i = 0; i < 3; ++i) cudaEventDestroy(ev[i]);
    return rc;
}

}  // extern "C"
