// Device helpers shared by the single-instance and the batched kernels:
// reference face numbering, the staggered trilinear interpolant, one
// particle step, the respawn generator and FP64 reductions.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "psf_b200.h"
#include "psf_internal.h"

namespace psf {

// --------------------------------------------- programmatic dependent launch
// The kernels of a step run back to back in one stream (or one branch of a
// graph).  Each one touches only constant data (C, Phi, face maps, prefix
// sums) before griddepcontrol.wait, and lets its own dependents launch only
// after that wait: at most two kernels are in flight, and the second never
// reads what the first is still writing.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Launch configuration of a kernel that may start while the previous kernel in
// the stream finishes (programmatic stream serialisation), if `after_kernel`.
struct PdlLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    PdlLaunch(unsigned grid, unsigned block, cudaStream_t st, bool after_kernel, size_t smem = 0)
    {
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(block);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = after_kernel ? 1 : 0;
    }
};

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }
// glm::mix(x, y, a) = x (1 - a) + y a, evaluated as x + a (y - x) (one FMA).
__device__ __forceinline__ float mixf(float x, float y, float a) { return fmaf(a, y - x, x); }

// Counter-based generator for respawns (SplitMix64 output function); the
// oracle uses the same function so respawns are reproducible.
__host__ __device__ __forceinline__ uint32_t respawn_hash(uint64_t seed, uint64_t step, uint32_t idx,
                                                          uint32_t k)
{
    uint64_t x = seed ^ (step * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)idx << 32) ^
                 ((uint64_t)k * 0xD1B54A32D192ED03ull);
    x ^= x >> 30;
    x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27;
    x *= 0x94D049BB133111EBull;
    x ^= x >> 31;
    return (uint32_t)(x >> 32);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block sum over 256 threads; result valid in every thread.
__device__ inline double block_sum_256(double v, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i];
    return t;
}

// ------------------------------------------------------------------ tracing
// The tracer reads the face field through a per-voxel copy ("face pairs"):
// for voxel v, pairs[v] = (u of its x-face at x, at x+1), pairs[V + v] the
// same for y, pairs[2V + v] for z, already carrying the tracer's face signs.
// One trilinear component then needs four aligned float2 loads instead of
// eight scalar gathers.  The interpolant is the reference's
// (psfsolver.cpp:80-212): clamped staggered cell indices, eight face samples
// per component mixed along y, then x, then z, weights not clamped.
__device__ __forceinline__ uint32_t voxel(const GridDev &g, int x, int y, int z)
{
    return (uint32_t)z * (uint32_t)(g.nx * g.ny) + (uint32_t)(y * g.nx + x);
}

// Staggered cell of a position.  Every index the three component stencils
// use derives from k = floor(2 * gi) per axis (gi = the reference's index
// coordinate): floor(gi) = k >> 1 and floor(gi - 1/2) = (k - 1) >> 1, the
// latter exact because gi - 1/2 is exact in FP32 wherever the clamp to the
// grid does not decide the index anyway.  Two positions share a cell when
// their k, clamped to [-1, 2n], agree: the key packs those.
__device__ __forceinline__ unsigned long long cell_key(const GridDev &g, float px, float py, float pz, int &kx,
                                                       int &ky, int &kz)
{
    const float gix = (g.shift[0] + px) * g.inv_h;
    const float giy = (g.shift[1] + py) * g.inv_h;
    const float giz = (g.shift[2] + pz) * g.inv_h;
    kx = clampi(__float2int_rd(2.0f * gix), -1, 2 * g.nx);
    ky = clampi(__float2int_rd(2.0f * giy), -1, 2 * g.ny);
    kz = clampi(__float2int_rd(2.0f * giz), -1, 2 * g.nz);
    return (unsigned long long)(uint32_t)(kx + 1) | ((unsigned long long)(uint32_t)(ky + 1) << 21) |
           ((unsigned long long)(uint32_t)(kz + 1) << 42);
}

// The gathered cell: stencil origins as floats and the 24 face samples as 12
// face pairs, each second sample of a lerp stored as its difference to the
// first (mixf(x, y, t) = fma(t, y - x, x) then costs one FMA).
struct CellCache {
    int kx, ky, kz;        // the cell: floor(2 gi) per axis, clamped to [-1, 2n]
    float oxO, oyO, ozO;   // xO, yO, zO
    float oxM, oyM, ozM;   // xM + 1/2, yM + 1/2, zM + 1/2
    float2 x00, dx10, x01, dx11;  // x faces at (xO, yM|yP, zM|zP), differences along y
    float2 yM0, yP0, yM1, yP1;    // y face pairs at (xM|xP, yO, zM|zP), .y = difference along y
    float2 zMM, dzMP, zPM, dzPP;  // z faces at (xM|xP, yM|yP, zO), differences along y
};

__device__ __forceinline__ void gather_cell(const GridDev &g, const float2 *__restrict__ pairs, int kx, int ky,
                                            int kz, CellCache &c)
{
    const int xO = clampi(kx >> 1, 0, g.nx - 1), yO = clampi(ky >> 1, 0, g.ny - 1), zO = clampi(kz >> 1, 0, g.nz - 1);
    const int xr = (kx - 1) >> 1, yr = (ky - 1) >> 1, zr = (kz - 1) >> 1;
    const int xM = clampi(xr, 0, g.nx - 1), xP = clampi(xr + 1, 0, g.nx - 1);
    const int yM = clampi(yr, 0, g.ny - 1), yP = clampi(yr + 1, 0, g.ny - 1);
    const int zM = clampi(zr, 0, g.nz - 1), zP = clampi(zr + 1, 0, g.nz - 1);
    c.oxO = (float)xO;
    c.oyO = (float)yO;
    c.ozO = (float)zO;
    c.oxM = (float)xM + 0.5f;
    c.oyM = (float)yM + 0.5f;
    c.ozM = (float)zM + 0.5f;
    const uint32_t V = (uint32_t)g.nx * (uint32_t)g.ny * (uint32_t)g.nz;
    const float2 *__restrict__ pxp = pairs;
    const float2 *__restrict__ pyp = pairs + V;
    const float2 *__restrict__ pzp = pairs + 2 * (size_t)V;
    const float2 x00 = __ldg(pxp + voxel(g, xO, yM, zM));
    const float2 x10 = __ldg(pxp + voxel(g, xO, yP, zM));
    const float2 x01 = __ldg(pxp + voxel(g, xO, yM, zP));
    const float2 x11 = __ldg(pxp + voxel(g, xO, yP, zP));
    const float2 yM0 = __ldg(pyp + voxel(g, xM, yO, zM));
    const float2 yP0 = __ldg(pyp + voxel(g, xP, yO, zM));
    const float2 yM1 = __ldg(pyp + voxel(g, xM, yO, zP));
    const float2 yP1 = __ldg(pyp + voxel(g, xP, yO, zP));
    const float2 zMM = __ldg(pzp + voxel(g, xM, yM, zO));
    const float2 zMP = __ldg(pzp + voxel(g, xM, yP, zO));
    const float2 zPM = __ldg(pzp + voxel(g, xP, yM, zO));
    const float2 zPP = __ldg(pzp + voxel(g, xP, yP, zO));
    c.x00 = x00;
    c.dx10 = make_float2(x10.x - x00.x, x10.y - x00.y);
    c.x01 = x01;
    c.dx11 = make_float2(x11.x - x01.x, x11.y - x01.y);
    c.yM0 = make_float2(yM0.x, yM0.y - yM0.x);
    c.yP0 = make_float2(yP0.x, yP0.y - yP0.x);
    c.yM1 = make_float2(yM1.x, yM1.y - yM1.x);
    c.yP1 = make_float2(yP1.x, yP1.y - yP1.x);
    c.zMM = zMM;
    c.dzMP = make_float2(zMP.x - zMM.x, zMP.y - zMM.y);
    c.zPM = zPM;
    c.dzPP = make_float2(zPP.x - zPM.x, zPP.y - zPM.y);
}

__device__ __forceinline__ float3 interpolate(const CellCache &c, const float3 &gw)
{
    float3 v;
    {  // x: faces (xO | xO+1, yM | yP, zM | zP)
        const float tx = gw.x - c.oxO, ty = gw.y - c.oyM, tz = gw.z - c.ozM;
        const float a = fmaf(ty, c.dx10.x, c.x00.x);
        const float b = fmaf(ty, c.dx10.y, c.x00.y);
        const float cc = fmaf(ty, c.dx11.x, c.x01.x);
        const float d = fmaf(ty, c.dx11.y, c.x01.y);
        v.x = mixf(mixf(a, b, tx), mixf(cc, d, tx), tz);
    }
    {  // y: faces (xM | xP, yO | yO+1, zM | zP)
        const float tx = gw.x - c.oxM, ty = gw.y - c.oyO, tz = gw.z - c.ozM;
        const float a = fmaf(ty, c.yM0.y, c.yM0.x);
        const float b = fmaf(ty, c.yP0.y, c.yP0.x);
        const float cc = fmaf(ty, c.yM1.y, c.yM1.x);
        const float d = fmaf(ty, c.yP1.y, c.yP1.x);
        v.y = mixf(mixf(a, b, tx), mixf(cc, d, tx), tz);
    }
    {  // z: faces (xM | xP, yM | yP, zO | zO+1)
        const float tx = gw.x - c.oxM, ty = gw.y - c.oyM, tz = gw.z - c.ozO;
        const float a = fmaf(ty, c.dzMP.x, c.zMM.x);
        const float b = fmaf(ty, c.dzPP.x, c.zPM.x);
        const float cc = fmaf(ty, c.dzMP.y, c.zMM.y);
        const float d = fmaf(ty, c.dzPP.y, c.zPM.y);
        v.z = mixf(mixf(a, b, tx), mixf(cc, d, tx), tz);
    }
    return v;
}

// Velocity at a position of a box whose index and weight coordinates differ;
// `c` carries the last gathered cell, and the samples are loaded again only
// when the position lies in another cell.
struct AnyBox {
    using Ptr = const float2 *__restrict__;
    CellCache c;
    bool have = false;
    __device__ __forceinline__ float3 velocity(const GridDev &g, const float2 *__restrict__ pairs, float px, float py,
                                               float pz)
    {
        int kx, ky, kz;
        cell_key(g, px, py, pz, kx, ky, kz);
        if (!have || kx != c.kx || ky != c.ky || kz != c.kz) {
            c.kx = kx;
            c.ky = ky;
            c.kz = kz;
            gather_cell(g, pairs, kx, ky, kz, c);
            have = true;
        }
        return interpolate(c, make_float3((px - g.mn[0]) * g.inv_h, (py - g.mn[1]) * g.inv_h,
                                          (pz - g.mn[2]) * g.inv_h));
    }
};

// The two forms of a face field and the two faces of voxel (x, y, z) along an
// axis, with the tracer's signs.  PairField holds them side by side, every
// face twice: one load.  FaceField is the reference's face numbering, every
// face once: two loads, half the memory.
struct PairField {
    using Ptr = const float2 *__restrict__;
    Ptr px, py, pz;
    uint32_t nx, nxy;
    __device__ __forceinline__ PairField(const GridDev &g, Ptr p) : px(p), nx((uint32_t)g.nx)
    {
        nxy = nx * (uint32_t)g.ny;
        py = p + nxy * (uint32_t)g.nz;
        pz = p + 2 * (size_t)(nxy * (uint32_t)g.nz);
    }
    __device__ __forceinline__ float2 x(uint32_t i, uint32_t j, uint32_t k) const { return __ldg(px + (k * nxy + j * nx + i)); }
    __device__ __forceinline__ float2 y(uint32_t i, uint32_t j, uint32_t k) const { return __ldg(py + (k * nxy + j * nx + i)); }
    __device__ __forceinline__ float2 z(uint32_t i, uint32_t j, uint32_t k) const { return __ldg(pz + (k * nxy + j * nx + i)); }
};

struct FaceField {
    using Ptr = const float *__restrict__;
    Ptr px, py, pz;
    uint32_t nx, ny, nxy;
    __device__ __forceinline__ FaceField(const GridDev &g, Ptr u)
        : px(u + g.xoff), py(u + g.yoff), pz(u), nx((uint32_t)g.nx), ny((uint32_t)g.ny), nxy((uint32_t)(g.nx * g.ny))
    {
    }
    __device__ __forceinline__ float2 x(uint32_t i, uint32_t j, uint32_t k) const
    {
        const uint32_t f = (k * ny + j) * (nx + 1) + i;
        return make_float2(__ldg(px + f), __ldg(px + f + 1));
    }
    __device__ __forceinline__ float2 y(uint32_t i, uint32_t j, uint32_t k) const
    {
        const uint32_t f = k * (nxy + nx) + j * nx + i;
        return make_float2(__ldg(py + f), __ldg(py + f + nx));
    }
    __device__ __forceinline__ float2 z(uint32_t i, uint32_t j, uint32_t k) const
    {
        const uint32_t f = k * nxy + j * nx + i;
        return make_float2(__ldg(pz + f), __ldg(pz + f + nxy));
    }
};

// One staggered component in a half-cell: its value and its y, x and xy
// differences on the two z planes of its stencil.
struct Trilinear {
    float v0, dy0, dx0, dxy0, v1, dy1, dx1, dxy1;
    __device__ __forceinline__ float at(float tx, float ty, float tz) const
    {
        const float a = fmaf(tx, fmaf(ty, dxy0, dx0), fmaf(ty, dy0, v0));
        const float b = fmaf(tx, fmaf(ty, dxy1, dx1), fmaf(ty, dy1, v1));
        return mixf(a, b, tz);
    }
};

// The same on a centred box (shift == -mn exactly, as for every domain built
// here), where the reference's index coordinate (shift + p) / h and the weight
// coordinate (p - mn) / h are the same number.  A half-cell is k = floor(2 gw)
// per axis; in it the coordinate from the whole-cell origin (own axis of a
// component) and the one from the half-shifted origin (other axes) differ by
// 1/2 either way, and the smaller of them is the place in the half-cell.  So
// a position lies in the gathered half-cell when that minimum is in [0, 1/2]
// (an unsigned compare of the bits; the interpolant is continuous, so either
// side may take a shared boundary), and the two coordinates are all the
// interpolation needs.  In the lowest half-cell the half-shifted stencil has
// one sample on both sides, so its coordinate does not matter there and keeps
// the unclamped origin.
//
// Bound by the latency and L1 lookups of the gathers (RK1, which has one per
// particle and little else, takes 70 us where RK4 takes 96 on 16 x 262,144
// particles of the 32^3 box with a sphere).  Measured with particles in Morton
// order, against three cell keys and nested lerps: 102 against 111 us at 0.001
// voxel per step, 129 against 133 us at 0.03; 513 x 16,384 on three domains: 284
// against 297 us.  Storing the pairs in bricks of 4 x 2 x 2 voxels made RK1 73
// instead of 80 us but RK4 139 instead of 129 (the places cost more in the
// repeated gathers) and the 512-slot reconstruction 353 instead of 302.
template <class Field>
struct CentredBox {
    using Ptr = typename Field::Ptr;
    float ox, oy, oz;     // whole-cell origin
    float sx, sy, sz;     // half-shifted origin
    Trilinear x, y, z;
    bool have = false;

    __device__ __forceinline__ void gather(const GridDev &g, typename Field::Ptr u, float qx, float qy, float qz)
    {
        const int kx = clampi(__float2int_rd(2.0f * (qx * g.inv_h)), 0, 2 * g.nx - 1);
        const int ky = clampi(__float2int_rd(2.0f * (qy * g.inv_h)), 0, 2 * g.ny - 1);
        const int kz = clampi(__float2int_rd(2.0f * (qz * g.inv_h)), 0, 2 * g.nz - 1);
        const int xO = kx >> 1, yO = ky >> 1, zO = kz >> 1;
        const int xr = (kx - 1) >> 1, yr = (ky - 1) >> 1, zr = (kz - 1) >> 1;
        ox = (float)xO;
        oy = (float)yO;
        oz = (float)zO;
        sx = (float)xr + 0.5f;
        sy = (float)yr + 0.5f;
        sz = (float)zr + 0.5f;
        const uint32_t xM = (uint32_t)max(xr, 0), xP = (uint32_t)min(xr + 1, g.nx - 1);
        const uint32_t yM = (uint32_t)max(yr, 0), yP = (uint32_t)min(yr + 1, g.ny - 1);
        const uint32_t zM = (uint32_t)max(zr, 0), zP = (uint32_t)min(zr + 1, g.nz - 1);
        const Field f(g, u);
        const float2 x00 = f.x(xO, yM, zM), x10 = f.x(xO, yP, zM), x01 = f.x(xO, yM, zP), x11 = f.x(xO, yP, zP);
        const float2 y00 = f.y(xM, yO, zM), y10 = f.y(xP, yO, zM), y01 = f.y(xM, yO, zP), y11 = f.y(xP, yO, zP);
        const float2 z00 = f.z(xM, yM, zO), z01 = f.z(xM, yP, zO), z10 = f.z(xP, yM, zO), z11 = f.z(xP, yP, zO);
        auto plane = [](float v, float vy, float vx, float vxy, float &o, float &dy, float &dx, float &dxy) {
            o = v;
            dy = vy - v;
            dx = vx - v;
            dxy = (vxy - vx) - dy;
        };
        plane(x00.x, x10.x, x00.y, x10.y, x.v0, x.dy0, x.dx0, x.dxy0);
        plane(x01.x, x11.x, x01.y, x11.y, x.v1, x.dy1, x.dx1, x.dxy1);
        plane(y00.x, y00.y, y10.x, y10.y, y.v0, y.dy0, y.dx0, y.dxy0);
        plane(y01.x, y01.y, y11.x, y11.y, y.v1, y.dy1, y.dx1, y.dxy1);
        plane(z00.x, z01.x, z10.x, z11.x, z.v0, z.dy0, z.dx0, z.dxy0);
        plane(z00.y, z01.y, z10.y, z11.y, z.v1, z.dy1, z.dx1, z.dxy1);
    }

    __device__ __forceinline__ static bool inside(float a, float b)
    {
        return __float_as_uint(fminf(a, b)) <= 0x3F000000u;  // [0, 1/2]
    }

    // Velocity at a position that lies in the gathered half-cell; false where it
    // does not.
    __device__ __forceinline__ bool velocity_inside(const GridDev &g, float px, float py, float pz, float3 &v) const
    {
        const float qx = px - g.mn[0], qy = py - g.mn[1], qz = pz - g.mn[2];
        const float ax = fmaf(qx, g.inv_h, -ox), ay = fmaf(qy, g.inv_h, -oy), az = fmaf(qz, g.inv_h, -oz);
        const float bx = fmaf(qx, g.inv_h, -sx), by = fmaf(qy, g.inv_h, -sy), bz = fmaf(qz, g.inv_h, -sz);
        v = make_float3(x.at(ax, by, bz), y.at(bx, ay, bz), z.at(bx, by, az));
        return inside(ax, bx) && inside(ay, by) && inside(az, bz);
    }

    __device__ __forceinline__ float3 velocity(const GridDev &g, typename Field::Ptr u, float px, float py, float pz)
    {
        const float qx = px - g.mn[0], qy = py - g.mn[1], qz = pz - g.mn[2];
        if (!have) {
            gather(g, u, qx, qy, qz);
            have = true;
        } else {
            const bool same = inside(fmaf(qx, g.inv_h, -ox), fmaf(qx, g.inv_h, -sx)) &&
                              inside(fmaf(qy, g.inv_h, -oy), fmaf(qy, g.inv_h, -sy)) &&
                              inside(fmaf(qz, g.inv_h, -oz), fmaf(qz, g.inv_h, -sz));
            if (!same) gather(g, u, qx, qy, qz);
        }
        const float ax = fmaf(qx, g.inv_h, -ox), ay = fmaf(qy, g.inv_h, -oy), az = fmaf(qz, g.inv_h, -oz);
        const float bx = fmaf(qx, g.inv_h, -sx), by = fmaf(qy, g.inv_h, -sy), bz = fmaf(qz, g.inv_h, -sz);
        return make_float3(x.at(ax, by, bz), y.at(bx, ay, bz), z.at(bx, by, az));
    }
};

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

// x / 6 for the RK4 average: the product with r = RN(1/6) and one residual
// correction by FMA (Markstein's correction step; for a constant divisor see
// Brisebarre and Muller, "Correctly rounded multiplication by arbitrary
// precision constants", 2008).  An exhaustive check over all floats finds it
// equal to the correctly rounded quotient for every |x| >= 2^-120; below
// that the residual underflows and the result may differ in the last place,
// which moves no position (|dt x / 6| is then far below an ulp of any
// coordinate but the smallest).
__device__ __forceinline__ float div6(float x)
{
    const float r = 1.0f / 6.0f;
    const float q = x * r;
    return fmaf(fmaf(-q, 6.0f, x), r, q);
}

// A particle's step whose stages all stay in its first half-cell: the same
// operations as advance_particle, with one gather and no other path.  False
// (and p as it was) where a stage leaves it or the particle's life is over.
template <class Field>
__device__ __forceinline__ bool advance_inside(float4 &p, const GridDev &g, typename Field::Ptr u,
                                               const TraceParams &tp)
{
    if (!(p.w > 0.f)) return false;
    const float dt = tp.dt;
    CentredBox<Field> box;
    float3 v = box.velocity(g, u, p.x, p.y, p.z);
    bool stays = true;
    if (tp.rk4) {
        const float3 k1 = v;
        float3 k2, k3, k4;
        stays = box.velocity_inside(g, clampf(p.x + 0.5f * dt * k1.x, g.mn[0], g.mx[0]),
                                    clampf(p.y + 0.5f * dt * k1.y, g.mn[1], g.mx[1]),
                                    clampf(p.z + 0.5f * dt * k1.z, g.mn[2], g.mx[2]), k2);
        stays &= box.velocity_inside(g, clampf(p.x + 0.5f * dt * k2.x, g.mn[0], g.mx[0]),
                                     clampf(p.y + 0.5f * dt * k2.y, g.mn[1], g.mx[1]),
                                     clampf(p.z + 0.5f * dt * k2.z, g.mn[2], g.mx[2]), k3);
        stays &= box.velocity_inside(g, clampf(p.x + dt * k3.x, g.mn[0], g.mx[0]),
                                     clampf(p.y + dt * k3.y, g.mn[1], g.mx[1]),
                                     clampf(p.z + dt * k3.z, g.mn[2], g.mx[2]), k4);
        v.x = div6(k1.x + 2.f * k2.x + 2.f * k3.x + k4.x);
        v.y = div6(k1.y + 2.f * k2.y + 2.f * k3.y + k4.y);
        v.z = div6(k1.z + 2.f * k2.z + 2.f * k3.z + k4.z);
    }
    if (!stays) return false;
    p.x = clampf(p.x + dt * v.x, g.mn[0], g.mx[0]);
    p.y = clampf(p.y + dt * v.y, g.mn[1], g.mx[1]);
    p.z = clampf(p.z + dt * v.z, g.mn[2], g.mx[2]);
    p.w = p.w - 1.f;
    return true;
}

// One particle step (psfsolver.cpp:75-224): RK1 or RK4 with the box clamp
// on every stage, lifetime decrement, and respawn from the counter-based
// generator keyed by the caller-order index `perm[idx]` when the lifetime ran
// out (read only then).  `step` is the index of the step being taken (0 for
// the first).
template <class Box, class Ptr>
__device__ __forceinline__ float4 advance_particle(float4 p, const GridDev &g, Ptr u,
                                                   const TraceParams &tp, uint64_t step,
                                                   const int32_t *__restrict__ perm, size_t idx)
{
    if (p.w > 0.f) {
        const float dt = tp.dt;
        Box box;
        float3 v;
        if (tp.rk4) {
            const float3 k1 = box.velocity(g, u, p.x, p.y, p.z);
            float qx = clampf(p.x + 0.5f * dt * k1.x, g.mn[0], g.mx[0]);
            float qy = clampf(p.y + 0.5f * dt * k1.y, g.mn[1], g.mx[1]);
            float qz = clampf(p.z + 0.5f * dt * k1.z, g.mn[2], g.mx[2]);
            const float3 k2 = box.velocity(g, u, qx, qy, qz);
            qx = clampf(p.x + 0.5f * dt * k2.x, g.mn[0], g.mx[0]);
            qy = clampf(p.y + 0.5f * dt * k2.y, g.mn[1], g.mx[1]);
            qz = clampf(p.z + 0.5f * dt * k2.z, g.mn[2], g.mx[2]);
            const float3 k3 = box.velocity(g, u, qx, qy, qz);
            qx = clampf(p.x + dt * k3.x, g.mn[0], g.mx[0]);
            qy = clampf(p.y + dt * k3.y, g.mn[1], g.mx[1]);
            qz = clampf(p.z + dt * k3.z, g.mn[2], g.mx[2]);
            const float3 k4 = box.velocity(g, u, qx, qy, qz);
            v.x = div6(k1.x + 2.f * k2.x + 2.f * k3.x + k4.x);
            v.y = div6(k1.y + 2.f * k2.y + 2.f * k3.y + k4.y);
            v.z = div6(k1.z + 2.f * k2.z + 2.f * k3.z + k4.z);
        } else {
            v = box.velocity(g, u, p.x, p.y, p.z);
        }
        p.x = clampf(p.x + dt * v.x, g.mn[0], g.mx[0]);
        p.y = clampf(p.y + dt * v.y, g.mn[1], g.mx[1]);
        p.z = clampf(p.z + dt * v.z, g.mn[2], g.mx[2]);
        p.w = p.w - 1.f;
    } else {
        // psfsolver.cpp:217-222 with the counter-based generator.
        // Particles are stored in cell order; the generator is keyed by the
        // caller's particle index so respawns do not depend on that order.
        const uint32_t id = (uint32_t)perm[idx];
        const uint32_t r1 = respawn_hash(tp.seed, step, id, 1) % 1024u;
        const uint32_t r2 = respawn_hash(tp.seed, step, id, 2) % 1024u;
        const uint32_t r3 = respawn_hash(tp.seed, step, id, 3) % 1024u;
        const float cz = g.mn[2] + 0.5f * (g.mx[2] - g.mn[2]);
        p.x = (float)(((double)r1 / 1024.0 - 0.5) * 0.25);
        p.y = g.mn[1] + 0.2f;
        p.z = (float)(-(double)cz + ((double)r3 / 1024.0 - 0.5) * 0.25);
        p.w = (float)((double)tp.lifetime * ((double)r2 / 1024.0));
    }
    return p;
}

// Storage order of particles: bricks of 16 x 2 x 2 voxels, in a brick the
// half-cells' rows along x.  A face field's rows run along x too, so the lanes
// of a warp gather from few 128-byte lines (a Morton order's 32 particles lie
// in twice as many rows), while a block's particles still share the rows in its
// L1.  Against Morton order: 64 x 16,384 particles on 64 x 32 x 32 41 against 51
// us, 513 x 16,384 on three domains 268 against 321 us, 16 x 262,144 on 32^3 RK1
// 70 against 80 us, RK4 99 against 102 us.
constexpr int BRICK_X = 4, BRICK_Y = 1, BRICK_Z = 1;                   // log2 of a brick's voxels
constexpr int BRICK_BITS = BRICK_X + (BRICK_Y + 1) + (BRICK_Z + 1);  // of a key, below the brick's number

struct Bricks {
    uint32_t nx, ny, nz;
    int key_bits;
    __device__ __forceinline__ uint32_t key(const GridDev &g, const float4 &p) const
    {
        const uint32_t x = (uint32_t)clampi(__float2int_rd((p.x - g.mn[0]) * g.inv_h), 0, g.nx - 1);
        const uint32_t hy = (uint32_t)clampi(__float2int_rd(2.0f * ((p.y - g.mn[1]) * g.inv_h)), 0, 2 * g.ny - 1);
        const uint32_t hz = (uint32_t)clampi(__float2int_rd(2.0f * ((p.z - g.mn[2]) * g.inv_h)), 0, 2 * g.nz - 1);
        const uint32_t brick = ((hz >> (BRICK_Z + 1)) * ny + (hy >> (BRICK_Y + 1))) * nx + (x >> BRICK_X);
        const uint32_t row = ((hz & ((2u << BRICK_Z) - 1)) << (BRICK_Y + 1)) | (hy & ((2u << BRICK_Y) - 1));
        return (brick << BRICK_BITS) | (row << BRICK_X) | (x & ((1u << BRICK_X) - 1));
    }
};

// At 1023 voxels per axis 64 x 512 x 512 bricks: 24 + 8 bits.
__host__ __device__ inline Bricks bricks_of(const GridDev &g)
{
    Bricks b;
    b.nx = ((uint32_t)g.nx + (1u << BRICK_X) - 1) >> BRICK_X;
    b.ny = ((uint32_t)g.ny + (1u << BRICK_Y) - 1) >> BRICK_Y;
    b.nz = ((uint32_t)g.nz + (1u << BRICK_Z) - 1) >> BRICK_Z;
    b.key_bits = BRICK_BITS;
    while (((uint64_t)1 << (b.key_bits - BRICK_BITS)) < (uint64_t)b.nx * b.ny * b.nz) ++b.key_bits;
    return b;
}

}  // namespace psf
