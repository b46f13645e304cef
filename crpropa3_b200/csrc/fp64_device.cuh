// fp64_device.cuh -- device code of the FP64 form of the stepping path, shared
// by its translation units (step_fp64.cu, step_fp64_bp.cu, step_fp64_ck.cu).
//
// Operation for operation the reference's arithmetic, in the reference's
// order: PropagationBP::dY (PropagationBP.cpp:19), PropagationCK::tryStep /
// dYdt (PropagationCK.cpp:28, :51), DiffusionSDE::process / tryStep
// (DiffusionSDE.cpp:47, :233), Grid<Vector3f>::trilinearInterpolate in float
// (Grid.h:540), PeriodicMagneticField (MagneticField.cpp:41) and the scalar
// PlaneWaveTurbulence sum (PlaneWaveTurbulence.cpp:233).  The translation
// units are compiled with -fmad=false so that no multiply-add is contracted:
// where the reference uses only + - * / sqrt floor (the Boris push over a
// Grid3f) the device result is bit-identical to the reference built without
// FMA.  pow in the step controllers and DiffusionSDE is cr_pow (crmath.cuh),
// correctly rounded, which agrees with glibc's pow except where glibc itself
// misrounds (about 1e-3 of inputs); cos in the wave sum and log/cos in the
// normal draws are CUDA's, within a few ulp of glibc's.
#pragma once

#include <type_traits>

#include "chain.cuh"
#include "crmath.cuh"
#include "engine_internal.h"
#include "grid_interp.cuh"
#include "uf23.cuh"
#include "pt11.cuh"
#include "tf17.cuh"
#include "jf12.cuh"
#include "kst24_cmz.cuh"
#include "advection.cuh"

// Resident blocks of 128 threads per SM the register budget of the
// fixed-step Boris and the Cash-Karp kernels is sized for (measured on the
// grid workloads: both are bound by gather latency, and more warps in
// flight pay until spills set in).
#ifndef CRP_BP_FIXED_MIN_BLOCKS
#define CRP_BP_FIXED_MIN_BLOCKS 6
#endif
// The general grid's code (clipVolume, reflection, other interpolations) needs
// more registers: 4 blocks (300 000 candidates x 1000 steps over a 100^3 grid:
// mixed 6.4 ms, FP64 12.6 ms; at 5 blocks 6.9 and 13.2; at 6 with spills 10.5
// and 15.3).
#ifndef CRP_BP_GRID_MIN_BLOCKS
#define CRP_BP_GRID_MIN_BLOCKS 4
#endif
// The adaptive Boris push: 3 blocks (50 000 candidates over a 100^3 grid, mixed:
// 2.32 ms at the 2 its 195 registers allowed, 1.43 ms at 3, 1.58 at 4 with spills;
// FP64 3.1, 2.1 and 2.4 ms).
#ifndef CRP_BP_ADAPTIVE_MIN_BLOCKS
#define CRP_BP_ADAPTIVE_MIN_BLOCKS 3
#endif
#ifndef CRP_CK_MIN_BLOCKS
#define CRP_CK_MIN_BLOCKS 3
#endif

namespace crp {
namespace {

struct d3 { double x, y, z; };
__device__ __forceinline__ d3 mk(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ d3 add(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 sub(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 muls(d3 a, double f) { return {a.x * f, a.y * f, a.z * f}; }
__device__ __forceinline__ d3 divs(d3 a, double f) { return {a.x / f, a.y / f, a.z / f}; }
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross(d3 a, d3 v) {
    return {a.y * v.z - v.y * a.z, a.z * v.x - v.z * a.x, a.x * v.y - v.x * a.y};
}
__device__ __forceinline__ double norm(d3 a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
__device__ __forceinline__ d3 unit(d3 a) { return divs(a, norm(a)); }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double clipd(double x, double lo, double hi) { return dmax(lo, dmin(x, hi)); }

// ------------------------------------------------- quotients without divisions
// IEEE divisions and square roots made half of the instructions of a Boris step
// (eighteen divisions and two square roots of 652) and a third of a Cash-Karp
// try's (36 divisions).  Every one of them divides by something known beforehand
// (the grid spacing, the candidate's mass, c), shared by three components (1 +
// t^2, the norms) or within rounding of 1 (a norm taken again), and the same
// correctly rounded quotients follow from a correctly rounded reciprocal by fused
// remainders:
//
// the scalar quotient, root_near_1 and reciprocal_near_1: crmath.cuh
using crp::quotient;
__device__ __forceinline__ d3 quotient(d3 a, double b, double rb) {
    return {quotient(a.x, b, rb), quotient(a.y, b, rb), quotient(a.z, b, rb)};
}

// u / |u| for n2 = u.u within 2^-27 of 1.
__device__ __forceinline__ d3 unit_near_1(d3 u, double n2) {
    const double r = root_near_1(n2);
    return quotient(u, r, reciprocal_near_1(r));
}

__device__ __forceinline__ int exponent_bits(double a) { return __double2hiint(a) & 0x7fffffff; }

// Every component above 2^-900, so that quotients by an ordinary number have
// exact remainders.
__device__ __forceinline__ bool ordinary(d3 u) {
    return min(exponent_bits(u.x), min(exponent_bits(u.y), exponent_bits(u.z))) > 0x07b00000;
}

// unit(u), value for value.
__device__ __forceinline__ d3 unit_fast(d3 u) {
    const double r = norm(u);
    if (ordinary(u) && r > 1e-100 && r < 1e100) return quotient(u, r, 1.0 / r);
    return divs(u, r);
}

// ParticleState::setDirection after getUnitVector: u / |u| twice, value for value.
__device__ __forceinline__ d3 unit_twice(d3 u) {
    const double n2 = u.x * u.x + u.y * u.y + u.z * u.z;
    if (ordinary(u) && n2 > 1e-100 && n2 < 1e100) {
        if (fabs(n2 - 1) < 0x1p-27) {
            u = unit_near_1(u, n2);
        } else {
            const double r = sqrt(n2);
            u = quotient(u, r, 1.0 / r);
        }
        const double again = u.x * u.x + u.y * u.y + u.z * u.z;
        if (ordinary(u) && fabs(again - 1) < 0x1p-27) return unit_near_1(u, again);
        return divs(u, norm(u));
    }
    u = unit(u);
    return divs(u, norm(u));
}

// i mod n in [0, n); positions inside the grid need no division.
__device__ __forceinline__ int grid_wrap(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    const int r = i % n;
    return r < 0 ? r + n : r;
}

// Grid<Vector3f>::interpolate (Grid.h:318) -> trilinearInterpolate (:540).
// With a cell cache (FS_GRID kernels) the 8 corners are loaded only when the
// cell changes.
// PER: the grid is periodic with power-of-two dimensions and has no
// clipVolume (FS_GRID_PERIODIC): those branches are compiled out and the
// periodic clamp is a mask (equal to the double modulo of Grid.h:31 there).
__device__ __forceinline__ d3 trilinear(const float (&c)[8][3], double fX0, double fY0, double fZ0) {
    const float fx1 = (float)(1 - fX0), fy1 = (float)(1 - fY0), fz1 = (float)(1 - fZ0);
    const float fx0 = (float)fX0, fy0 = (float)fY0, fz0 = (float)fZ0;
    const float wx[8] = {fx1, fx0, fx1, fx1, fx0, fx1, fx0, fx0};
    const float wy[8] = {fy1, fy1, fy0, fy1, fy1, fy0, fy0, fy0};
    const float wz[8] = {fz1, fz1, fz1, fz0, fz0, fz0, fz1, fz0};
    float bx = 0.f, by = 0.f, bz = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        bx += c[k][0] * wx[k] * wy[k] * wz[k];
        by += c[k][1] * wx[k] * wy[k] * wz[k];
        bz += c[k][2] * wx[k] * wy[k] * wz[k];
    }
    return mk(bx, by, bz);
}

// The periodic power-of-two grid (PER below) with its own corner cache.  The
// coordinates are quotients by the spacing (g.inv_s*: its correctly rounded
// reciprocal); where one is too small for an exact remainder its cell and
// single-precision fraction do not depend on the last bit.
template <bool AHEAD>
__device__ __forceinline__ d3 grid_periodic(const DevGrid &g, d3 pos, unsigned &tag, float (&corner)[8][3], d3 u) {
    const double rx = quotient(pos.x - g.gox, g.sx, g.inv_sx), ry = quotient(pos.y - g.goy, g.sy, g.inv_sy),
                 rz = quotient(pos.z - g.goz, g.sz, g.inv_sz);
    const CellIndex i = cell_index(rx, ry, rz);
    const unsigned sy = (unsigned)g.nz, sx = (unsigned)g.ny * (unsigned)g.nz;
    const int ix0 = i.ix & (g.nx - 1), iy0 = i.iy & (g.ny - 1), iz0 = i.iz & (g.nz - 1);
    const unsigned x0 = (unsigned)ix0 * sx, y0 = (unsigned)iy0 * sy;
    if (x0 + y0 + iz0 != tag) {
        const unsigned x1 = (unsigned)((ix0 + 1) & (g.nx - 1)) * sx, y1 = (unsigned)((iy0 + 1) & (g.ny - 1)) * sy;
        load_corner_pairs<true>(g.pairs, x0 + y0, x1 + y0, x0 + y1, x1 + y1, iz0, corner);
        tag = x0 + y0 + iz0;
        if (AHEAD)
            ask_next_cell(g, ix0, iy0, iz0, (float)(rx - i.flx), (float)(ry - i.fly), (float)(rz - i.flz), (float)u.x,
                          (float)u.y, (float)u.z);
    }
    return trilinear(corner, rx - i.flx, ry - i.fly, rz - i.flz);
}

template <bool CACHE, bool PER = false>
__device__ __forceinline__ d3 grid_field_t(const DevGrid &g, d3 pos, Cand *cc) {
    if (!PER && g.interp != CRP_INTERPOLATION_TRILINEAR) {  // tricubic, nearest (Grid.h:328-331)
        const gi3 v = gi_vector_other(g, pos.x, pos.y, pos.z);
        return mk(v.x, v.y, v.z);
    }
    if (!PER && g.clip_volume) {
        bool in = (pos.x >= g.ox) && (pos.x <= g.ex);
        in &= (pos.y >= g.oy) && (pos.y <= g.ey);
        in &= (pos.z >= g.oz) && (pos.z <= g.ez);
        if (!in) return mk(0, 0, 0);
    }
    const double rx = quotient(pos.x - g.gox, g.sx, g.inv_sx), ry = quotient(pos.y - g.goy, g.sy, g.inv_sy),
                 rz = quotient(pos.z - g.goz, g.sz, g.inv_sz);
    int ix0, ix1, iy0, iy1, iz0, iz1;
    double fX0, fY0, fZ0;
    if (!PER && g.reflective) {  // reflectiveClamp (Grid.h:49)
        double r[3] = {rx, ry, rz}, res[3];
        int n[3] = {g.nx, g.ny, g.nz}, lo[3], hi[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            double x = r[a];
            int guard = 0;
            while (((x < -0.5) || (x > (n[a] - 0.5))) && guard < 64) {
                x = 2 * n[a] * (x > (n[a] - 0.5)) - x - 1;
                guard++;
            }
            res[a] = x;
            lo[a] = (int)floor(x);
            hi[a] = lo[a] + (lo[a] < n[a] - 1);
            if (x < 0) { lo[a] = 0; hi[a] = 0; }
            // positions beyond 64 reflections are outside any physical use
            if (lo[a] < 0 || lo[a] >= n[a]) { lo[a] = 0; hi[a] = 0; }
        }
        ix0 = lo[0]; ix1 = hi[0]; iy0 = lo[1]; iy1 = hi[1]; iz0 = lo[2]; iz1 = hi[2];
        fX0 = res[0] - floor(res[0]);
        fY0 = res[1] - floor(res[1]);
        fZ0 = res[2] - floor(res[2]);
    } else if (PER) {  // periodicClamp (Grid.h:31), power-of-two dimensions
        const CellIndex i = cell_index(rx, ry, rz);
        ix0 = i.ix & (g.nx - 1); ix1 = (ix0 + 1) & (g.nx - 1);
        iy0 = i.iy & (g.ny - 1); iy1 = (iy0 + 1) & (g.ny - 1);
        iz0 = i.iz & (g.nz - 1); iz1 = (iz0 + 1) & (g.nz - 1);
        fX0 = rx - i.flx;
        fY0 = ry - i.fly;
        fZ0 = rz - i.flz;
    } else {  // periodicClamp (Grid.h:31)
        ix0 = grid_wrap((int)floor(rx), g.nx); ix1 = ix0 + 1 == g.nx ? 0 : ix0 + 1;
        iy0 = grid_wrap((int)floor(ry), g.ny); iy1 = iy0 + 1 == g.ny ? 0 : iy0 + 1;
        iz0 = grid_wrap((int)floor(rz), g.nz); iz1 = iz0 + 1 == g.nz ? 0 : iz0 + 1;
        fX0 = rx - floor(rx);
        fY0 = ry - floor(ry);
        fZ0 = rz - floor(rz);
    }
    // cell indices: 32-bit for FS_GRID_PERIODIC grids (fewer than 2^31 cells)
    using Index = typename std::conditional<PER, unsigned, size_t>::type;
    const Index sy = (Index)g.nz, sx = (Index)g.ny * (Index)g.nz;
    const Index b00 = (Index)ix0 * sx + (Index)iy0 * sy, b10 = (Index)ix1 * sx + (Index)iy0 * sy;
    const Index b01 = (Index)ix0 * sx + (Index)iy1 * sy, b11 = (Index)ix1 * sx + (Index)iy1 * sy;
    float lc[8][3];
    float (*c)[3] = CACHE ? cc->corner : lc;
    const long long k0 = (long long)(b00 + iz0), k7 = (long long)(b11 + iz1);
    if (!CACHE || (PER ? b00 + iz0 != cc->tag : (k0 != cc->cell0 || k7 != cc->cell7))) {
        if (PER || g.pairs) {
            load_corner_pairs<CACHE>(g.pairs, b00, b10, b01, b11, iz0, c);
            if (!PER && iz1 == iz0) {  // the reflective edge: no upper neighbour
#pragma unroll
                for (int a = 0; a < 3; a++) { c[3][a] = c[0][a]; c[4][a] = c[1][a]; c[5][a] = c[2][a]; c[7][a] = c[6][a]; }
            }
        } else {
            const float *v = g.values;
            const Index idx[8] = {b00 + iz0, b10 + iz0, b01 + iz0, b00 + iz1, b10 + iz1, b01 + iz1, b11 + iz0, b11 + iz1};
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float *p = v + 3 * (size_t)idx[k];
                c[k][0] = __ldg(p); c[k][1] = __ldg(p + 1); c[k][2] = __ldg(p + 2);
            }
        }
        if (CACHE) { cc->cell0 = k0; cc->cell7 = k7; cc->tag = (unsigned)(b00 + iz0); }
    }
    return trilinear(CACHE ? cc->corner : lc, fX0, fY0, fZ0);
}

__device__ d3 grid_field(const DevGrid &g, d3 pos) { return grid_field_t<false>(g, pos, nullptr); }

// PlaneWaveTurbulence::getField, scalar branch (PlaneWaveTurbulence.cpp:233).
__device__ d3 plane_wave_field(const DevPlaneWave &w, d3 pos) {
    d3 B = mk(0, 0, 0);
    const double *m = w.modes;
#pragma unroll 1
    for (int i = 0; i < w.n; i++, m += 9) {
        d3 xi = mk(__ldg(m), __ldg(m + 1), __ldg(m + 2));
        d3 kap = mk(__ldg(m + 3), __ldg(m + 4), __ldg(m + 5));
        double k = __ldg(m + 6), beta = __ldg(m + 7), ak = __ldg(m + 8);
        double z_ = dot(pos, kap);
        B = add(B, muls(muls(xi, ak), cos(k * z_ + beta)));
    }
    return B;
}

// The same sum for a block's candidates (FS_PLANE_WAVE_BLOCK kernels; every
// thread of the block calls it): the sum over the modes is one chain in the
// reference's order, but its terms are not.  The block's first 32 wp threads (wp 1 or
// 2) hold the candidates; per round of kWaveRound modes the four warps evaluate
// the cosines of a quarter of the modes each for all of them, and warp a < 3 adds
// component a of the round's terms in order.  3001 candidates x 60 steps x 77
// modes: 1.32 ms thread by thread, 0.83 ms here.
constexpr int kBatchThreads = 128, kWaveRound = 16, kWaveCandidates = 64;
inline size_t wave_table_bytes(const DevPlaneWave &w) { return (size_t)w.n * 72; }
__device__ __forceinline__ void stage_wave_table(const DevPlaneWave &w, unsigned char *to) {
    double *t = reinterpret_cast<double *>(to);
    for (int q = threadIdx.x; q < 9 * w.n; q += blockDim.x) t[q] = __ldg(w.modes + q);
}

__device__ __forceinline__ d3 plane_wave_block(const DevPlaneWave &w, d3 pos, int wp) {
    __shared__ double qpos[3][kWaveCandidates], cosine[kWaveRound][kWaveCandidates], sum[3][kWaveCandidates];
    extern __shared__ __align__(16) unsigned char pw_table[];
    const double *tab = reinterpret_cast<const double *>(pw_table);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int mine = t < kWaveCandidates ? t : 0;  // threads past the candidates take any sum
    if (t < kWaveCandidates) { qpos[0][t] = pos.x; qpos[1][t] = pos.y; qpos[2][t] = pos.z; }
    double acc[2] = {0, 0};  // of candidates lane + 32 j, component `warp`
    for (int m0 = 0; m0 < w.n; m0 += kWaveRound) {
        const int m1 = min(w.n - m0, kWaveRound);
        __syncthreads();
        for (int m = warp; m < m1; m += 4) {
            const double *q = tab + 9 * (m0 + m);
            const d3 kap = mk(q[3], q[4], q[5]);
            const double k = q[6], beta = q[7];
            for (int j = 0; j < wp; j++) {
                const int i = lane + 32 * j;
                cosine[m][i] = cos(k * dot(mk(qpos[0][i], qpos[1][i], qpos[2][i]), kap) + beta);
            }
        }
        __syncthreads();
        if (warp < 3)
            for (int m = 0; m < m1; m++) {
                const double *q = tab + 9 * (m0 + m);
                const double a = q[warp] * q[8];
#pragma unroll
                for (int j = 0; j < 2; j++)
                    if (j < wp) acc[j] = acc[j] + a * cosine[m][lane + 32 * j];
            }
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
        if (warp < 3 && j < wp) sum[warp][lane + 32 * j] = acc[j];
    __syncthreads();
    return mk(sum[0][mine], sum[1][mine], sum[2][mine]);
}

// ---------------------------------------------------------------- JF12Field
// The reference's arithmetic operation for operation (JF12Field.cpp:195-346);
// the regular field (JF12Field, PlanckJF12bField and JF12FieldSolenoidal) is
// in jf12.cuh.

__device__ __forceinline__ d3 jf12_regular(const crp_jf12_desc &J, d3 pos) {
    const u3 b = jf12_regular_fp64(J, pos.x, pos.y, pos.z);
    return mk(b.x, b.y, b.z);
}

// JF12Field::getTurbulentStrength (JF12Field.cpp:301)
__device__ double jf12_turbulent_strength(const crp_jf12_desc &J, d3 pos) {
    const double kpc = J.kpc;
    if (sqrt(pos.x * pos.x + pos.y * pos.y + pos.z * pos.z) > 20 * kpc) return 0;
    const double r = sqrt(pos.x * pos.x + pos.y * pos.y);
    const double phi = jf_phi(pos.x, pos.y);
    double bDisk = 0;
    if (r < 5 * kpc) {
        bDisk = J.b_disk_turb5;
    } else {
        const double r_negx = jf_r_negx(J, r, phi);
        for (int i = 7; i >= 0; i--)
            if (r_negx < J.r_arms[i]) bDisk = J.b_disk_turb[i];
        bDisk *= (5 * kpc) / r;
    }
    bDisk *= exp(-0.5 * jf_sq(pos.z / J.z_disk_turb));
    const double bHalo = J.b_halo_turb * exp(-r / J.r_halo_turb) * exp(-0.5 * jf_sq(pos.z / J.z_halo_turb));
    return sqrt(jf_sq(bDisk) + jf_sq(bHalo));
}

// JF12Field::getField (JF12Field.cpp:346): turbulent + (striated or regular).
// Not inlined: the generic-field kernels keep their register budget.
__device__ __noinline__ d3 jf12_field(const DevComponent &f, d3 pos) {
    const crp_jf12_desc &J = f.jf->d;
    d3 b = mk(0., 0., 0.);
    if (J.use_turbulent) {
        // Vector3f * double: the strength is rounded to float, the product is float
        const d3 g = grid_field(f.grid, pos);
        const float s = (float)jf12_turbulent_strength(J, pos);
        b = add(b, mk((double)__fmul_rn((float)g.x, s), (double)__fmul_rn((float)g.y, s),
                      (double)__fmul_rn((float)g.z, s)));
    }
    if (J.use_striated) {  // JF12Field.cpp:296, closestValue of the striated Grid1f
        const double v = (double)__ldg(f.mod.values + gi_nearest_cell(f.mod, pos.x, pos.y, pos.z));
        b = add(b, muls(jf12_regular(J, pos), 1. + J.sqrt_beta * v));
    } else if (J.use_regular) {
        b = add(b, jf12_regular(J, pos));
    }
    return b;
}

__device__ d3 component_field(const DevComponent &f, d3 position) {
    d3 pos = position;
    if (f.periodic) {  // PeriodicMagneticField::getField (MagneticField.cpp:41)
        d3 o = mk(f.po[0], f.po[1], f.po[2]), e = mk(f.pe[0], f.pe[1], f.pe[2]);
        d3 q = sub(position, o);
        d3 n = mk(floor(q.x / e.x), floor(q.y / e.y), floor(q.z / e.z));
        d3 p = sub(q, mk(n.x * e.x, n.y * e.y, n.z * e.z));
        if (f.periodic_reflective) {
            if ((long long)fabs(n.x) % 2 == 1) p.x = e.x - p.x;
            if ((long long)fabs(n.y) % 2 == 1) p.y = e.y - p.y;
            if ((long long)fabs(n.z) % 2 == 1) p.z = e.z - p.z;
        }
        pos = p;
    }
    switch (f.kind) {
    case CRP_FIELD_GRID: return grid_field(f.grid, pos);
    case CRP_FIELD_MODULATED_GRID: {  // ModulatedMagneticFieldGrid::getField (MagneticFieldGrid.cpp:51)
        const float m = gi_scalar(f.mod, pos.x, pos.y, pos.z);
        return muls(grid_field(f.grid, pos), (double)m);
    }
    case CRP_FIELD_PLANE_WAVE: return plane_wave_field(f.pw, pos);
    case CRP_FIELD_UNIFORM: return mk(f.uniform[0], f.uniform[1], f.uniform[2]);
    case CRP_FIELD_JF12: return jf12_field(f, pos);
    case CRP_FIELD_UF23: {
        const u3 b = uf23_field(*f.uf, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_PT11: {
        const u3 b = pt11_field(*f.pt, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_ARCHIMEDEAN_SPIRAL: {
        const u3 b = archimedean_field(f.arch, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_TF17: {
        const u3 b = tf17_field(*f.tf, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_SINGLE_MODE: {
        const u3 b = single_mode_field(f.mode, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_KST24: {
        const u3 b = kst24_field(*f.kst, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    case CRP_FIELD_CMZ: {
        const u3 b = cmz_field(*f.cmz, pos.x, pos.y, pos.z);
        return mk(b.x, b.y, b.z);
    }
    default: {
        double r = sqrt(pos.x * pos.x + pos.y * pos.y);
        return muls(mk(-pos.y, pos.x, 0.), f.b0 / r);
    }
    }
}

// MagneticFieldList::getField (MagneticField.cpp:64) or the single field.
__device__ __forceinline__ d3 field_sum(const DevComponent *f, int n, d3 pos) {
    if (n == 1) return component_field(f[0], pos);
    d3 b = mk(0, 0, 0);
#pragma unroll 1
    for (int i = 0; i < n; i++) b = add(b, component_field(f[i], pos));
    return b;
}
// The same as a call (why and where: field_sum_call in mixed_device.cuh; here also in
// DiffusionSDE, 30 000 pseudo-particles in a toroidal field 0.23 ms inlined, 0.18).
__device__ __noinline__ d3 field_sum_call(const DevComponent *f, int n, d3 pos) { return field_sum(f, n, pos); }

// A single galactic field, without the sum's tests and loads.
__device__ __forceinline__ d3 galactic_field(const DevComponent &f, d3 pos) {
    u3 b;
    switch (f.kind) {
    case CRP_FIELD_JF12: return jf12_field(f, pos);
    case CRP_FIELD_UF23: b = uf23_field(*f.uf, pos.x, pos.y, pos.z); break;
    case CRP_FIELD_PT11: b = pt11_field(*f.pt, pos.x, pos.y, pos.z); break;
    case CRP_FIELD_TF17: b = tf17_field(*f.tf, pos.x, pos.y, pos.z); break;
    default: b = kst24_field(*f.kst, pos.x, pos.y, pos.z);
    }
    return mk(b.x, b.y, b.z);
}

template <int FS, bool CALL = false>
__device__ __forceinline__ d3 field_at(const DevPlan &P, d3 pos, Cand *cc = nullptr) {
    if (FS == FS_GRID) return grid_field_t<true>(P.fields[0].grid, pos, cc);
    if (FS == FS_GRID_PERIODIC) return grid_field_t<true, true>(P.fields[0].grid, pos, cc);
    if (FS == FS_PLANE_WAVE) return plane_wave_field(P.fields[0].pw, pos);
    if (FS == FS_PLANE_WAVE_BLOCK) return plane_wave_block(P.fields[0].pw, pos, P.block_warps);
    if (FS == FS_GALACTIC) return galactic_field(P.fields[0], pos);
    return CALL ? field_sum_call(P.dev_fields, P.n_fields, pos) : field_sum(P.fields, P.n_fields, pos);
}

__device__ __forceinline__ void set_current_step(Cand &c, double s) {  // Candidate.cpp:92
    c.cur = s;
    c.len += s;
    c.time += s / kCLight;
}

// ---------------------------------------------------------------- Boris push
// A candidate's factors of the rotation vector t = B q / 2 / m * step / c.
// plain: the range in which every quotient of the push and its remainder is a
// normal number for any nonzero float field value and steps of 1e-60 to 1e60 m.
struct BorisFactors {
    double q, mass, rmass;
    bool plain;
    __device__ __forceinline__ BorisFactors(double charge, double E) : q(charge) {
        mass = E / (kCLight * kCLight);
        rmass = 1.0 / mass;
        plain = fabs(q) > 1e-60 && fabs(q) < 1e60 && mass > 1e-60 && mass < 1e60;
    }
};
__device__ __forceinline__ bool plain_step(double step) { return step > 1e-60 && step < 1e60; }

// PropagationBP::dY (PropagationBP.cpp:19) after the first half drift: the
// rotation in the field B.  PLAIN: the factors and the step are known to be plain.
template <bool PLAIN>
__device__ __forceinline__ d3 boris_rotate(d3 u, d3 B, double step, const BorisFactors &f) {
    d3 t, s;
    double D;
    const float least = fminf(fabsf((float)B.x), fminf(fabsf((float)B.y), fabsf((float)B.z)));
    bool plain = least > 0.f && (PLAIN || (f.plain && plain_step(step)));
    if (plain) {
        t = quotient(muls(quotient(divs(muls(B, f.q), 2), f.mass, f.rmass), step), kCLight, 1.0 / kCLight);
        D = 1 + dot(t, t);
        plain = D < 1e150;
        s = quotient(muls(t, 2), D, 1.0 / D);
    }
    if (!plain) {  // a component is zero or not finite
        t = divs(muls(divs(divs(muls(B, f.q), 2), f.mass), step), kCLight);
        D = 1 + dot(t, t);
        s = divs(muls(t, 2), D);
    }
    const d3 vh = add(u, cross(u, t));
    return add(u, cross(vh, s));
}

template <int FS>
__device__ __forceinline__ void bp_dy(const DevPlan &P, d3 &x, d3 &u, double step, const BorisFactors &f, Cand *cc) {
    x = add(x, divs(muls(u, step), 2.));
    u = boris_rotate<false>(u, field_at<FS>(P, x, cc), step, f);
    x = add(x, divs(muls(u, step), 2.));
}

// The step of a neutral candidate (PropagationBP.cpp:67, PropagationCK.cpp:81).
__device__ __forceinline__ void neutral_step(const DevModule &m, Cand &c) {
    const double step = clipd(c.next, m.min_step, m.max_step);
    c.x = c.x + c.dx * step; c.y = c.y + c.dy * step; c.z = c.z + c.dz * step;
    set_current_step(c, step);
    c.next = m.max_step;
}

__device__ __forceinline__ void set_direction(Cand &c, d3 uo) {
    const d3 u = unit_twice(uo);  // ParticleState::setDirection normalises again
    c.dx = u.x; c.dy = u.y; c.dz = u.z;
}

template <int FS, int MODE>
struct BP {
    static constexpr bool kBorisKernel = MODE == 1;  // its own kernel for CS_PM over FS_GRID_PERIODIC
    static constexpr bool kReadsStepCount = false;
    static constexpr bool kCashKarp = false;
    static constexpr bool kBlockField = true;  // takes its field from the block (attempt's `on`)
    static constexpr bool kTogether = MODE != 1;  // advance()
    // PropagationBP::process (PropagationBP.cpp:62): its start (false when the
    // step is done, neutral candidates) and one try (true when it is done; threads
    // that only take part in its field evaluations pass on = false).
    struct Try {
        double step;
        int guard;
    };
    __device__ __forceinline__ static bool begin(const DevPlan &P, const DevModule &m, Cand &c, Try &t) {
        c.px = c.x; c.py = c.y; c.pz = c.z;
        if (c.q == 0) {
            neutral_step(m, c);
            return false;
        }
        t.step = MODE == 1 ? m.max_step : clipd(c.next, m.min_step, m.max_step);
        t.guard = 0;
        return true;
    }
    __device__ __forceinline__ static bool attempt(const DevPlan &P, const DevModule &m, Cand &c, Try &t,
                                                   StepCount &sc, bool on = true) {
        double step = t.step, newStep = step;
        const BorisFactors f(c.q, c.E);
        d3 xo = mk(c.x, c.y, c.z), uo = mk(c.dx, c.dy, c.dz);
        if (MODE == 1) {
            bp_dy<FS>(P, xo, uo, step, f, &c);
            if (!on) return false;
            sc.tries++; sc.evals++;
        } else {
            // the full step, then two half steps: one loop body for the three
            d3 x = xo, u = uo;
            double h = step;
#pragma unroll 1
            for (int i = 0; i < 3; i++) {
                bp_dy<FS>(P, x, u, h, f, &c);
                if (i == 0) {
                    xo = x; uo = u;
                    x = mk(c.x, c.y, c.z); u = mk(c.dx, c.dy, c.dz);
                    h = step / 2;
                }
            }
            if (!on) return false;
            sc.tries++; sc.evals += 3;
            const double S = norm(sub(xo, x)) / (step * (1 - 1 / 4.));
            const double r = norm(mk(S, S, S)) / m.tolerance;
            if (step_control(m, r, step, newStep, cr_pow) && ++t.guard < 4096) {
                t.step = newStep;
                return false;
            }
            if (t.guard == 4096) step = newStep;
        }
        c.x = xo.x; c.y = xo.y; c.z = xo.z;
        set_direction(c, uo);
        set_current_step(c, step);
        c.next = newStep;
        return true;
    }
};

// The push of boris_body in the FP64 form: BP<FS_GRID_PERIODIC, 1>'s step, value
// for value.  AHEAD: ask_next_cell.
template <bool AHEAD>
struct BorisPush {
    static constexpr bool kAhead = AHEAD;
    BorisFactors f;
    unsigned tag;
    float corner[8][3];
    __device__ __forceinline__ static bool sane(const DevPlan &P, double q, double E) {
        return BorisFactors(q, E).plain && plain_step(P.modules[0].max_step);
    }
    __device__ __forceinline__ static double later(double time, double step) { return time + step / kCLight; }
    __device__ __forceinline__ BorisPush(const DevPlan &, double q, double E) : f(q, E) { tag = kNoCell; }
    __device__ __forceinline__ void step(const DevPlan &P, double &x, double &y, double &z, double &ux, double &uy,
                                         double &uz) {
        const double h = P.modules[0].max_step;
        d3 X = mk(x, y, z), u = mk(ux, uy, uz);
        X = add(X, divs(muls(u, h), 2.));
        u = boris_rotate<true>(u, grid_periodic<AHEAD>(P.fields[0].grid, X, tag, corner, u), h, f);
        X = add(X, divs(muls(u, h), 2.));
        u = unit_twice(u);
        x = X.x; y = X.y; z = X.z;
        ux = u.x; uy = u.y; uz = u.z;
    }
};

// --------------------------------------------------------------- Cash-Karp
__constant__ double ck_a[36] = {
    0., 0., 0., 0., 0., 0.,
    1. / 5., 0., 0., 0., 0., 0.,
    3. / 40., 9. / 40., 0., 0., 0., 0.,
    3. / 10., -9. / 10., 6. / 5., 0., 0., 0.,
    -11. / 54., 5. / 2., -70. / 27., 35. / 27., 0., 0.,
    1631. / 55296., 175. / 512., 575. / 13824., 44275. / 110592., 253. / 4096., 0.};
__constant__ double ck_b[6] = {37. / 378., 0, 250. / 621., 125. / 594., 0., 512. / 1771.};
__constant__ double ck_bs[6] = {2825. / 27648., 0., 18575. / 48384., 13525. / 55296.,
                                277. / 14336., 1. / 4.};

template <int FS, bool CALL>
__device__ __forceinline__ void ck_try(const DevPlan &P, d3 x, d3 u, double h, double q, double E,
                                       d3 &xo, d3 &uo, d3 &eu, Cand *cc) {
    d3 kx[6], ku[6];
    xo = x; uo = u;
    eu = mk(0, 0, 0);
    const double qcE = q * kCLight / E;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        d3 yx = x, yu = u;
#pragma unroll
        for (int j = 0; j < i; j++) {
            yx = add(yx, muls(muls(kx[j], ck_a[i * 6 + j]), h));
            yu = add(yu, muls(muls(ku[j], ck_a[i * 6 + j]), h));
        }
        d3 vel = muls(unit_fast(yu), kCLight);
        d3 B = field_at<FS, CALL>(P, yx, cc);
        d3 dudt = muls(cross(vel, B), qcE);
        kx[i] = vel; ku[i] = dudt;
        if (i != 1 && i != 4) {  // b_1 = b_4 = 0
            xo = add(xo, muls(muls(kx[i], ck_b[i]), h));
            uo = add(uo, muls(muls(ku[i], ck_b[i]), h));
        }
        if (i != 1) eu = add(eu, muls(muls(ku[i], ck_b[i] - ck_bs[i]), h));
    }
}

template <int FS, int MODE, bool CALLED>
struct CK {
    static constexpr bool kBorisKernel = false;  // its own kernel for CS_PM over FS_GRID_PERIODIC
    static constexpr bool kReadsStepCount = false;
    static constexpr bool kCashKarp = true;
    static constexpr bool kBlockField = true;  // takes its field from the block (attempt's `on`)
    static constexpr bool kTogether = MODE != 1 || FS == FS_GENERIC;  // advance()
    // PropagationCK::process (PropagationCK.cpp:77): its start (false when the
    // step is done, neutral candidates) and one try (true when it is done; threads
    // that only take part in its field evaluations pass on = false).
    struct Try {
        double step;
        int guard;
    };
    __device__ __forceinline__ static bool begin(const DevPlan &P, const DevModule &m, Cand &c, Try &t) {
        c.px = c.x; c.py = c.y; c.pz = c.z;
        if (c.q == 0) {
            neutral_step(m, c);
            return false;
        }
        t.step = MODE == 1 ? m.max_step : clipd(c.next, m.min_step, m.max_step);
        t.guard = 0;
        return true;
    }
    __device__ __forceinline__ static bool attempt(const DevPlan &P, const DevModule &m, Cand &c, Try &t,
                                                   StepCount &sc, bool on = true) {
        double step = t.step, newStep = step;
        d3 xo, uo, eu;
        ck_try<FS, CALLED>(P, mk(c.x, c.y, c.z), mk(c.dx, c.dy, c.dz), step / kCLight, c.q, c.E, xo, uo, eu, &c);
        if (!on) return false;
        sc.tries++; sc.evals += 6;
        if (MODE != 1) {
            const double r = norm(eu) / m.tolerance;
            if (step_control(m, r, step, newStep, cr_pow) && ++t.guard < 4096) {
                t.step = newStep;
                return false;
            }
            if (t.guard == 4096) step = newStep;
        }
        c.x = xo.x; c.y = xo.y; c.z = xo.z;
        set_direction(c, uo);
        set_current_step(c, step);
        c.next = newStep;
        return true;
    }
};

// ------------------------------------------------------------ DiffusionSDE
__device__ __forceinline__ double s_rand(Stream &s) { return (double)s.next_u32() * (1.0 / 4294967295.0); }
__device__ __forceinline__ double s_uniform(Stream &s, double a, double b) { return a + (b - a) * s_rand(s); }
__device__ __forceinline__ double s_norm(Stream &s) {  // Random::randNorm (Random.cpp:104)
    double dblexc = ((double)s.next_u32() + 0.5) * (1.0 / 4294967296.0);
    double r = sqrt(-2.0 * log(1.0 - dblexc)) * 1.0;
    double phi = 2.0 * 3.14159265358979323846264338328 * ((double)s.next_u32() * (1.0 / 4294967296.0));
    return 0.0 + r * cos(phi);
}
__device__ __forceinline__ d3 s_vector(Stream &s) {  // Random::randVector (Random.cpp:141)
    double z = s_uniform(s, -1.0, 1.0);
    double t = s_uniform(s, -1.0 * kPi, kPi);
    double r = sqrt(1 - z * z);
    return mk(r * cos(t), r * sin(t), z);
}
__device__ __forceinline__ d3 rotated(d3 v, d3 axis, double angle) {  // Vector3.h:206
    d3 u = axis;
    if (norm(u) != 0.) u = divs(u, norm(u));
    double c = cos(angle), s = sin(angle);
    d3 Rx = mk(c + u.x * u.x * (1 - c), u.x * u.y * (1 - c) - u.z * s, u.x * u.z * (1 - c) + u.y * s);
    d3 Ry = mk(u.y * u.x * (1 - c) + u.z * s, c + u.y * u.y * (1 - c), u.y * u.z * (1 - c) - u.x * s);
    d3 Rz = mk(u.z * u.x * (1 - c) - u.y * s, u.z * u.y * (1 - c) + u.x * s, c + u.z * u.z * (1 - c));
    return mk(dot(v, Rx), dot(v, Ry), dot(v, Rz));
}

template <int FS>
__device__ __forceinline__ void sde_try(const DevPlan &P, d3 PosIn, d3 &POut, d3 &PosErr,
                                        double propStep, Cand *cc) {
    d3 k[6];
    POut = PosIn;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        d3 y_n = PosIn;
#pragma unroll
        for (int j = 0; j < i; j++) y_n = add(y_n, muls(muls(k[j], ck_a[i * 6 + j]), propStep));
        d3 B = field_at<FS, true>(P, y_n, cc);
        k[i] = muls(unit(B), kCLight);
        POut = add(POut, muls(muls(k[i], ck_b[i]), propStep));
        PosErr = add(PosErr, divs(muls(muls(k[i], ck_b[i] - ck_bs[i]), propStep), CRP_KPC));
    }
}

template <int FS>
struct SDE {
    static constexpr bool kBorisKernel = false;  // its own kernel for CS_PM over FS_GRID_PERIODIC
    static constexpr bool kReadsStepCount = true;  // the Philox counter
    static constexpr bool kBlockField = false;
    static constexpr bool kTogether = false;  // advance()
    struct Try {};
    __device__ __forceinline__ static bool begin(const DevPlan &, const DevModule &, Cand &, Try &) { return true; }
    __device__ __forceinline__ static bool attempt(const DevPlan &P, const DevModule &m, Cand &c, Try &,
                                                   StepCount &sc) {
        process(P, m, c, sc);
        return true;
    }
    // DiffusionSDE::process (DiffusionSDE.cpp:47); the advection drift of
    // driftStep (:255) is LinProp = 0 + v_adv(PosIn) h.
    __device__ static d3 lin_prop(const DevModule &m, d3 pos, double h, double t) {
        if (m.n_adv == 0) return mk(0, 0, 0);
        const u3 v = advection_at(m.adv, m.n_adv, pos.x, pos.y, pos.z, t);
        return add(mk(0, 0, 0), muls(mk(v.x, v.y, v.z), h));
    }
    __device__ static void process(const DevPlan &P, const DevModule &m, Cand &c, StepCount &sc) {
        c.px = c.x; c.py = c.y; c.pz = c.z;
        double h = clipd(c.next, m.min_step, m.max_step) / kCLight;
        d3 PosIn = mk(c.x, c.y, c.z);
        if (c.q == 0) {
            d3 p = add(add(PosIn, lin_prop(m, PosIn, h, c.time)), muls(muls(mk(c.dx, c.dy, c.dz), h), kCLight));
            c.x = p.x; c.y = p.y; c.z = p.z;
            set_current_step(c, h * kCLight);
            c.next = m.max_step;
            return;
        }
        double rig = c.E / c.q;
        double DifCoeff = m.scale * 6.1e24 * cr_pow((fabs(rig) / 4.0e9), m.alpha);
        double BT0 = cr_pow(2 * DifCoeff, 0.5);
        double BT4 = cr_pow(2 * m.eps * DifCoeff, 0.5);
        Stream s{P.seed, c.index, c.steps, make_uint4(0, 0, 0, 0), 0};
        double eta0 = s_norm(s), eta1 = s_norm(s), eta2 = s_norm(s);
        double TStep = BT0 * eta0, NStep = BT4 * eta1, BStep = BT4 * eta2;
        double propTime = TStep * sqrt(h) / kCLight;
        unsigned counter = 0;
        double r = 42.;
        do {
            d3 PosOut = mk(0, 0, 0), PosErr = mk(0, 0, 0);
            sde_try<FS>(P, PosIn, PosOut, PosErr, propTime, &c);
            sc.tries++; sc.evals += 6;
            r = norm(PosErr) / m.tolerance;
            propTime *= 0.5;
            counter += 1;
        } while (r > 1 && fabs(propTime) >= m.min_step / kCLight && counter < 60);
        unsigned long long stepNumber = (unsigned long long)pow(2.0, (double)(counter - 1));
        double allowedTime = TStep * sqrt(h) / kCLight / (double)stepNumber;
        d3 Start = PosIn, PosOut = mk(0, 0, 0), PosErr = mk(0, 0, 0);
        for (unsigned long long j = 0; j < stepNumber; j++) {
            sde_try<FS>(P, Start, PosOut, PosErr, allowedTime, &c);
            sc.tries++; sc.evals += 6;
            Start = PosOut;
        }
        d3 TVec = unit(sub(PosOut, PosIn));
        double tTest = norm(TVec);
        if (tTest != tTest) {
            if (m.n_adv) {  // only the advection drift
                const d3 p = add(PosIn, lin_prop(m, PosIn, h, c.time));
                c.x = p.x; c.y = p.y; c.z = p.z;
            } else {
                c.x = c.x + c.dx * h * kCLight; c.y = c.y + c.dy * h * kCLight; c.z = c.z + c.dz * h * kCLight;
            }
            set_current_step(c, h * kCLight);
            double newStep = 5 * h * kCLight;
            c.next = clipd(newStep, m.min_step, m.max_step);
            return;
        }
        d3 NVec = mk(0, 0, 0);
        for (int guard = 0; norm(NVec) == 0. && guard < 3; guard++) NVec = cross(TVec, s_vector(s));
        if (norm(NVec) == 0.) { c.active = false; c.flags |= CRP_FLAG_NAN; return; }
        NVec = unit(NVec);
        d3 BVec = unit(cross(TVec, NVec));
        d3 PO = add(add(PosOut, lin_prop(m, PosIn, h, c.time)), muls(add(muls(NVec, NStep), muls(BVec, BStep)), sqrt(h)));
        if (isnan(norm(PO))) { c.active = false; c.flags |= CRP_FLAG_NAN; return; }
        s.cursor = 12;  // the cone draw takes the fourth block of the step
        double theta = acos(s_uniform(s, 1, cos(kPi / 2.)));
        d3 axis = cross(TVec, s_vector(s));
        d3 DirOut = rotated(TVec, axis, theta);
        c.x = PO.x; c.y = PO.y; c.z = PO.z;
        DirOut = divs(DirOut, norm(DirOut));
        c.dx = DirOut.x; c.dy = DirOut.y; c.dz = DirOut.z;
        set_current_step(c, h * kCLight);
        double nextStep;
        if (stepNumber > 1) nextStep = h * pow((double)stepNumber, -2.) * kCLight;
        else nextStep = 4 * h * kCLight;
        c.next = nextStep;
    }
};

// step-mode variants selected by the launcher from min_step == max_step, so
// that a fixed-step kernel carries no adaptive-controller registers
template <int FS> using BPFixed = BP<FS, 1>;
// resident blocks of 128 threads per SM the register budget is sized for:
// the fixed-step Boris push is latency bound on its gathers and wants warps
template <class T> struct MinBlocks { static constexpr int value = 1; };
template <int FS, int MODE> struct MinBlocks<BP<FS, MODE>> {
    static constexpr int value = MODE != 1 ? CRP_BP_ADAPTIVE_MIN_BLOCKS : FS == FS_GRID ? CRP_BP_GRID_MIN_BLOCKS : CRP_BP_FIXED_MIN_BLOCKS;
};
template <int FS, int MODE, bool CALLED> struct MinBlocks<CK<FS, MODE, CALLED>> {
    static constexpr int value = CRP_CK_MIN_BLOCKS;
};
template <int FS> using BPAdaptive = BP<FS, 2>;
template <int FS> using CKFixed = CK<FS, 1, FS == FS_GENERIC>;
template <int FS> using CKFixedInlined = CK<FS, 1, false>;  // lists of fields, warps full (step_*_ck.cu)
template <int FS> using CKAdaptive = CK<FS, 2, FS == FS_GENERIC>;

template <template <int> class Prop, int FS, int CS>
__global__ void __launch_bounds__(128, MinBlocks<Prop<FS>>::value)
fp64_chunk_kernel(const __grid_constant__ DevPlan P, DevState s, uint64_t n, int lanes, int max_steps, uint64_t step_cap,
                   DevCounters *cnt, DevRecords rec, const uint32_t *perm, uint32_t *perm_out) {
    chunk_body<Prop<FS>, CS>(P, s, n, lanes, max_steps, step_cap, cnt, rec, perm, perm_out);
}

template <template <int> class Prop, int FS, int CS>
__global__ void __launch_bounds__(128, MinBlocks<Prop<FS>>::value) fp64_persistent_kernel(
    const __grid_constant__ DevPlan P, DevState s, PersistentArgs a, DevCounters *cnt, DevRecords rec) {
    // the queue is written only between launches (advance_kernel)
    const DevQueue q = *a.q;
    const uint32_t *pending_in = q.cur ? a.list_b : a.list_a;
    uint32_t *pending_out = q.cur ? a.list_a : a.list_b;
    persistent_body<Prop<FS>, CS>(P, s, pending_in, q.n_pending, q.main_base, q.n_main, pending_out,
                              a.burst, a.refill, a.budget_ns, a.step_cap, cnt, rec);
}

// The kernel of a field signature and chain shape: compiled chain shapes for
// the single-field signatures (galactic fields: the backtracking chain
// [propagation, MaximumTrajectoryLength, Observer]); otherwise the module list is
// walked.
template <class F>
void for_signature(int fs, int shape, F f) {
    using std::integral_constant;
    integral_constant<int, CS_PM> pm;
    integral_constant<int, CS_PMO> pmo;
    integral_constant<int, CS_GENERIC> any;
    if (fs == FS_GRID_PERIODIC) {
        integral_constant<int, FS_GRID_PERIODIC> s;
        if (shape == CS_PM) f(s, pm);
        else if (shape == CS_PMO) f(s, pmo);
        else f(s, any);
    } else if (fs == FS_GRID) {
        f(integral_constant<int, FS_GRID>(), any);
    } else if (fs == FS_PLANE_WAVE) {
        integral_constant<int, FS_PLANE_WAVE> s;
        if (shape == CS_PM) f(s, pm);
        else if (shape == CS_PMO) f(s, pmo);
        else f(s, any);
    } else if (fs == FS_GALACTIC) {
        integral_constant<int, FS_GALACTIC> s;
        if (shape == CS_PMO) f(s, pmo);
        else f(s, any);
    } else {
        f(integral_constant<int, FS_GENERIC>(), any);
    }
}

// The boris_body kernel, 4 resident blocks of 128 threads per SM: bound by the
// latency of dependent FP64 operations, which 116 registers hold without spills
// (200 001 candidates x 1000 steps over 256^3 cells: 6.85 ms for the chain kernel
// with its divisions, here 4.20 ms at 4 blocks, 4.31 at 5, 4.58 at 6; 20 011
// candidates x 1500 steps over 64^3: 3.54 ms, then 1.49, 1.55 and 1.98 ms).
constexpr int kBorisMinBlocks = 4;
template <class Push>
__global__ void __launch_bounds__(128, Push::kAhead ? 4 : kBorisMinBlocks)
fp64_boris_kernel(const __grid_constant__ DevPlan P, DevState s, uint64_t n, int lanes, int max_steps, uint64_t step_cap,
                   DevCounters *cnt, DevRecords rec, const uint32_t *perm, uint32_t *perm_out) {
    boris_body<Push, BPFixed<FS_GRID_PERIODIC>>(P, s, n, lanes, max_steps, step_cap, cnt, rec, perm, perm_out);
}

// Kernels of FS_PLANE_WAVE_BLOCK: the mode table staged in dynamic shared memory.
template <template <int> class Prop, int CS>
__global__ void __launch_bounds__(kBatchThreads, wave_blocks(true, Prop<FS_PLANE_WAVE_BLOCK>::kCashKarp))
fp64_wave_kernel(const __grid_constant__ DevPlan P, DevState s, uint64_t n, int max_steps, uint64_t step_cap,
                  DevCounters *cnt, DevRecords rec, const uint32_t *perm, uint32_t *perm_out) {
    extern __shared__ __align__(16) unsigned char pw_table[];
    stage_wave_table(P.fields[0].pw, pw_table);
    __syncthreads();
    chunk_block_body<Prop<FS_PLANE_WAVE_BLOCK>, CS>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out);
}

template <template <int> class Prop>
cudaError_t launch_waves(DevPlan P, const DevState &s, uint64_t n, int max_steps, uint64_t step_cap, DevCounters *cnt,
                         const DevRecords &rec, const uint32_t *perm, uint32_t *perm_out, int warps, cudaStream_t st) {
    P.block_warps = warps;
    const size_t smem = wave_table_bytes(P.fields[0].pw);
    const unsigned grid = (unsigned)((n + 32 * warps - 1) / (32 * warps));
    auto launch = [&](auto c) {
        auto kernel = fp64_wave_kernel<Prop, decltype(c)::value>;
        const cudaError_t e = allow_shared<(size_t)kWaveMaxModesFp64 * 72>(kernel);
        if (e != cudaSuccess) return e;
        kernel<<<grid, kBatchThreads, smem, st>>>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out);
        return cudaGetLastError();
    };
    if (P.shape == CS_PM) return launch(std::integral_constant<int, CS_PM>());
    if (P.shape == CS_PMO) return launch(std::integral_constant<int, CS_PMO>());
    return launch(std::integral_constant<int, CS_GENERIC>());
}

template <template <int> class Prop>
cudaError_t launch_prop(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                        uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                        const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                        cudaStream_t st) {
    if constexpr (Prop<FS_PLANE_WAVE>::kBlockField) {
        const int warps =
            fs == FS_PLANE_WAVE
                ? wave_block_warps(n, P.fields[0].pw.n, P.num_sms, true, Prop<FS_PLANE_WAVE>::kCashKarp, P.shape == CS_PM)
                : 0;
        if (warps) return launch_waves<Prop>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, warps, st);
    }
    const uint64_t slots = (uint64_t)(block / 32) * (uint64_t)lanes;
    const unsigned grid = (unsigned)((n + slots - 1) / slots);
    for_signature(fs, P.shape, [&](auto f, auto c) {
        constexpr int FS = decltype(f)::value, CS = decltype(c)::value;
        // (fp64_boris_kernel takes these)
        if constexpr (!(Prop<FS>::kBorisKernel && FS == FS_GRID_PERIODIC && CS == CS_PM))
            fp64_chunk_kernel<Prop, FS, CS><<<grid, block, 0, st>>>(P, s, n, lanes, max_steps, step_cap, cnt, rec, perm,
                                                                     perm_out);
    });
    return cudaGetLastError();
}

template <template <int> class Prop>
cudaError_t launch_persistent_prop(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                   DevCounters *cnt, const DevRecords &rec, int fs, int grid,
                                   cudaStream_t st) {
    for_signature(fs, P.shape, [&](auto f, auto c) {
        fp64_persistent_kernel<Prop, decltype(f)::value, decltype(c)::value><<<grid, 128, 0, st>>>(P, s, a, cnt, rec);
    });
    return cudaGetLastError();
}

}  // namespace
}  // namespace crp
