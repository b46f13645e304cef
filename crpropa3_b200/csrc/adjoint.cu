// adjoint.cu -- reverse-mode derivative of the fixed-step Boris push over a
// Grid3f (no reference counterpart; the forward step is
// PropagationBP::dY, PropagationBP.cpp:19, with the grid values taken as
// doubles and double trilinear weights in the corner order of Grid.h:571,
// then the direction normalised).
//
// Loss: L = sum_i (1 - u_final,i . target_i).  Gradients with respect to the
// initial directions, the energies and every grid value.
//
// One thread per candidate.  The forward pass stores the state (x, u) every
// K steps (checkpoints, FP64, in the caller's workspace).  The reverse pass
// walks the segments backwards: it recomputes one segment's K states from its
// checkpoint into thread-local memory and applies the adjoint of each step
// (normalisation, second half drift, Boris rotation, rotation vectors,
// field interpolation, first half drift).  The grid gradient is scattered
// with 64-bit integer atomics on fixed-point values (scale 2^36 / max kappa,
// kappa = q h c / 2E): integer addition is associative, so the result does
// not depend on the order the atomics land in.  Divisions are reciprocal
// multiplies and multiply-adds are contracted, so results agree with the
// oracle's CPU adjoint (which divides) to rounding, not bit for bit.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>

#include "crp_gpu.h"
#include "engine_internal.h"

namespace crp {
void set_last_error(const char *msg);
}

using namespace crp;

namespace {

constexpr int kMaxK = 128;
constexpr double kC = 2.99792458e8;

struct v3 { double x, y, z; };
__device__ __forceinline__ v3 mk(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ v3 add(v3 a, v3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ v3 muls(v3 a, double f) { return {a.x * f, a.y * f, a.z * f}; }
__device__ __forceinline__ double dot(v3 a, v3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

struct AdjGrid {
    const float *g;
    int nx, ny, nz;
    bool pow2;  // every dimension a power of two: indices wrap with a mask
    double gox, goy, goz;
    double isx, isy, isz;  // 1 / spacing
};

// Grids below this take 32-bit linear indices (3 * cell + component < 2^32).
constexpr size_t kSmallGrid = (size_t)1 << 30;

// periodic index: i mod n in [0, n) (a mask for power-of-two n, the same value)
__device__ __forceinline__ int wrap_index(int i, int n, bool pow2) {
    return pow2 ? (i & (n - 1)) : ((i % n) + n) % n;
}

// A candidate's position on the grid: the lower corner's index and the
// linear fraction on each axis.
struct CellPos {
    int lo[3];
    double f[3];
};

// floor(r) of |r| < 2^31 as integer and double without the conversion unit:
// adding 1.5 * 2^52 towards minus infinity leaves floor(r) in the low mantissa
// bits.  (The conversions and roundings of FP64 run at a quarter of the FP64
// rate on sm_100, and the corner loads need 24 of them per step already.)
__device__ __forceinline__ CellPos locate(const AdjGrid &G, v3 x) {
    const double magic = 6755399441055744.0;
    const double r[3] = {__dmul_rn(x.x - G.gox, G.isx), __dmul_rn(x.y - G.goy, G.isy), __dmul_rn(x.z - G.goz, G.isz)};
    const int n[3] = {G.nx, G.ny, G.nz};
    CellPos c;
    int i[3];
    const int big = max(max(__double2hiint(r[0]) & 0x7fffffff, __double2hiint(r[1]) & 0x7fffffff),
                        __double2hiint(r[2]) & 0x7fffffff);
    if (big < 0x41e00000) {  // every |r| < 2^31
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double t = __dadd_rd(r[a], magic);
            i[a] = __double2loint(t);
            c.f[a] = r[a] - (t - magic);
        }
    } else {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double fl = floor(r[a]);
            i[a] = (int)fl;
            c.f[a] = r[a] - fl;
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) c.lo[a] = wrap_index(i[a], n[a], G.pow2);
    return c;
}

// corner q of the Grid.h:571 order: which of lower / upper on each axis
__device__ __forceinline__ constexpr int bit(int q, int a) {
    constexpr int t[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 0}, {1, 1, 1}};
    return t[q][a];
}

// linear indices of the 8 corners
template <class Index>
__device__ __forceinline__ void corner_indices(const AdjGrid &G, const int lo[3], Index idx[8]) {
    const Index sx = (Index)G.ny * (Index)G.nz, sy = (Index)G.nz;
    const Index x0 = (Index)lo[0] * sx, x1 = lo[0] + 1 == G.nx ? 0 : x0 + sx;
    const Index y0 = (Index)lo[1] * sy, y1 = lo[1] + 1 == G.ny ? 0 : y0 + sy;
    const Index z0 = (Index)lo[2], z1 = lo[2] + 1 == G.nz ? 0 : z0 + 1;
#pragma unroll
    for (int q = 0; q < 8; q++) idx[q] = (bit(q, 0) ? x1 : x0) + (bit(q, 1) ? y1 : y0) + (bit(q, 2) ? z1 : z0);
}

// The 8 corner values of the cell a candidate is in, held in registers: at
// 1 kpc per step through 10 kpc cells a candidate leaves its cell on every
// seventh step or so, and without the cache each step's 24 loads of every lane
// bound the forward kernel (L1 wavefronts; lg_throttle 4.9 and long_scoreboard
// 8.1 cycles per issued instruction, 7.0 ms of 10^5 candidates x 2000 steps).
struct Corners {
    int lo[3];
    float v[8][3];
};

template <class Index>
__device__ __forceinline__ void load_corners(const AdjGrid &G, const CellPos &c, Corners &k) {
    if (c.lo[0] == k.lo[0] && c.lo[1] == k.lo[1] && c.lo[2] == k.lo[2]) return;
    Index idx[8];
    corner_indices(G, c.lo, idx);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float *g = G.g + 3 * idx[q];
        k.v[q][0] = __ldg(g); k.v[q][1] = __ldg(g + 1); k.v[q][2] = __ldg(g + 2);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) k.lo[a] = c.lo[a];
}

__device__ __forceinline__ void weights(const CellPos &c, double w[8]) {
    const double x0 = c.f[0], y0 = c.f[1], z0 = c.f[2], x1 = 1 - x0, y1 = 1 - y0, z1 = 1 - z0;
    const double a = x1 * y1, b = x0 * y1, d = x1 * y0, e = x0 * y0;
    w[0] = a * z1; w[1] = b * z1; w[2] = d * z1; w[3] = a * z0;
    w[4] = b * z0; w[5] = d * z0; w[6] = e * z1; w[7] = e * z0;
}

__device__ __forceinline__ v3 interpolate(const Corners &k, const double w[8]) {
    v3 B = mk(0, 0, 0);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        B.x = fma(w[q], (double)k.v[q][0], B.x);
        B.y = fma(w[q], (double)k.v[q][1], B.y);
        B.z = fma(w[q], (double)k.v[q][2], B.z);
    }
    return B;
}

// 1 / D for D = 1 + |t|^2 >= 1 by Newton's iteration from the single-precision
// reciprocal (relative error 2^-23 -> 2^-46 -> below 2^-52); D beyond the
// single-precision range (|t| > 10^19, no physical step) divides.
__device__ __forceinline__ double reciprocal(double D) {
    if (!(D < 1e38)) return 1 / D;
    double y = (double)__frcp_rn((float)D);
    y = fma(y, fma(-D, y, 1.0), y);
    return fma(y, fma(-D, y, 1.0), y);
}

// 1 / |u| from n2 = |u|^2.  The Boris rotation preserves |u|, so after the
// first step n2 is 1 within rounding and one Newton step of 1/sqrt from 1 is
// exact to rounding (error 3/8 (n2 - 1)^2).
__device__ __forceinline__ double inverse_norm(double n2) {
    if (fabs(n2 - 1) > 1e-9) return 1 / sqrt(n2);
    return fma(-0.5, n2, 1.5);
}

// a x v and its sum with c, multiply-adds written out: the forward pass and
// the reverse pass's recomputation have to agree bit for bit.
__device__ __forceinline__ v3 cross_add(v3 c, v3 a, v3 v) {
    return mk(fma(-v.y, a.z, fma(a.y, v.z, c.x)), fma(-v.z, a.x, fma(a.z, v.x, c.y)),
              fma(-v.x, a.y, fma(a.x, v.y, c.z)));
}
__device__ __forceinline__ double dotf(v3 a, v3 b) { return fma(a.x, b.x, fma(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ v3 axpy(v3 a, double f, v3 c) { return mk(fma(a.x, f, c.x), fma(a.y, f, c.y), fma(a.z, f, c.z)); }

// The Boris rotation of u0 in the field B: u2 = u0 + v x s.
struct Rotation {
    v3 t, s, v, u2;
    double iD;
};

__device__ __forceinline__ Rotation rotate(v3 u0, v3 B, double kappa) {
    Rotation r;
    r.t = muls(B, kappa);
    r.iD = reciprocal(fma(r.t.x, r.t.x, fma(r.t.y, r.t.y, fma(r.t.z, r.t.z, 1.0))));
    r.s = muls(r.t, 2 * r.iD);
    r.v = cross_add(u0, u0, r.t);
    r.u2 = cross_add(u0, r.v, r.s);
    return r;
}

template <class Index>
__device__ __forceinline__ void step(const AdjGrid &G, Corners &k, v3 &x, v3 &u, double hh, double kappa) {
    const v3 x1 = axpy(u, hh, x);
    const CellPos c = locate(G, x1);
    load_corners<Index>(G, c, k);
    double w[8];
    weights(c, w);
    const Rotation r = rotate(u, interpolate(k, w), kappa);
    x = axpy(r.u2, hh, x1);
    u = muls(r.u2, inverse_norm(dotf(r.u2, r.u2)));
}

struct IO {
    uint64_t n;
    const double *x, *y, *z, *dx, *dy, *dz, *energy, *charge, *tx, *ty, *tz;
    double *loss, *ux, *uy, *uz, *gdx, *gdy, *gdz, *ge;
};

__global__ void kappa_max_kernel(IO io, double h, unsigned long long *kmax) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double k = 0;
    if (i < io.n) k = fabs(io.charge[i] * h * kC / (2 * io.energy[i]));
    unsigned long long b = __double_as_longlong(k);  // non-negative doubles order as integers
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long ob = __shfl_xor_sync(0xffffffffu, b, o);
        b = ob > b ? ob : b;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(kmax, b);
}

// forward pass; with ckpt != null the state before every K-th step is stored.
// Blocks of 64: 10^5 candidates are 1563 blocks, which fill the 148 SMs more
// evenly than 782 blocks of 128.
constexpr int kForwardBlock = 64, kReverseBlock = 64;

template <class Index>
__global__ void __launch_bounds__(kForwardBlock, 10) forward_kernel(AdjGrid G, IO io, double h, int n_steps, int K,
                                                                    double *ckpt) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= io.n) return;
    const double kappa = io.charge[i] * h * kC / (2 * io.energy[i]);
    const double hh = h / 2;
    v3 x = mk(io.x[i], io.y[i], io.z[i]), u = mk(io.dx[i], io.dy[i], io.dz[i]);
    const uint64_t n = io.n;
    Corners corners;
    corners.lo[0] = -1;
    const int every = ckpt ? K : n_steps;
    for (int k0 = 0; k0 < n_steps; k0 += every) {
        if (ckpt) {
            double *c = ckpt + (size_t)(k0 / K) * 6 * n;
            c[i] = x.x; c[n + i] = x.y; c[2 * n + i] = x.z;
            c[3 * n + i] = u.x; c[4 * n + i] = u.y; c[5 * n + i] = u.z;
        }
        const int m = n_steps - k0 < every ? n_steps - k0 : every;
        for (int k = 0; k < m; k++) step<Index>(G, corners, x, u, hh, kappa);
    }
    io.loss[i] = 1 - dot(u, mk(io.tx[i], io.ty[i], io.tz[i]));
    if (io.ux) { io.ux[i] = u.x; io.uy[i] = u.y; io.uz[i] = u.z; }
}

// Add one cell's summed contributions to the fixed-point accumulator: g times
// scale rounded to an integer.  `most` bounds every |g|: where the integers
// stay below 2^50 the rounding is one multiply-add onto 1.5 * 2^52 and the
// integer its low mantissa bits (24 FP64-to-integer conversions per flush
// occupied the conversion unit longer than the multiply-adds do).
template <class Index>
__device__ __forceinline__ void flush(const AdjGrid &G, unsigned long long *acc, const int lo[3], double g[8][3],
                                      double scale, double &most) {
    if (lo[0] >= 0) {
        Index idx[8];
        corner_indices(G, lo, idx);
        if (most * scale < 1125899906842624.0) {
#pragma unroll
            for (int q = 0; q < 8; q++)
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const double t = fma(g[q][a], scale, 6755399441055744.0);
                    atomicAdd(acc + (3 * idx[q] + a), (unsigned long long)__double_as_longlong(t) - 0x4338000000000000ull);
                }
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++)
#pragma unroll
                for (int a = 0; a < 3; a++)
                    atomicAdd(acc + (3 * idx[q] + a), (unsigned long long)__double2ll_rn(g[q][a] * scale));
        }
    }
#pragma unroll
    for (int q = 0; q < 8; q++) g[q][0] = g[q][1] = g[q][2] = 0;
    most = 0;
}

// Bound by the issue and latency of some 620 instructions per step (250 of
// them FP64) at the warps its registers allow: 6 blocks of 64 (168 registers,
// of which 72 hold the cell's corners and gradient sums).  Measured over 10^5
// candidates x 2000 steps, 128^3 grid, checkpoints every 100, forward and
// reverse kernels with their Python wrapper: 27.0 ms before the corner cache,
// Newton reciprocals and FP64-to-integer rounding by addition; 19.1 ms now
// (forward pass 8.5 -> 3.6 ms); 25.2 ms at 8 blocks (128 registers, 656 B of
// spills), 19.5 ms at 5.  A copy of the grid in pair records (a cell and its upper
// z neighbour in 32 bytes, four wide loads per cell) gave another 1 % here, but cost
// 44 B per cell of traffic on every tape: 0.43 -> 1.51 ms for 1000 candidates x 100
// steps through 512^3 cells.
constexpr int kReverseMinBlocks = 6;
template <class Index>
__global__ void __launch_bounds__(kReverseBlock, kReverseMinBlocks) reverse_kernel(AdjGrid G, IO io, double h,
                                                      int n_steps, int K, const double *ckpt,
                                                      unsigned long long *acc,
                                                      const unsigned long long *kmax_bits) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= io.n) return;
    const uint64_t n = io.n;
    const double kappa = io.charge[i] * h * kC / (2 * io.energy[i]);
    const double hh = h / 2;
    const double kmax = __longlong_as_double((long long)*kmax_bits);
    const double scale = (acc && kmax > 0) ? ldexp(1.0 / kmax, 36) : 0.0;
    v3 xs[kMaxK], us[kMaxK];
    v3 xb = mk(0, 0, 0), ub = mk(-io.tx[i], -io.ty[i], -io.tz[i]);
    double kb = 0;
    // the cell the candidate is in: its corner values (shared by the
    // recomputation and the reverse steps), and the grid-gradient
    // contributions of the cell glo, summed in registers and flushed with
    // atomics when the reverse steps leave it
    Corners corners;
    corners.lo[0] = -1;
    int glo[3] = {-1, -1, -1};
    double gacc[8][3], most = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) gacc[q][0] = gacc[q][1] = gacc[q][2] = 0;
    const int nseg = (n_steps + K - 1) / K;
    for (int j = nseg - 1; j >= 0; j--) {
        const double *c = ckpt + (size_t)j * 6 * n;
        const int m = (j * K + K < n_steps) ? K : n_steps - j * K;
        v3 x = mk(c[i], c[n + i], c[2 * n + i]), u = mk(c[3 * n + i], c[4 * n + i], c[5 * n + i]);
        // the states before each step of the segment (the last one stays in x
        // and u: checkpoint_every = 1 recomputes and stores nothing)
        for (int k = 0; k + 1 < m; k++) {
            xs[k] = x; us[k] = u;
            step<Index>(G, corners, x, u, hh, kappa);
        }
        for (int k = m - 1; k >= 0; k--) {
            const v3 u0 = u;
            const CellPos cp = locate(G, axpy(u0, hh, x));
            // the state before the previous step, asked for a step ahead
            if (k > 0) { x = xs[k - 1]; u = us[k - 1]; }
            if (acc && (cp.lo[0] != glo[0] || cp.lo[1] != glo[1] || cp.lo[2] != glo[2])) {
                flush<Index>(G, acc, glo, gacc, scale, most);
#pragma unroll
                for (int a = 0; a < 3; a++) glo[a] = cp.lo[a];
            }
            load_corners<Index>(G, cp, corners);
            double w[8];
            weights(cp, w);
            const v3 B = interpolate(corners, w);
            const Rotation r = rotate(u0, B, kappa);
            const double inn = inverse_norm(dotf(r.u2, r.u2));
            const v3 un = muls(r.u2, inn);
            // reverse of: normalisation, second half drift, Boris rotation
            v3 u2b = muls(axpy(un, -dotf(un, ub), ub), inn);
            u2b = axpy(xb, hh, u2b);
            const v3 vb = cross_add(mk(0, 0, 0), r.s, u2b);
            const v3 sb = cross_add(mk(0, 0, 0), u2b, r.v);
            const v3 ubar = cross_add(add(u2b, vb), r.t, vb);
            v3 tb = axpy(sb, 2 * r.iD, cross_add(mk(0, 0, 0), vb, u0));
            tb = axpy(r.t, -4 * dotf(r.t, sb) * (r.iD * r.iD), tb);
            const v3 Bb = muls(tb, kappa);
            most += fabs(Bb.x) + fabs(Bb.y) + fabs(Bb.z);
            kb = fma(tb.x, B.x, fma(tb.y, B.y, fma(tb.z, B.z, kb)));
            // reverse of the interpolation.  Grid values: weight times Bb.
            // Position: the gradient of the trilinear form of g_q = Bb . c_q by
            // differences and lerps, z first, corners g[x][y][z].
            double g[2][2][2];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                g[bit(q, 0)][bit(q, 1)][bit(q, 2)] =
                    fma(Bb.x, (double)corners.v[q][0],
                        fma(Bb.y, (double)corners.v[q][1], Bb.z * (double)corners.v[q][2]));
                gacc[q][0] = fma(w[q], Bb.x, gacc[q][0]);
                gacc[q][1] = fma(w[q], Bb.y, gacc[q][1]);
                gacc[q][2] = fma(w[q], Bb.z, gacc[q][2]);
            }
            double a[2], dy[2], dz[2];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const double z0 = g[p][0][1] - g[p][0][0], z1 = g[p][1][1] - g[p][1][0];
                const double h0 = fma(cp.f[2], z0, g[p][0][0]), h1 = fma(cp.f[2], z1, g[p][1][0]);
                dz[p] = fma(cp.f[1], z1 - z0, z0);
                dy[p] = h1 - h0;
                a[p] = fma(cp.f[1], dy[p], h0);
            }
            xb.x = fma(a[1] - a[0], G.isx, xb.x);
            xb.y = fma(fma(cp.f[0], dy[1] - dy[0], dy[0]), G.isy, xb.y);
            xb.z = fma(fma(cp.f[0], dz[1] - dz[0], dz[0]), G.isz, xb.z);
            ub = axpy(xb, hh, ubar);
        }
    }
    if (acc) flush<Index>(G, acc, glo, gacc, scale, most);
    io.gdx[i] = ub.x; io.gdy[i] = ub.y; io.gdz[i] = ub.z;
    io.ge[i] = kb * (-kappa / io.energy[i]);
}

__global__ void finalize_kernel(const unsigned long long *acc, uint64_t m,
                                const unsigned long long *kmax_bits, double *out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double kmax = __longlong_as_double((long long)*kmax_bits);
    out[i] = (double)(long long)acc[i] * ldexp(kmax, -36);
}

crp_status fail(crp_status st, const char *msg) {
    set_last_error(msg);
    return st;
}

crp_status cuda_fail(cudaError_t e, const char *what) {
    char buf[512];
    snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    set_last_error(buf);
    return e == cudaErrorMemoryAllocation ? CRP_ERR_OUT_OF_MEMORY : CRP_ERR_CUDA;
}

crp_status check_desc(const crp_adjoint_desc *d, const crp_adjoint_io *io) {
    if (!d || !io) return fail(CRP_ERR_INVALID_ARGUMENT, "NULL argument");
    if (!d->grid_values || !d->nx || !d->ny || !d->nz) return fail(CRP_ERR_INVALID_ARGUMENT, "Grid3f: empty grid");
    if (d->nx > (1u << 20) || d->ny > (1u << 20) || d->nz > (1u << 20))
        return fail(CRP_ERR_CAPACITY, "Grid3f: a dimension beyond 2^20 cells");
    if (!(d->step > 0)) return fail(CRP_ERR_INVALID_ARGUMENT, "step must be > 0");
    if (d->n_steps < 0) return fail(CRP_ERR_INVALID_ARGUMENT, "n_steps < 0");
    if (d->checkpoint_every < 1 || d->checkpoint_every > kMaxK)
        return fail(CRP_ERR_CAPACITY, "checkpoint_every must be 1..128");
    if (io->n && (!io->x || !io->y || !io->z || !io->dx || !io->dy || !io->dz || !io->energy ||
                  !io->charge || !io->tx || !io->ty || !io->tz || !io->loss))
        return fail(CRP_ERR_INVALID_ARGUMENT, "an input array is NULL");
    return CRP_OK;
}

AdjGrid make_grid(const crp_adjoint_desc *d) {
    AdjGrid G;
    G.g = d->grid_values;
    G.nx = (int)d->nx; G.ny = (int)d->ny; G.nz = (int)d->nz;
    auto p2 = [](uint64_t v) { return v && !(v & (v - 1)); };
    G.pow2 = p2(d->nx) && p2(d->ny) && p2(d->nz);
    G.gox = d->origin[0] + d->spacing[0] / 2;
    G.goy = d->origin[1] + d->spacing[1] / 2;
    G.goz = d->origin[2] + d->spacing[2] / 2;
    G.isx = 1.0 / d->spacing[0]; G.isy = 1.0 / d->spacing[1]; G.isz = 1.0 / d->spacing[2];
    return G;
}

IO make_io(const crp_adjoint_io *a) {
    IO io;
    io.n = a->n;
    io.x = a->x; io.y = a->y; io.z = a->z; io.dx = a->dx; io.dy = a->dy; io.dz = a->dz;
    io.energy = a->energy; io.charge = a->charge; io.tx = a->tx; io.ty = a->ty; io.tz = a->tz;
    io.loss = a->loss; io.ux = a->ux; io.uy = a->uy; io.uz = a->uz;
    io.gdx = a->grad_dx; io.gdy = a->grad_dy; io.gdz = a->grad_dz; io.ge = a->grad_energy;
    return io;
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

bool small_grid(const crp_adjoint_desc *d) { return (size_t)d->nx * d->ny * d->nz <= kSmallGrid; }

void launch_forward(const crp_adjoint_desc *d, const crp_adjoint_io *a, double *ckpt, cudaStream_t s) {
    auto forward = small_grid(d) ? forward_kernel<unsigned> : forward_kernel<size_t>;
    forward<<<(unsigned)((a->n + kForwardBlock - 1) / kForwardBlock), kForwardBlock, 0, s>>>(
        make_grid(d), make_io(a), d->step, d->n_steps, d->checkpoint_every, ckpt);
}

}  // namespace

extern "C" {

crp_status crp_bp_adjoint_workspace(const crp_adjoint_desc *d, uint64_t n, size_t *bytes) {
    if (!d || !bytes) return fail(CRP_ERR_INVALID_ARGUMENT, "NULL argument");
    if (d->checkpoint_every < 1 || d->checkpoint_every > kMaxK)
        return fail(CRP_ERR_CAPACITY, "checkpoint_every must be 1..128");
    const size_t nck = (size_t)((d->n_steps + d->checkpoint_every - 1) / d->checkpoint_every);
    const size_t cells = (size_t)d->nx * d->ny * d->nz;
    *bytes = align256(256) + align256(nck * 6 * n * sizeof(double)) + align256(cells * 3 * sizeof(unsigned long long));
    return CRP_OK;
}

crp_status crp_bp_forward_loss(const crp_adjoint_desc *d, const crp_adjoint_io *a, void *stream) {
    crp_status st = check_desc(d, a);
    if (st) return st;
    if (a->n == 0) return CRP_OK;
    launch_forward(d, a, nullptr, (cudaStream_t)stream);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CRP_OK : cuda_fail(e, "adjoint forward kernel launch");
}

static crp_status adjoint_impl(const crp_adjoint_desc *d, const crp_adjoint_io *a, void *workspace,
                               size_t workspace_bytes, void *stream, bool do_forward,
                               bool do_backward) {
    crp_status st = check_desc(d, a);
    if (st) return st;
    if (do_backward && (!a->grad_dx || !a->grad_dy || !a->grad_dz || !a->grad_energy))
        return fail(CRP_ERR_INVALID_ARGUMENT, "a gradient array is NULL");
    size_t need = 0;
    st = crp_bp_adjoint_workspace(d, a->n, &need);
    if (st) return st;
    if (!workspace || workspace_bytes < need) return fail(CRP_ERR_CAPACITY, "workspace smaller than crp_bp_adjoint_workspace");
    if (a->n == 0) return CRP_OK;
    cudaStream_t s = (cudaStream_t)stream;
    char *w = static_cast<char *>(workspace);
    unsigned long long *kmax = reinterpret_cast<unsigned long long *>(w);
    const size_t nck = (size_t)((d->n_steps + d->checkpoint_every - 1) / d->checkpoint_every);
    double *ckpt = reinterpret_cast<double *>(w + align256(256));
    const size_t cells3 = (size_t)d->nx * d->ny * d->nz * 3;
    unsigned long long *acc = reinterpret_cast<unsigned long long *>(w + align256(256) + align256(nck * 6 * a->n * sizeof(double)));
    const AdjGrid G = make_grid(d);
    const IO io = make_io(a);
    auto blocks = [&](unsigned threads) { return (unsigned)((a->n + threads - 1) / threads); };
    cudaError_t e = cudaSuccess;
    if (do_forward) {
        e = cudaMemsetAsync(kmax, 0, 8, s);
        if (e != cudaSuccess) return cuda_fail(e, "clearing the adjoint workspace");
        kappa_max_kernel<<<blocks(128), 128, 0, s>>>(io, d->step, kmax);
        launch_forward(d, a, ckpt, s);
    }
    if (do_backward) {
        if (a->grad_grid) {
            e = cudaMemsetAsync(acc, 0, cells3 * sizeof(unsigned long long), s);
            if (e != cudaSuccess) return cuda_fail(e, "clearing the adjoint workspace");
        }
        auto reverse = small_grid(d) ? reverse_kernel<unsigned> : reverse_kernel<size_t>;
        reverse<<<blocks(kReverseBlock), kReverseBlock, 0, s>>>(G, io, d->step, d->n_steps, d->checkpoint_every, ckpt,
                                                                a->grad_grid ? acc : nullptr, kmax);
        if (a->grad_grid)
            finalize_kernel<<<(unsigned)((cells3 + 255) / 256), 256, 0, s>>>(acc, cells3, kmax, a->grad_grid);
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? CRP_OK : cuda_fail(e, "adjoint kernel launch");
}

crp_status crp_bp_adjoint(const crp_adjoint_desc *d, const crp_adjoint_io *a, void *workspace,
                          size_t workspace_bytes, void *stream) {
    return adjoint_impl(d, a, workspace, workspace_bytes, stream, true, true);
}

crp_status crp_bp_adjoint_forward(const crp_adjoint_desc *d, const crp_adjoint_io *a, void *workspace,
                                  size_t workspace_bytes, void *stream) {
    return adjoint_impl(d, a, workspace, workspace_bytes, stream, true, false);
}

crp_status crp_bp_adjoint_backward(const crp_adjoint_desc *d, const crp_adjoint_io *a, void *workspace,
                                   size_t workspace_bytes, void *stream) {
    return adjoint_impl(d, a, workspace, workspace_bytes, stream, false, true);
}

}  // extern "C"
