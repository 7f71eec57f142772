// Lagrangian particle advance (m_particles.f90:815-1230, 1451-1508): trilinear or
// 4-point cubic (CINT) interpolation of the level-n physical velocity, then
// Adams-Bashforth 2 (Euler on the first step) in grid units.  The whole field is
// resident, so the reference's slab halos and migration are periodic wrap-around.
#pragma once
#include "common.cuh"

struct PartArgs {
    int n;
    int scheme;               // 0 trilinear, 1 CINT
    int64_t np;
    double dt, dx;
    const double *U;          // physical u,v,w: [f][z][y][x], row pitch rp, field stride fs
    int64_t fs, rp;
    double *xyz, *uvw;        // (np, 3) each, particle-major as xyzp(3,np)
};

H3D_D void cint_r(double x, double *r)
{
    double s = (x - 1.0) * (x - 2.0);
    r[0] = -x * s;
    r[1] = 3.0 * (x + 1.0) * s;
    s = (x + 1.0) * x;
    r[2] = -3.0 * s * (x - 2.0);
    r[3] = s * (x - 1.0);
}

// Four lanes per particle, eight particles per warp.  The gather is what costs:
// a stencil row is four (CINT) or two (trilinear) adjacent values, 32 bytes in
// one or two sectors, so each lane takes one x of the stencil and walks the rows
// of the three components: one load instruction touches 8 to 16 sectors a warp,
// where a lane per component walking whole stencils touched 30.  10^6 CINT
// particles at 256^3: 0.45 ms against 0.66.  Each lane sums its column over the rows,
// two shuffles add the columns, and lanes 0..2 advance one coordinate each.
// Every coordinate and the first-step flag V[0] are read before any lane of the
// particle writes (__syncwarp between).
constexpr int kPartPerWarp = 8;

__global__ void __launch_bounds__(256) k_particles(const PartArgs a)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t p = warp * kPartPerWarp + (lane >> 2);
    const int c = lane & 3;
    const bool active = p < a.np;
    const int n = a.n;
    double *X = a.xyz + 3 * p, *V = a.uvw + 3 * p;
    double x0 = 1.0, y0 = 1.0, z0 = 1.0, v0 = 0.0, vc = 0.0;
    if (active) {
        x0 = X[0]; y0 = X[1]; z0 = X[2];
        v0 = V[0];
        if (c < 3) vc = V[c];
    }
    __syncwarp();
    int i = (int)floor(x0), j = (int)floor(y0), k = (int)floor(z0);
    double xp = x0 - (double)i, yp = y0 - (double)j, zp = z0 - (double)k;
    // keep every cell index inside [1, n]: a coordinate that landed exactly on
    // n+1 (fraction 1.0 after a step) would otherwise read past the field
    i = ((i - 1) % n + n) % n + 1;
    j = ((j - 1) % n + n) % n + 1;
    k = ((k - 1) % n + n) % n + 1;
    // 0-based periodic index of cell t (1-based) + d, -1 <= d <= 2
    auto wrap = [n](int t, int d) {
        const int q = t - 1 + d;
        return q < 0 ? q + n : q >= n ? q - n : q;
    };
    double s[3] = {0.0, 0.0, 0.0};
    if (a.scheme == 0) {
        // lane c: x offset c & 1, y offset c >> 1
        const int dx = c & 1, dy = c >> 1;
        const double w = (dx ? xp : 1.0 - xp) * (dy ? yp : 1.0 - yp);
        const double *f = a.U + wrap(i, dx) + a.rp * (int64_t)wrap(j, dy);
#pragma unroll
        for (int dz = 0; dz < 2; dz++) {
            const double wz = w * (dz ? zp : 1.0 - zp);
            const double *g = f + a.rp * n * (int64_t)wrap(k, dz);
#pragma unroll
            for (int d = 0; d < 3; d++) s[d] += wz * g[d * a.fs];
        }
    } else {
        double rx[4], ry[4], rz[4];
        cint_r(xp, rx);
        cint_r(yp, ry);
        cint_r(zp, rz);
        const double wx = (c == 0 ? rx[0] : c == 1 ? rx[1] : c == 2 ? rx[2] : rx[3]) / 216.0;
        const double *f = a.U + wrap(i, c - 1);
        int64_t oy[4];
#pragma unroll
        for (int q = 0; q < 4; q++) oy[q] = a.rp * (int64_t)wrap(j, q - 1);
#pragma unroll
        for (int kq = 0; kq < 4; kq++) {
            const double *g = f + a.rp * n * (int64_t)wrap(k, kq - 1);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                double t = ry[0] * g[oy[0] + d * a.fs];
#pragma unroll
                for (int q = 1; q < 4; q++) t += ry[q] * g[oy[q] + d * a.fs];
                s[d] += rz[kq] * t;
            }
        }
#pragma unroll
        for (int d = 0; d < 3; d++) s[d] *= wx;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        s[d] += __shfl_xor_sync(0xffffffffu, s[d], 1);
        s[d] += __shfl_xor_sync(0xffffffffu, s[d], 2);
    }
    if (!active || c == 3) return;
    const double up = c == 0 ? s[0] : c == 1 ? s[1] : s[2];
    const double dx = a.dx, dt = a.dt;
    // this lane's coordinate: fraction and 1-based cell
    double fr = c == 0 ? xp : c == 1 ? yp : zp;
    int cell = c == 0 ? i : c == 1 ? j : k;
    if (v0 == -999.0) fr = fr + dt * up / dx;
    else fr = fr + (1.50 * up - 0.50 * vc) * dt / dx;
    V[c] = up;
    if (c < 2) {
        if (fr > 1.0) { fr = fr - 1.0; cell = cell + 1; if (cell > n) cell = cell - n; }
        if (fr < 0.0) { fr = fr + 1.0; cell = cell - 1; if (cell < 1) cell = cell + n; }
        X[c] = fr + (double)cell;
    } else {
        if (fr > 1.0) { fr = fr - 1.0; cell = cell + 1; }
        if (fr < 0.0) { fr = fr + 1.0; cell = cell - 1; }
        double zn = fr + (double)cell;
        // migration between slabs on one periodic slab (m_particles.f90:1270-1319)
        if (zn >= (double)(n + 1)) zn = zn - (double)n;
        else if (zn < 1.0) zn = zn + (double)n;
        X[2] = zn;
    }
}

// CTAs of 256 threads for np particles (eight per warp)
inline unsigned particle_blocks(int64_t np)
{
    const int64_t warps = (np + kPartPerWarp - 1) / kPartPerWarp;
    return (unsigned)((warps * 32 + 255) / 256);
}
