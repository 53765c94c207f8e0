// 3-D acoustic staggered-grid step, 4th order
// (geobrain/physics/wave/kernels/acoustic_3d.py:20-300, driver :303-476).
//
// Per time step, for every shot:
//   p  <- (1 - k1) p - a1 (dvx/dx + dvy/dy + dvz/dz)        (ref :117-150)
//         on z [fs+1, Nz-2), y [2, Ny-2), x [2, Nx-2)
//   p[sz, sy, sx] += dt * w[s, it]                            (ref :153-163)
//   p[fs-1] = -p[fs+1]          free surface                  (ref :166-167)
//   vx <- (1 - k2) vx - a2 dp/dx   z [fs, Nz-1), y [1, Ny-1), x [1, Nx-2)
//   vy <- (1 - k3) vy - a2 dp/dy   z [fs, Nz-1), y [1, Ny-2), x [1, Nx-1)
//   vz <- (1 - k4) vz - a2 dp/dz   z [fs, Nz-2), y [1, Ny-1), x [1, Nx-1)
//                                                              (ref :170-233)
//   vz[fs-1] = vz[fs]                                          (ref :236-237)
//   traces[s, it, r] = (p, vx, vy, vz)[receiver r]             (ref :240-243)
//   energy += sum_s (p^2, vx^2, vy^2, vz^2) on the interior    (ref :246-258)
// with d/dq f = c1 (f[q] - f[q-1]) + c2 (f[q+1] - f[q-2]) at the staggered
// points, c1 = 9/8, c2 = -1/24, every operation rounded separately in the
// reference's order.
//
// Layout: [shot][p | vx | vy | vz][Nz][Ny][pitch] fp32 with pitch =
// roundup(Nx, 32); vx's last column, vy's last row and vz's last plane
// (absent in the reference) stay zero.  A thread owns 4 adjacent x cells
// of one (z, y) row and loops over the shots, so the coefficients are read
// once per step and the energy sums need no atomics.  Each update reads
// only the other fields and writes only its own, so both run in place.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gb {

struct Geo3 {
    int Nz, Ny, Nx, pitch;
    int nz, ny, nx, pml, fs;
    int n_shots, nt, n_rcv;
    float dt;
    long long plane;   // Ny * pitch
    long long vol;     // Nz * plane
};

// The shot loops below ask L2 for the next shot's cells of this thread while
// the current shot computes.  At 16-24 resident warps per SM the loads of one
// shot alone leave DRAM idle between shots; with the prefetch the 200^3,
// 4-shot forward runs 1.27x faster (the arithmetic is unchanged).  Every
// prefetched address is inside the state / imaging arrays.
__device__ __forceinline__ void prefetch_l2(const float *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

constexpr float kC1 = 9.0f / 8.0f;
constexpr float kC2 = -1.0f / 24.0f;

__device__ __forceinline__ float4 ld4z(const float *base, long long o, bool ok)
{
    return ok ? *reinterpret_cast<const float4 *>(base + o) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float f4(const float4 &v, int q)
{
    return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w;
}
// c1 (a - b) + c2 (c - d), rounded as the reference evaluates it
__device__ __forceinline__ float d4(float a, float b, float c, float d)
{
    return __fadd_rn(__fmul_rn(kC1, __fsub_rn(a, b)), __fmul_rn(kC2, __fsub_rn(c, d)));
}

// Coefficients from the unpadded vp / rho (edge-replicated padding as
// pad_model_3d, kernels/acoustic_2d.py:70-120) and the padded damping, in the
// reference's fp32 operation order (acoustic_3d.py:410-441).
__global__ void coef3_kernel(const Geo3 g, const float *__restrict__ vp, const float *__restrict__ rho,
                             const float *__restrict__ damp, float dz, float *a1, float *k1, float *a2, float *k2,
                             float *k3, float *k4)
{
    const long long n = (long long)g.Nz * g.Ny * g.Nx;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % g.Nx), y = (int)((i / g.Nx) % g.Ny), z = (int)(i / ((long long)g.Nx * g.Ny));
        const int zi = min(max(z - g.pml, 0), g.nz - 1), yi = min(max(y - g.pml, 0), g.ny - 1),
                  xi = min(max(x - g.pml, 0), g.nx - 1);
        const long long m = ((long long)zi * g.ny + yi) * g.nx + xi;
        const float c = vp[m], den = rho[m];
        const long long d = ((long long)z * g.Ny + y) * g.Nx + x;
        const long long o = (long long)z * g.plane + (long long)y * g.pitch + x;
        a1[o] = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(den, c), c), g.dt), dz);
        k1[o] = __fmul_rn(damp[d], g.dt);
        a2[o] = __fdiv_rn(g.dt, __fmul_rn(den, dz));
        k2[o] = (x >= 1 && x < g.Nx - 2) ? __fmul_rn(__fmul_rn(0.5f, __fadd_rn(damp[d], damp[d + 1])), g.dt) : 0.f;
        k3[o] = (y >= 1 && y < g.Ny - 2) ? __fmul_rn(__fmul_rn(0.5f, __fadd_rn(damp[d], damp[d + g.Nx])), g.dt)
                                         : 0.f;
        k4[o] = (z >= g.fs && z < g.Nz - 2)
                    ? __fmul_rn(__fmul_rn(0.5f, __fadd_rn(damp[d], damp[d + (long long)g.Nx * g.Ny])), g.dt)
                    : 0.f;
    }
}

struct Args3 {
    Geo3 g;
    int it;
    const int *step_base;                 // device step counter (graph replay) or null
    float *state;                         // [S][4][Nz][Ny][pitch]
    const float *a1, *k1, *a2, *k2, *k3, *k4;
    const int *src;                       // [3][S]: padded z, y, x
    const float *wavelet;                 // [S][nt]
    float *energy[4];                     // (nz, ny, nx) accumulators or null
    float *img_i;                         // gradient recompute: -(dvx+dvy+dvz) per p cell [S][vol], or null
    float *img_j;                         // and dp/dx, dp/dy, dp/dz per v cell [3][S][vol] (density), or null
};

__device__ __forceinline__ int step_of(const Args3 &A)
{
    return A.step_base ? *reinterpret_cast<const volatile int *>(A.step_base) + A.it : A.it;
}

// p update and source (block: 32 x-quads x 4 rows; grid: x-blocks, y-blocks, Nz).
// The register bounds of the four step kernels (8, 7, 4, 4 CTAs per SM) trade
// a few spilled bytes for resident warps; measured at 200^3 with 4 shots,
// the forward runs 7 % faster than at the compiler's own choice.
__global__ void __launch_bounds__(128, 8) p3_kernel(const Args3 A)
{
    const Geo3 &g = A.g;
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    const int y = blockIdx.y * 4 + threadIdx.y;
    const int z = blockIdx.z;
    if (x0 >= g.Nx || y >= g.Ny) return;
    const int it = step_of(A);
    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x0;
    const bool row_in = z >= g.fs + 1 && z < g.Nz - 2 && y >= 2 && y < g.Ny - 2 && x0 + 3 >= 2 && x0 < g.Nx - 2;
    float4 a1 = make_float4(0.f, 0.f, 0.f, 0.f), k1 = a1;
    if (row_in) {
        a1 = *reinterpret_cast<const float4 *>(A.a1 + o);
        k1 = *reinterpret_cast<const float4 *>(A.k1 + o);
    }
    // the p energy is complete once p is: the free-surface mirror plane
    // (fs - 1 = pml - 1) lies outside the interior
    const bool energy = A.energy[0] && z >= g.pml && z < g.pml + g.nz && y >= g.pml && y < g.pml + g.ny;
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < g.n_shots; ++s) {
        float *P = A.state + (long long)s * 4 * g.vol;
        const float *VX = P + g.vol, *VY = P + 2 * g.vol, *VZ = P + 3 * g.vol;
        if (s + 1 < g.n_shots) {
            const float *N = P + 4 * g.vol + o;
            prefetch_l2(N); prefetch_l2(N + g.vol); prefetch_l2(N + 2 * g.vol); prefetch_l2(N + 3 * g.vol);
        }
        float4 p = *reinterpret_cast<const float4 *>(P + o);
        if (row_in) {
            const float4 xl = ld4z(VX, o - 4, x0 >= 4), xc = ld4z(VX, o, true),
                         xr = ld4z(VX, o + 4, x0 + 4 < g.pitch);
            const float xs[12] = {xl.x, xl.y, xl.z, xl.w, xc.x, xc.y, xc.z, xc.w, xr.x, xr.y, xr.z, xr.w};
            const float4 ym2 = ld4z(VY, o - 2 * g.pitch, true), ym1 = ld4z(VY, o - g.pitch, true),
                         y0 = ld4z(VY, o, true), yp1 = ld4z(VY, o + g.pitch, true);
            const float4 zm2 = ld4z(VZ, o - 2 * g.plane, true), zm1 = ld4z(VZ, o - g.plane, true),
                         z0 = ld4z(VZ, o, true), zp1 = ld4z(VZ, o + g.plane, true);
            float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int x = x0 + q;
                if (x < 2 || x >= g.Nx - 2) continue;
                const float dvx = d4(xs[q + 4], xs[q + 3], xs[q + 5], xs[q + 2]);
                const float dvy = d4(f4(y0, q), f4(ym1, q), f4(yp1, q), f4(ym2, q));
                const float dvz = d4(f4(z0, q), f4(zm1, q), f4(zp1, q), f4(zm2, q));
                const float sum = __fadd_rn(__fadd_rn(dvx, dvy), dvz);
                pv[q] = __fsub_rn(__fmul_rn(__fsub_rn(1.f, f4(k1, q)), pv[q]), __fmul_rn(f4(a1, q), sum));
                if (A.img_i) A.img_i[(long long)s * g.vol + o + q] = -sum;
            }
            p = make_float4(pv[0], pv[1], pv[2], pv[3]);
        }
        const int sz = A.src[s], sy = A.src[g.n_shots + s], sx = A.src[2 * g.n_shots + s];
        if (sz == z && sy == y && sx >= x0 && sx < x0 + 4) {
            const float amp = __fmul_rn(g.dt, A.wavelet[(long long)s * g.nt + it]);
            const int q = sx - x0;
            if (q == 0) p.x = __fadd_rn(p.x, amp);
            else if (q == 1) p.y = __fadd_rn(p.y, amp);
            else if (q == 2) p.z = __fadd_rn(p.z, amp);
            else p.w = __fadd_rn(p.w, amp);
        }
        *reinterpret_cast<float4 *>(P + o) = p;
        if (energy) {
#pragma unroll
            for (int q = 0; q < 4; ++q) e[q] = __fadd_rn(e[q], __fmul_rn(f4(p, q), f4(p, q)));
        }
    }
    if (energy) {
        const long long eo = ((long long)(z - g.pml) * g.ny + (y - g.pml)) * g.nx - g.pml;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int x = x0 + q;
            if (x >= g.pml && x < g.pml + g.nx) A.energy[0][eo + x] = __fadd_rn(A.energy[0][eo + x], e[q]);
        }
    }
}

// Free-surface mirror plane of field f: f[fs-1] = sign * f[fs - 1 + from]
__global__ void mirror3_kernel(const Geo3 g, float *state, int field, int from, float sign)
{
    const long long n = (long long)g.n_shots * g.plane;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long s = i / g.plane, r = i % g.plane;
        float *F = state + (s * 4 + field) * g.vol;
        F[(long long)(g.fs - 1) * g.plane + r] = sign * F[(long long)(g.fs - 1 + from) * g.plane + r];
    }
}

// vx, vy, vz updates and their energy sums (same blocks as p3_kernel).  The
// planes run down where p3_kernel's run up, so that each kernel starts on
// planes the one before left in L2: 200^3, 4 shots, 30 steps 18.5 -> 18.2 ms,
// and with adj_v3_kernel the other way from adj_p3_kernel a 130 x 149 x 171
// gradient of 40 steps 24.4 -> 23.9.
__global__ void __launch_bounds__(128, 7) v3_kernel(const Args3 A)
{
    const Geo3 &g = A.g;
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    const int y = blockIdx.y * 4 + threadIdx.y;
    const int z = g.Nz - 1 - blockIdx.z;
    if (x0 >= g.Nx || y >= g.Ny) return;
    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x0;
    const bool zin = z >= g.fs && z < g.Nz - 1;
    const bool vx_row = zin && y >= 1 && y < g.Ny - 1;
    const bool vy_row = zin && y >= 1 && y < g.Ny - 2;
    const bool vz_row = z >= g.fs && z < g.Nz - 2 && y >= 1 && y < g.Ny - 1;
    const bool any = vx_row || vy_row || vz_row;
    float4 a2 = make_float4(0.f, 0.f, 0.f, 0.f), k2 = a2, k3 = a2, k4 = a2;
    if (any) {
        a2 = *reinterpret_cast<const float4 *>(A.a2 + o);
        k2 = *reinterpret_cast<const float4 *>(A.k2 + o);
        k3 = *reinterpret_cast<const float4 *>(A.k3 + o);
        k4 = *reinterpret_cast<const float4 *>(A.k4 + o);
    }
    const bool interior_row = z >= g.pml && z < g.pml + g.nz && y >= g.pml && y < g.pml + g.ny;
    const bool energy = interior_row && A.energy[0];
    float e[3][4] = {};
    for (int s = 0; s < g.n_shots; ++s) {
        float *P = A.state + (long long)s * 4 * g.vol;
        float *VX = P + g.vol, *VY = P + 2 * g.vol, *VZ = P + 3 * g.vol;
        if (s + 1 < g.n_shots) {
            const float *N = P + 4 * g.vol + o;
            prefetch_l2(N); prefetch_l2(N + g.vol); prefetch_l2(N + 2 * g.vol); prefetch_l2(N + 3 * g.vol);
        }
        const float4 pc = *reinterpret_cast<const float4 *>(P + o);
        float4 vx = *reinterpret_cast<const float4 *>(VX + o);
        float4 vy = *reinterpret_cast<const float4 *>(VY + o);
        float4 vz = *reinterpret_cast<const float4 *>(VZ + o);
        if (any) {
            const float4 pl = ld4z(P, o - 4, x0 >= 4), pr = ld4z(P, o + 4, x0 + 4 < g.pitch);
            const float ps[12] = {pl.x, pl.y, pl.z, pl.w, pc.x, pc.y, pc.z, pc.w, pr.x, pr.y, pr.z, pr.w};
            float rx[4] = {vx.x, vx.y, vx.z, vx.w}, ry[4] = {vy.x, vy.y, vy.z, vy.w}, rz[4] = {vz.x, vz.y, vz.z, vz.w};
            if (vx_row) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int x = x0 + q;
                    if (x < 1 || x >= g.Nx - 2) continue;
                    const float dp = d4(ps[q + 5], ps[q + 4], ps[q + 6], ps[q + 3]);
                    rx[q] = __fsub_rn(__fmul_rn(__fsub_rn(1.f, f4(k2, q)), rx[q]), __fmul_rn(f4(a2, q), dp));
                    if (A.img_j) A.img_j[(long long)s * g.vol + o + q] = dp;
                }
            }
            if (vy_row) {
                const float4 ym1 = ld4z(P, o - g.pitch, true), yp1 = ld4z(P, o + g.pitch, true),
                             yp2 = ld4z(P, o + 2 * g.pitch, true);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int x = x0 + q;
                    if (x < 1 || x >= g.Nx - 1) continue;
                    const float dp = d4(f4(yp1, q), f4(pc, q), f4(yp2, q), f4(ym1, q));
                    ry[q] = __fsub_rn(__fmul_rn(__fsub_rn(1.f, f4(k3, q)), ry[q]), __fmul_rn(f4(a2, q), dp));
                    if (A.img_j) A.img_j[((long long)g.n_shots + s) * g.vol + o + q] = dp;
                }
            }
            if (vz_row) {
                const float4 zm1 = ld4z(P, o - g.plane, true), zp1 = ld4z(P, o + g.plane, true),
                             zp2 = ld4z(P, o + 2 * g.plane, true);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int x = x0 + q;
                    if (x < 1 || x >= g.Nx - 1) continue;
                    const float dp = d4(f4(zp1, q), f4(pc, q), f4(zp2, q), f4(zm1, q));
                    rz[q] = __fsub_rn(__fmul_rn(__fsub_rn(1.f, f4(k4, q)), rz[q]), __fmul_rn(f4(a2, q), dp));
                    if (A.img_j) A.img_j[(2LL * g.n_shots + s) * g.vol + o + q] = dp;
                }
            }
            vx = make_float4(rx[0], rx[1], rx[2], rx[3]);
            vy = make_float4(ry[0], ry[1], ry[2], ry[3]);
            vz = make_float4(rz[0], rz[1], rz[2], rz[3]);
            *reinterpret_cast<float4 *>(VX + o) = vx;
            *reinterpret_cast<float4 *>(VY + o) = vy;
            *reinterpret_cast<float4 *>(VZ + o) = vz;
        }
        if (energy) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                e[0][q] = __fadd_rn(e[0][q], __fmul_rn(f4(vx, q), f4(vx, q)));
                e[1][q] = __fadd_rn(e[1][q], __fmul_rn(f4(vy, q), f4(vy, q)));
                e[2][q] = __fadd_rn(e[2][q], __fmul_rn(f4(vz, q), f4(vz, q)));
            }
        }
    }
    if (energy) {
        // this thread is the only writer of these cells
        const long long eo = ((long long)(z - g.pml) * g.ny + (y - g.pml)) * g.nx;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int x = x0 + q;
            if (x < g.pml || x >= g.pml + g.nx) continue;
            for (int f = 0; f < 3; ++f)
                A.energy[f + 1][eo + x - g.pml] = __fadd_rn(A.energy[f + 1][eo + x - g.pml], e[f][q]);
        }
    }
}

// Receivers: traces[f][s][it][r] = field f at the receiver (padded z, y, x)
__global__ void rec3_kernel(const Geo3 g, const float *state, const int *rcv, float *tr_p, float *tr_vx,
                            float *tr_vy, float *tr_vz, int it, const int *step_base)
{
    const long long n = (long long)g.n_shots * g.n_rcv;
    if (step_base) it += *reinterpret_cast<const volatile int *>(step_base);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(i / g.n_rcv), r = (int)(i % g.n_rcv);
        const long long o = (long long)rcv[r] * g.plane + (long long)rcv[g.n_rcv + r] * g.pitch + rcv[2 * g.n_rcv + r];
        const float *P = state + (long long)s * 4 * g.vol;
        const long long t = ((long long)s * g.nt + it) * g.n_rcv + r;
        if (tr_p) tr_p[t] = P[o];
        if (tr_vx) tr_vx[t] = P[g.vol + o];
        if (tr_vy) tr_vy[t] = P[2 * g.vol + o];
        if (tr_vz) tr_vz[t] = P[3 * g.vol + o];
    }
}

// ---------------------------------------------------------------------------
// Adjoint (reverse time) of one step, in the scaled variables mu_p = a1 lam_p
// and mu_c = a2 lam_c (lam: the adjoint of the state).  In those the adjoint
// has the forward's shape, and each kernel reads only its own cell's
// coefficients and updates in place, as the forward's do:
//   inject   mu_c[receiver] += a2 dL/dtrace_c
//   adj_p3   mu_p  <- (1 - k1) mu_p + a1 (div mu_v)                (p mask)
//   inject   mu_p[receiver] += a1 dL/dtrace_p
//   adj_v3   G1 += mu_p I,  G2 += sum_c mu_c J_c,
//            mu_c  <- (1 - k_c) mu_c + a2 d_c(mu_p)               (mask of c)
// The damping of mu_p belongs to the end of the step: it is applied when the
// next step reads the value, so that adj_v3's neighbours see it undamped.
// Cells off the masks never depend on the model; their adjoint is dropped
// (held at zero), which keeps every stencil read mask-free.  Free surface: the
// mirror planes p[fs-1] = -p[fs+1] and vz[fs-1] = vz[fs] hand their share to
// planes fs + 1 and fs; with all off-mask cells at zero each share is one term.
// Unscaled, in gather form with two state buffers, the two kernels held 28
// neighbour coefficients a thread and moved 68 bytes per cell and shot: 449 us
// a step at 166 x 185 x 207 with 4 shots.
// ---------------------------------------------------------------------------
struct AdjArgs3 {
    Geo3 g;
    int free_surface;
    float *mu;                    // [S][4][vol] adjoint state, updated in place
    const float *a1, *k1, *a2, *k2, *k3, *k4;
    const float *img_i, *img_j;   // this step's imaging fields
    float *G1, *C1, *G2, *C2;     // [vol] gradient sums and compensations (G2 / C2 null without density)
};

__device__ __forceinline__ void neumaier3(float &s, float &c, float x)
{
    const float t = s + x;
    if (fabsf(s) >= fabsf(x))
        c += (s - t) + x;
    else
        c += (x - t) + s;
    s = t;
}

__device__ __forceinline__ bool in_p(const Geo3 &g, int z, int y, int x)
{
    return z >= g.fs + 1 && z < g.Nz - 2 && y >= 2 && y < g.Ny - 2 && x >= 2 && x < g.Nx - 2;
}
__device__ __forceinline__ bool in_vx(const Geo3 &g, int z, int y, int x)
{
    return z >= g.fs && z < g.Nz - 1 && y >= 1 && y < g.Ny - 1 && x >= 1 && x < g.Nx - 2;
}
__device__ __forceinline__ bool in_vy(const Geo3 &g, int z, int y, int x)
{
    return z >= g.fs && z < g.Nz - 1 && y >= 1 && y < g.Ny - 2 && x >= 1 && x < g.Nx - 1;
}
__device__ __forceinline__ bool in_vz(const Geo3 &g, int z, int y, int x)
{
    return z >= g.fs && z < g.Nz - 2 && y >= 1 && y < g.Ny - 1 && x >= 1 && x < g.Nx - 1;
}

// c1 (a - b) + c2 (c - d)
__device__ __forceinline__ float d4f(float a, float b, float c, float d) { return kC1 * (a - b) + kC2 * (c - d); }

// mu_p (the blocks of p3_kernel)
__global__ void __launch_bounds__(128, 8) adj_p3_kernel(const AdjArgs3 A)
{
    const Geo3 &g = A.g;
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    const int y = blockIdx.y * 4 + threadIdx.y;
    const int z = blockIdx.z;
    if (x0 >= g.Nx - 2 || y < 2 || y >= g.Ny - 2 || z < g.fs + 1 || z >= g.Nz - 2) return;
    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x0;
    const float4 a1 = *reinterpret_cast<const float4 *>(A.a1 + o);
    const float4 k1 = *reinterpret_cast<const float4 *>(A.k1 + o);
    for (int s = 0; s < g.n_shots; ++s) {
        float *P = A.mu + (long long)s * 4 * g.vol;
        const float *VX = P + g.vol, *VY = P + 2 * g.vol, *VZ = P + 3 * g.vol;
        if (s + 1 < g.n_shots) {
            const float *N = P + 4 * g.vol + o;
            prefetch_l2(N); prefetch_l2(N + g.vol); prefetch_l2(N + 2 * g.vol); prefetch_l2(N + 3 * g.vol);
        }
        const float4 p = *reinterpret_cast<const float4 *>(P + o);
        const float4 xl = ld4z(VX, o - 4, x0 >= 4), xc = ld4z(VX, o, true), xr = ld4z(VX, o + 4, x0 + 4 < g.pitch);
        const float xs[12] = {xl.x, xl.y, xl.z, xl.w, xc.x, xc.y, xc.z, xc.w, xr.x, xr.y, xr.z, xr.w};
        const float4 ym2 = ld4z(VY, o - 2 * g.pitch, true), ym1 = ld4z(VY, o - g.pitch, true), y0 = ld4z(VY, o, true),
                     yp1 = ld4z(VY, o + g.pitch, true);
        const float4 zm2 = ld4z(VZ, o - 2 * g.plane, z >= 2), zm1 = ld4z(VZ, o - g.plane, true), z0 = ld4z(VZ, o, true),
                     zp1 = ld4z(VZ, o + g.plane, true);
        float pv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float sum = d4f(xs[q + 4], xs[q + 3], xs[q + 5], xs[q + 2]) + d4f(f4(y0, q), f4(ym1, q), f4(yp1, q), f4(ym2, q)) +
                        d4f(f4(z0, q), f4(zm1, q), f4(zp1, q), f4(zm2, q));
            // the mirror plane's divergence, c2 mu_vz[fs], with the sign of p[fs-1] = -p[fs+1]
            if (A.free_surface && z == g.fs + 1) sum -= kC2 * f4(zm1, q);
            const int x = x0 + q;
            pv[q] = x >= 2 && x < g.Nx - 2 ? (1.f - f4(k1, q)) * f4(p, q) + f4(a1, q) * sum : 0.f;
        }
        *reinterpret_cast<float4 *>(P + o) = make_float4(pv[0], pv[1], pv[2], pv[3]);
    }
}

// mu_vx, mu_vy, mu_vz and the gradient sums (one owner per cell)
template <bool RHO>
__global__ void __launch_bounds__(128, RHO ? 4 : 5) adj_v3_kernel(const AdjArgs3 A)
{
    const Geo3 &g = A.g;
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    const int y = blockIdx.y * 4 + threadIdx.y;
    const int z = g.Nz - 1 - blockIdx.z;
    if (x0 >= g.Nx - 1 || y < 1 || y >= g.Ny - 1 || z < g.fs || z >= g.Nz - 1) return;
    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x0;
    const bool vy_row = y < g.Ny - 2, vz_row = z < g.Nz - 2;
    const float4 a2 = *reinterpret_cast<const float4 *>(A.a2 + o), k2 = *reinterpret_cast<const float4 *>(A.k2 + o),
                 k3 = *reinterpret_cast<const float4 *>(A.k3 + o), k4 = *reinterpret_cast<const float4 *>(A.k4 + o);
    const bool p_row = z >= g.fs + 1 && z < g.Nz - 2 && y >= 2 && y < g.Ny - 2;
    float g1[4] = {0.f, 0.f, 0.f, 0.f}, g2[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < g.n_shots; ++s) {
        const float *P = A.mu + (long long)s * 4 * g.vol;
        float *VX = A.mu + ((long long)s * 4 + 1) * g.vol, *VY = VX + g.vol, *VZ = VY + g.vol;
        const long long jo = (long long)s * g.vol + o, js = (long long)g.n_shots * g.vol;
        if (s + 1 < g.n_shots) {
            const float *N = P + 4 * g.vol + o;
            prefetch_l2(N); prefetch_l2(N + g.vol); prefetch_l2(N + 2 * g.vol); prefetch_l2(N + 3 * g.vol);
            prefetch_l2(A.img_i + jo + g.vol);
            if (RHO) {
                prefetch_l2(A.img_j + jo + g.vol); prefetch_l2(A.img_j + js + jo + g.vol);
                prefetch_l2(A.img_j + 2 * js + jo + g.vol);
            }
        }
        const float4 pc = *reinterpret_cast<const float4 *>(P + o);
        const float4 pl = ld4z(P, o - 4, x0 >= 4), pr = ld4z(P, o + 4, x0 + 4 < g.pitch);
        const float ps[12] = {pl.x, pl.y, pl.z, pl.w, pc.x, pc.y, pc.z, pc.w, pr.x, pr.y, pr.z, pr.w};
        const float4 ym1 = ld4z(P, o - g.pitch, true), yp1 = ld4z(P, o + g.pitch, true),
                     yp2 = ld4z(P, o + 2 * g.pitch, vy_row);
        const float4 zm1 = ld4z(P, o - g.plane, z >= 1), zp1 = ld4z(P, o + g.plane, true),
                     zp2 = ld4z(P, o + 2 * g.plane, vz_row);
        const float4 vx = *reinterpret_cast<const float4 *>(VX + o), vy = *reinterpret_cast<const float4 *>(VY + o),
                     vz = *reinterpret_cast<const float4 *>(VZ + o);
        if (p_row) {
            const float4 im = *reinterpret_cast<const float4 *>(A.img_i + jo);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (x0 + q >= 2 && x0 + q < g.Nx - 2) g1[q] += f4(pc, q) * f4(im, q);
        }
        if (RHO) {
            // on the masks only: the imaging fields need not be written elsewhere
            const float4 jx = *reinterpret_cast<const float4 *>(A.img_j + jo);
            const float4 jy = ld4z(A.img_j, js + jo, vy_row), jz = ld4z(A.img_j, 2 * js + jo, vz_row);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int x = x0 + q;
                if (x >= 1 && x < g.Nx - 2) g2[q] += f4(vx, q) * f4(jx, q);
                if (x >= 1 && x < g.Nx - 1) g2[q] += f4(vy, q) * f4(jy, q) + f4(vz, q) * f4(jz, q);
            }
        }
        float rx[4], ry[4], rz[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int x = x0 + q;
            const bool in = x >= 1 && x < g.Nx - 1;
            const float dx = d4f(ps[q + 5], ps[q + 4], ps[q + 6], ps[q + 3]);
            const float dy = d4f(f4(yp1, q), f4(pc, q), f4(yp2, q), f4(ym1, q));
            float dz = d4f(f4(zp1, q), f4(pc, q), f4(zp2, q), f4(zm1, q));
            // the p update read vz[fs-1] as vz[fs]: the mirror plane's gradient, c2 mu_p[fs+1]
            if (A.free_surface && z == g.fs) dz += kC2 * f4(zp1, q);
            rx[q] = in && x < g.Nx - 2 ? (1.f - f4(k2, q)) * f4(vx, q) + f4(a2, q) * dx : 0.f;
            ry[q] = in && vy_row ? (1.f - f4(k3, q)) * f4(vy, q) + f4(a2, q) * dy : 0.f;
            rz[q] = in && vz_row ? (1.f - f4(k4, q)) * f4(vz, q) + f4(a2, q) * dz : 0.f;
        }
        *reinterpret_cast<float4 *>(VX + o) = make_float4(rx[0], rx[1], rx[2], rx[3]);
        *reinterpret_cast<float4 *>(VY + o) = make_float4(ry[0], ry[1], ry[2], ry[3]);
        *reinterpret_cast<float4 *>(VZ + o) = make_float4(rz[0], rz[1], rz[2], rz[3]);
    }
    auto add = [&](float *G, float *C, const float (&v)[4]) {
        float4 s = *reinterpret_cast<float4 *>(G + o), c = *reinterpret_cast<float4 *>(C + o);
        neumaier3(s.x, c.x, v[0]);
        neumaier3(s.y, c.y, v[1]);
        neumaier3(s.z, c.z, v[2]);
        neumaier3(s.w, c.w, v[3]);
        *reinterpret_cast<float4 *>(G + o) = s;
        *reinterpret_cast<float4 *>(C + o) = c;
    };
    if (p_row) add(A.G1, A.C1, g1);
    if (RHO) add(A.G2, A.C2, g2);
}

// dL/dwavelet[s, it] = dt * lam_p at the source cell, after adj_p3 and the
// pressure injection (lam_p is then the adjoint of p just after the source was
// added, acoustic_3d.py:153-163).  The state keeps lam_p on the p mask only;
// for a source off it, lam_p is the running sum of what reaches the cell: the
// receivers in it and the divergence of mu_v, kept in off[s].  In plane fs + 1
// under a free surface the cell is read a second time, as the mirror cell
// p[fs-1] = -p[fs+1]: minus the receivers in that one and minus its share of
// the divergence, c2 mu_vz[fs] (all else there is zero).  A source in the
// mirror plane is overwritten by the mirror: zero.
// One block per shot: a source off the mask looks through all receivers at
// every step.  (Gradient of one shot, 56 x 80 x 80 cells, 20 steps, 4096
// receivers: 5.95 ms with one thread a shot, 1.71 with a block, 1.65 for a
// source on the mask.)
constexpr int kWaveletThreads = 256;
__global__ void __launch_bounds__(kWaveletThreads)
wavelet_grad3_kernel(const AdjArgs3 A, const int *src, const int *rcv, const float *res_p, float *grad_wavelet,
                     float *off, int it)
{
    const Geo3 &g = A.g;
    const int s = blockIdx.x;
    const int z = src[s], y = src[g.n_shots + s], x = src[2 * g.n_shots + s];
    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x;
    const float *P = A.mu + (long long)s * 4 * g.vol;
    const bool on_mask = in_p(g, z, y, x), overwritten = A.free_surface && z == g.fs - 1;
    const bool mirrored = A.free_surface && z == g.fs + 1;
    float lam = 0.f;
    if (!on_mask && !overwritten && res_p) {
        __shared__ float part[kWaveletThreads / 32];
        for (int r = threadIdx.x; r < g.n_rcv; r += kWaveletThreads)
            if (rcv[g.n_rcv + r] == y && rcv[2 * g.n_rcv + r] == x) {
                const float v = res_p[((long long)s * g.nt + it) * g.n_rcv + r];
                if (rcv[r] == z) lam += v;
                if (mirrored && rcv[r] == g.fs - 1) lam -= v;
            }
        for (int d = 16; d > 0; d >>= 1) lam += __shfl_down_sync(0xffffffffu, lam, d);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = lam;
        __syncthreads();
        lam = 0.f;
        for (int i = 0; i < kWaveletThreads / 32; ++i) lam += part[i];
    }
    if (threadIdx.x != 0) return;
    if (on_mask) {
        lam = P[o] / A.a1[o];
    } else if (!overwritten) {
        auto at = [&](int f, int zz, int yy, int xx) {
            return zz < 0 || zz >= g.Nz || yy < 0 || yy >= g.Ny || xx < 0 || xx >= g.Nx
                       ? 0.f
                       : P[(long long)f * g.vol + (long long)zz * g.plane + (long long)yy * g.pitch + xx];
        };
        lam += off[s];
        lam += d4f(at(1, z, y, x), at(1, z, y, x - 1), at(1, z, y, x + 1), at(1, z, y, x - 2)) +
               d4f(at(2, z, y, x), at(2, z, y - 1, x), at(2, z, y + 1, x), at(2, z, y - 2, x)) +
               d4f(at(3, z, y, x), at(3, z - 1, y, x), at(3, z + 1, y, x), at(3, z - 2, y, x));
        if (mirrored) lam -= kC2 * at(3, g.fs, y, x);
        off[s] = lam;
    }
    grad_wavelet[(long long)s * g.nt + it] = g.dt * lam;
}

// Adjoint of the recording: mu_f[receiver cell] += coefficient * res_f[s][it][r]
// on the mask of field f; a receiver in the mirror plane fs - 1 recorded
// -p[fs+1] and vz[fs].  pressure: p, else the velocities.
__global__ void inj3_kernel(const AdjArgs3 A, const int *rcv, const float *res_p, const float *res_vx,
                            const float *res_vy, const float *res_vz, int pressure, int it)
{
    const Geo3 &g = A.g;
    const long long n = (long long)g.n_shots * g.n_rcv;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(i / g.n_rcv), r = (int)(i % g.n_rcv);
        const int z = rcv[r], y = rcv[g.n_rcv + r], x = rcv[2 * g.n_rcv + r];
        const bool mir = A.free_surface && z == g.fs - 1;
        const long long row = (long long)y * g.pitch + x, o = (long long)z * g.plane + row;
        float *M = A.mu + (long long)s * 4 * g.vol;
        const long long t = ((long long)s * g.nt + it) * g.n_rcv + r;
        // receivers may share a cell
        if (pressure) {
            const int zp = mir ? g.fs + 1 : z;
            const long long op = (long long)zp * g.plane + row;
            if (in_p(g, zp, y, x)) atomicAdd(M + op, mir ? -A.a1[op] * res_p[t] : A.a1[op] * res_p[t]);
            continue;
        }
        if (res_vx && in_vx(g, z, y, x)) atomicAdd(M + g.vol + o, A.a2[o] * res_vx[t]);
        if (res_vy && in_vy(g, z, y, x)) atomicAdd(M + 2 * g.vol + o, A.a2[o] * res_vy[t]);
        const int zv = mir ? g.fs : z;
        const long long ov = (long long)zv * g.plane + row;
        if (res_vz && in_vz(g, zv, y, x)) atomicAdd(M + 3 * g.vol + ov, A.a2[ov] * res_vz[t]);
    }
}

// dL/dvp, dL/drho on the unpadded grid: G1 = sum mu_p I and G2 = sum mu_v J
// are a1 dL/da1 and -a2 dL/da2, so with a1 = rho c^2 dt / dz and a2 = dt /
// (rho dz) dL/dc = 2 G1 / c and dL/drho = (G1 + G2) / rho, summed over the padded
// cells each model cell was replicated into (the adjoint of pad_model_3d).  A
// cell on an edge or a corner of the model collects pml^2 or pml^3 of them: a
// warp shares those (one thread per corner took 0.67 ms at 18 layers).
__global__ void grad3_finish_kernel(const Geo3 g, const float *vp, const float *rho, const float *G1,
                                    const float *C1, const float *G2, const float *C2, float *grad_vp,
                                    float *grad_rho)
{
    auto span = [&](int idx, int n_in, int &lo, int &len) {
        lo = idx == 0 ? 0 : idx + g.pml;
        len = (idx == n_in - 1 ? n_in + 2 * g.pml - 1 : idx + g.pml) - lo + 1;
    };
    auto write = [&](long long i, double s1, double s2) {
        grad_vp[i] = (float)(2.0 * s1 / (double)vp[i]);
        if (grad_rho) grad_rho[i] = (float)((s1 + s2) / (double)rho[i]);
    };
    auto edge = [&](int idx, int n_in) { return idx == 0 || idx == n_in - 1 ? 1 : 0; };
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, threads = (long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    // the lines of cells where two or three faces meet: 4 along each axis
    // (each corner cell belongs to three of them; the x line keeps it)
    const int L = max(g.nx, max(g.ny, g.nz));
    for (long long k = tid >> 5; k < 12LL * L; k += threads >> 5) {
        const int line = (int)(k / L), at = (int)(k % L), axis = line / 4;
        const int a = line & 1, b = (line >> 1) & 1;
        int ix, iy, iz;
        if (axis == 0) { ix = at; iy = a ? g.ny - 1 : 0; iz = b ? g.nz - 1 : 0; }
        else if (axis == 1) { ix = a ? g.nx - 1 : 0; iy = at; iz = b ? g.nz - 1 : 0; }
        else { ix = a ? g.nx - 1 : 0; iy = b ? g.ny - 1 : 0; iz = at; }
        if (ix >= g.nx || iy >= g.ny || iz >= g.nz) continue;
        if (axis == 1 && edge(iy, g.ny)) continue;
        if (axis == 2 && edge(iz, g.nz)) continue;
        int z0, y0, x0, nz, ny, nx;
        span(iz, g.nz, z0, nz);
        span(iy, g.ny, y0, ny);
        span(ix, g.nx, x0, nx);
        double s1 = 0.0, s2 = 0.0;
        for (long long m = lane; m < (long long)nz * ny * nx; m += 32) {
            const long long o = (long long)(z0 + (int)(m / nx / ny)) * g.plane + (long long)(y0 + (int)(m / nx % ny)) * g.pitch +
                                x0 + (int)(m % nx);
            s1 += (double)G1[o] + (double)C1[o];
            if (G2) s2 += (double)G2[o] + (double)C2[o];
        }
        for (int o = 16; o > 0; o >>= 1) {
            s1 += __shfl_down_sync(0xffffffffu, s1, o);
            s2 += __shfl_down_sync(0xffffffffu, s2, o);
        }
        if (lane == 0) write(((long long)iz * g.ny + iy) * g.nx + ix, s1, s2);
    }
    const long long n = (long long)g.nz * g.ny * g.nx;
    for (long long i = tid; i < n; i += threads) {
        const int ix = (int)(i % g.nx), iy = (int)((i / g.nx) % g.ny), iz = (int)(i / ((long long)g.nx * g.ny));
        if (edge(ix, g.nx) + edge(iy, g.ny) + edge(iz, g.nz) >= 2) continue;
        int z0, y0, x0, nz, ny, nx;
        span(iz, g.nz, z0, nz);
        span(iy, g.ny, y0, ny);
        span(ix, g.nx, x0, nx);
        double s1 = 0.0, s2 = 0.0;
        for (int z = z0; z < z0 + nz; ++z)
            for (int y = y0; y < y0 + ny; ++y)
                for (int x = x0; x < x0 + nx; ++x) {
                    const long long o = (long long)z * g.plane + (long long)y * g.pitch + x;
                    s1 += (double)G1[o] + (double)C1[o];
                    if (G2) s2 += (double)G2[o] + (double)C2[o];
                }
        write(i, s1, s2);
    }
}

}  // namespace gb
