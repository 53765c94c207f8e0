// Resident adjoint: the reverse time loop of a gradient in one launch, the
// adjoint state of a tile and its coefficients in shared memory and its
// gradient sums in registers for every step.
//
// A gradient of one shot, or of a few on a small grid, is bound by what the
// tile kernel (gb_adj.cuh) does around a step: a launch, the fill of the
// stage, its drain (140 x 240, one shot, 4th order: 4.7 us a step against
// 2.2 of the resident forward; here 2.0, and a gradient of 600 steps 3.14 ms
// where the tile adjoint behind the resident forward took 5.02).  The adjoint step has the forward's shape in
// mu_p = a1 lambda_p, mu_v = a2 lambda_v, so this kernel runs the resident
// forward's schedule (gb_resident.cuh: interior, receive, boundary, twice a
// step, through (value, tag) words in global memory) with its tilings and
// its exchange:
//
//   mu_p <- d1 mu_p (+ residual at the receivers) + a1m div(mu_v);  G1 += mu_p I
//   mu_v <- d2|d3 mu_v + a2x|a2z grad(mu_p);                        G2 += mu_v J
//
// The arithmetic is the tile kernel's, tap for tap, so the gradients are the
// same bits (one shot a group there).  What it does not run, and leaves to
// the tile kernel: residuals of vx or vz, checkpoint segments, CPML.
//
// mu_p as the stencils of a step read it is undamped, and as the next step
// starts it damped and with the residuals added: the first is in the rect,
// the second in a plane of its own (sQ, owned rows), which saves the barrier
// between the last read and the damping.  Cells off the update masks start
// at zero and stay there: their folded coefficients are zero and residuals
// off the pressure mask are dropped.
//
// Imaging fields and residuals of the next step are loaded into registers
// while this one waits for its neighbours.
#pragma once

#include "gb_adj.cuh"
#include "gb_resident.cuh"

namespace gb {

template <int R, int NW, int TZ>
struct ResAdjGeo {
    using G = ResGeo<R, NW, TZ>;
    static_assert(G::NITEM <= G::NTH, "one boundary item per thread");
    static constexpr int NC = G::LI + 1;          // 4-cell groups of a thread: its interior rows and a boundary item
    static constexpr size_t SMEM = G::SMEM + (size_t)G::CF * 4;
};

// mu_p of the 4 cells of rect row r, lane l: stage A of the tile kernel.
// wz[u + R] is mu_vz row r.  Returns the undamped new values.
template <int R>
__device__ __forceinline__ float4 res_mu_p(const ResArgs &A, const ResCtx &C, float *sQ, int r, int l, const float4 *wz,
                                           int u)
{
    const StepGeom &g = A.g;
    const int o = (r - R) * RS + 4 * l;
    float4 pv = lds4(sQ + o);
    const float4 a1 = lds4(C.cA1 + o);
    float D[4];
    divergence4<R>(C.sVX + r * RS - 4, l, wz, u, g.c, D);
    if (A.free_surface && C.z0 - R + r == g.fs + 1) {
        // share of the mirror row p[fs-1] = -p[fs+1]
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float M = 0.f;
#pragma unroll
            for (int kk = 0; kk < R; ++kk) M = __fmaf_rn(g.c[kk], at(wz[u + R - 2 + kk], q), M);
            D[q] -= M;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) at(pv, q) = __fmaf_rn(at(a1, q), D[q], at(pv, q));
    sts4(C.sP + r * RS + 4 * l, pv);
    float4 nx = pv;
    if (!C.fast) {
        const float4 d1 = lds4(C.cD1 + o);
#pragma unroll
        for (int q = 0; q < 4; ++q) at(nx, q) = at(d1, q) * at(pv, q);
    }
    sts4(sQ + o, nx);
    return pv;
}

// mu_vx, mu_vz of the 4 cells: stage B.  wp[u + R] is mu_p row r + 1.
// vx1, vz1 return the values before the update.
template <int R>
__device__ __forceinline__ void res_mu_v(const ResArgs &A, const ResCtx &C, int r, int l, const float4 *wp, int u,
                                         float4 &vx1, float4 &vz1, float4 &vx, float4 &vz)
{
    const StepGeom &g = A.g;
    float Dx[4], Dz[4];
    grad_x4<R>(C.sP + r * RS, l, g.c, Dx, wp[u + R - 1]);
    grad_z4<R>(wp, u, g.c, Dz);
    vx1 = lds4(C.sVX + r * RS + 4 * l);
    vz1 = lds4(C.sVZ + r * RS + 4 * l);
    const int o = (r - R) * RS + 4 * l;
    const float4 ax = lds4(C.cA2X + o);
    if (C.fast) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            at(vx, q) = __fmaf_rn(at(ax, q), Dx[q], at(vx1, q));
            at(vz, q) = __fmaf_rn(at(ax, q), Dz[q], at(vz1, q));
        }
    } else {
        const float4 d2 = lds4(C.cD2 + o), az = lds4(C.cA2Z + o), d3 = lds4(C.cD3 + o);
        if (A.free_surface && C.z0 - R + r == g.fs) {
            // the p update reads vz[fs-1] as vz[fs]
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int kk = 0; kk < R; ++kk) Dz[q] = __fmaf_rn(g.c[kk], at(wp[u + R - 1 + kk], q), Dz[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            at(vx, q) = __fmaf_rn(at(ax, q), Dx[q], at(d2, q) * at(vx1, q));
            at(vz, q) = __fmaf_rn(at(az, q), Dz[q], at(d3, q) * at(vz1, q));
        }
    }
    sts4(C.sVX + r * RS + 4 * l, vx);
    sts4(C.sVZ + r * RS + 4 * l, vz);
}

// A.rcv_ent: (row in tile, column in tile, receiver, 0), as the forward's.
template <int R, int NW, int TZ, bool RHO>
__global__ void __launch_bounds__(NW * 32, 1) resident_adj_kernel(const ResArgs A)
{
    using G = ResGeo<R, NW, TZ>;
    constexpr int NC = ResAdjGeo<R, NW, TZ>::NC;
    extern __shared__ __align__(128) float sm[];
    ResCtx C;
    C.sP = sm;
    C.sVX = sm + G::FL;
    C.sVZ = sm + 2 * G::FL;
    float *cf = sm + 3 * G::FL;
    C.cA1 = cf;
    C.cD1 = cf + G::CF;
    C.cA2X = cf + 2 * G::CF;
    C.cD2 = cf + 3 * G::CF;
    C.cA2Z = cf + 4 * G::CF;
    C.cD3 = cf + 5 * G::CF;
    float *sQ = cf + 6 * G::CF;
    float *sP = C.sP, *sVX = C.sVX, *sVZ = C.sVZ;
    const StepGeom &g = A.g;
    const int tile = (int)(blockIdx.x % A.n_tiles);
    const int s = A.shot0 + (int)(blockIdx.x / A.n_tiles);
    const int ti = tile / A.tiles_x, tj = tile % A.tiles_x;
    const int z0 = ti * TZ, x0 = tj * TX;
    C.z0 = z0;
    C.x0 = x0;
    C.s = s;
    C.sz = A.src_z[s];
    C.sx = A.src_x[s];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint2 *xb = A.xbuf + (size_t)s * A.n_tiles * kResParts * G::PART;
    ResLinks K;
    K.nb[0] = ti > 0 ? tile - A.tiles_x : -1;
    K.nb[1] = ti + 1 < A.tiles_z ? tile + A.tiles_x : -1;
    K.nb[2] = tj > 0 ? tile - 1 : -1;
    K.nb[3] = tj + 1 < A.tiles_x ? tile + 1 : -1;
    K.my = A.xbuf + ((size_t)s * A.n_tiles + tile) * kResParts * G::PART;
    K.part = G::PART;
#pragma unroll
    for (int k = 0; k < 4; ++k) K.rP[k] = K.rVX[k] = K.rVZ[k] = 0;

    for (int e = threadIdx.x; e < 3 * G::FL / 4; e += G::NTH) sts4(sm + 4 * e, zero4());
    for (int e = threadIdx.x; e < G::CF / 4; e += G::NTH) sts4(sQ + 4 * e, zero4());
    C.fast = res_load_coef<R, NW, TZ>(A, cf, z0, x0);

    // this thread's 4-cell groups: c < LI interior row ri + c of its lane,
    // c = LI its boundary item; element offset of each in a plane (-1: none)
    const bool ilane = lane >= 2 && lane <= 29;
    const int ri = 2 * R + warp * G::LI;
    const bool interior = G::NI > 0 && ilane && ri < TZ;
    const bool item = threadIdx.x < G::NITEM;
    int br = 0, bl = 0;
    if (item) res_item<R, NW, TZ>(threadIdx.x, br, bl);
    ResRecv<R, NW, TZ> recv;
    recv.init(sP, sVX, sVZ, xb, K.nb);
    int off[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int r = c < G::LI ? ri + c : br, l = c < G::LI ? lane : bl;
        const bool mine = c < G::LI ? interior && ri + c < TZ : item;
        const int gz = z0 - R + r, gx = x0 - 4 + 4 * l;
        off[c] = mine && gz < g.Nz && gx < g.Nx ? gz * g.pitch + gx : -1;
    }
    const long long so = (long long)s * g.plane;
    ImgRaw im[NC], jx[RHO ? NC : 1], jz[RHO ? NC : 1];
    const auto load_i = [&](int it) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
            im[c] = off[c] >= 0 ? load_img_raw(res_img_step(A, it), so + off[c], A.img_fmt) : img_raw_zero();
    };
    const auto load_j = [&](int it) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float *b = res_img_step(A, it);
            jx[c] = off[c] >= 0 ? load_img_raw(b, so + A.img_field_stride + off[c], A.img_fmt) : img_raw_zero();
            jz[c] = off[c] >= 0 ? load_img_raw(b, so + 2 * A.img_field_stride + off[c], A.img_fmt) : img_raw_zero();
        }
    };
    float4 s1[NC], c1[NC], s2[RHO ? NC : 1], c2[RHO ? NC : 1];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        s1[c] = c1[c] = zero4();
        if (RHO) s2[c] = c2[c] = zero4();
    }
    const auto sum_p = [&](int c, const float4 &mu) {
        const float4 v = decode_img4(im[c], A.img_fmt);
#pragma unroll
        for (int q = 0; q < 4; ++q) neumaier_add(at(s1[c], q), at(c1[c], q), __fmul_rn(at(mu, q), at(v, q)));
    };
    const auto sum_v = [&](int c, const float4 &vx1, const float4 &vz1) {
        const float4 a = decode_img4(jx[c], A.img_fmt), b = decode_img4(jz[c], A.img_fmt);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            neumaier_add(at(s2[c], q), at(c2[c], q), __fmaf_rn(at(vz1, q), at(b, q), __fmul_rn(at(vx1, q), at(a, q))));
    };

    // residuals: this thread's first receiver of the tile is loaded a step ahead
    const int rcv0 = A.rcv_ptr[tile], rcv1 = A.rcv_ptr[tile + 1];
    const int e0 = rcv0 + (int)threadIdx.x;
    const auto residual = [&](int e, int it) {
        return A.res_p[((long long)s * g.nt + it) * g.n_rcv + A.rcv_ent[e].z];
    };
    const auto inject = [&](int e, float v) {
        const int4 en = A.rcv_ent[e];
        int z = z0 + en.x;
        const int x = x0 + en.y;
        // a receiver in the mirror row fs-1 records p[fs-1] = -p[fs+1]
        const bool mir = A.free_surface && z == g.fs - 1;
        if (mir) z = g.fs + 1;
        if (z < g.p_r0 || z > g.p_r1 || x < g.p_c0 || x > g.p_c1) return;
        const int o = (z - z0) * RS + en.y + 4;
        const float v1 = C.cA1[o] * v;
        atomicAdd(&sQ[o], mir ? -v1 : v1);
    };
    __syncthreads();
    load_i(A.it1 - 1);
    for (int e = e0; e < rcv1; e += G::NTH) inject(e, residual(e, A.it1 - 1));
    __syncthreads();

    for (int it = A.it1 - 1; it >= A.it0; --it) {
        const int n = A.it1 - 1 - it;
        if (RHO) load_j(it);
        const float rnext = it > A.it0 && e0 < rcv1 ? residual(e0, it - 1) : 0.f;
        // ---- mu_p interior --------------------------------------------------
        if (interior) {
            float4 wz[G::LI + 2 * R - 1];
#pragma unroll
            for (int t = 0; t < G::LI + 2 * R - 1; ++t) wz[t] = lds4(sVZ + (ri - R + t) * RS + 4 * lane);
#pragma unroll
            for (int u = 0; u < G::LI; ++u)
                if (ri + u < TZ) sum_p(u, res_mu_p<R>(A, C, sQ, ri + u, lane, wz, u));
        }
        // ---- the neighbours' mu_v boundary cells of the previous step --------
        if (n > 0 && !recv.template get<true>(tag_v(n - 1), A.err)) return;
        // ---- mu_p boundary (sent on as computed) ----------------------------
        if (item) {
            float4 wz[2 * R];
#pragma unroll
            for (int t = 0; t < 2 * R; ++t) wz[t] = lds4(sVZ + (br - R + t) * RS + 4 * bl);
            const float4 pv = res_mu_p<R>(A, C, sQ, br, bl, wz, 0);
            res_send4<R, TZ, false>(K, K.rP, 0, 2, true, true, br, bl, pv, tag_p(n));
            sum_p(G::LI, pv);
        }
        __syncthreads();
        if (A.grad_wavelet && threadIdx.x == 0 && C.sz >= z0 && C.sz < z0 + TZ && C.sx >= x0 && C.sx < x0 + TX)
            // mu_p / a1 at the source cell is lambda_p
            A.grad_wavelet[(long long)s * g.nt + it] =
                g.dt * (sP[(C.sz - z0 + R) * RS + C.sx - x0 + 4] / C.cA1[(C.sz - z0) * RS + C.sx - x0 + 4]);
        if (it > A.it0) {
            load_i(it - 1);
            if (e0 < rcv1) inject(e0, rnext);
            for (int e = e0 + G::NTH; e < rcv1; e += G::NTH) inject(e, residual(e, it - 1));
        }
        // ---- mu_v interior (reads the tile's own mu_p only) ------------------
        if (interior) {
            float4 wp[G::LI + 2 * R - 1];
#pragma unroll
            for (int t = 0; t < G::LI + 2 * R - 1; ++t) wp[t] = lds4(sP + (ri - R + 1 + t) * RS + 4 * lane);
#pragma unroll
            for (int u = 0; u < G::LI; ++u)
                if (ri + u < TZ) {
                    float4 vx1, vz1, vx, vz;
                    res_mu_v<R>(A, C, ri + u, lane, wp, u, vx1, vz1, vx, vz);
                    if (RHO) sum_v(u, vx1, vz1);
                }
        }
        // ---- the neighbours' mu_p boundary cells -----------------------------
        if (!recv.template get<false>(tag_p(n), A.err)) return;
        // ---- mu_v boundary (sent on unless this is the last step) -------------
        if (item) {
            float4 wp[2 * R];
#pragma unroll
            for (int t = 0; t < 2 * R; ++t) wp[t] = lds4(sP + (br - R + 1 + t) * RS + 4 * bl);
            float4 vx1, vz1, vx, vz;
            res_mu_v<R>(A, C, br, bl, wp, 0, vx1, vz1, vx, vz);
            if (it > A.it0) {
                res_send4<R, TZ, false>(K, K.rVZ, 4, 6, true, false, br, bl, vz, tag_v(n));
                res_send4<R, TZ, false>(K, K.rVX, 4, 6, false, true, br, bl, vx, tag_v(n));
            }
            if (RHO) sum_v(G::LI, vx1, vz1);
        }
        // the next step writes mu_p, which this one's stencils read
        __syncthreads();
    }
    // G1 and C1 hold zeros: groups wholly off the p mask stay so.  Their sums
    // are zeros times whatever is in a store that the tile forward made, which
    // writes I on the mask only.
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (off[c] >= 0) {
            const int gz = z0 - R + (c < G::LI ? ri + c : br), gx = x0 - 4 + 4 * (c < G::LI ? lane : bl);
            if (gz >= g.p_r0 && gz <= g.p_r1 && gx + 3 >= g.p_c0 && gx <= g.p_c1) {
                stg4(A.G1 + so + off[c], s1[c]);
                stg4(A.C1 + so + off[c], c1[c]);
            }
            if (RHO) {
                stg4(A.G2 + so + off[c], s2[c]);
                stg4(A.C2 + so + off[c], c2[c]);
            }
        }
}

}  // namespace gb
