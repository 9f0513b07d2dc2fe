// lbm_node.cuh -- the step of one node by one thread (pull, moments, collisions,
// wall and injection rules), shared by the step kernels; see lbm.cu.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace ehd {

namespace {

struct PullIdx {
    unsigned row[3][3];  // [e_y+1][e_z+1] -> NX*(ys + NY*zs) for source (y - e_y, z - e_z)
    int xs[3];           // [e_x+1] -> source x - e_x
};

__device__ __forceinline__ void make_pull(PullIdx &P, int x, int y, int z, int NX, int NY,
                                          int NZ) {
    const int xm = x == 0 ? NX - 1 : x - 1, xp = x == NX - 1 ? 0 : x + 1;
    const int ym = y == 0 ? NY - 1 : y - 1, yp = y == NY - 1 ? 0 : y + 1;
    const int zm = z == 0 ? NZ - 1 : z - 1, zp = z == NZ - 1 ? 0 : z + 1;
    P.xs[0] = xp;  // e_x = -1: source x + 1
    P.xs[1] = x;
    P.xs[2] = xm;  // e_x = +1: source x - 1
    const int ys[3] = {yp, y, ym};
    const int zs[3] = {zp, z, zm};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            P.row[a][b] = (unsigned)NX * ((unsigned)ys[a] + (unsigned)NY * (unsigned)zs[b]);
}

__device__ __forceinline__ unsigned pull_src(const PullIdx &P, int d) {
    return P.row[ey_of(d) + 1][ez_of(d) + 1] + (unsigned)P.xs[ex_of(d) + 1];
}

// e_d . (a, b, c) with the components of e_d in {-1, 0, 1}
template <typename R>
__device__ __forceinline__ R dot_e(int d, R a, R b, R c) {
    R s = 0;
    if (ex_of(d)) s = ex_of(d) > 0 ? a : -a;
    if (ey_of(d)) s = ey_of(d) > 0 ? s + b : s - b;
    if (ez_of(d)) s = ez_of(d) > 0 ? s + c : s - c;
    return s;
}

// Per-plane reference state.  Populations are stored as deviations
// f_d - w_d rho_w(z), g_d - w_d q_w(z) from the reference (rho_w, q_w) of the
// step that wrote them and of the plane z they are stored in.  A step reads
// populations written against the previous step's references (rho_r, q_r) and
// writes against its own, so a population pulled from plane z - e_z is moved
// to this step's reference of plane z by adding w_d (rho_r(z - e_z) -
// rho_w(z)).  The kernel table holds per plane, in the compute type:
// {rho_w, q_w, drho[e_z = -1, 0, +1], dq[e_z = -1, 0, +1], q_w(z) - q_w(z+1),
// unused} with drho[e] = rho_r(z - e) - rho_w(z), z - e periodic.
constexpr int kZRefStride = 10;

template <typename R>
struct ZRef {
    R rref, qref, drm, dr0, drp, dqm, dq0, dqp, up;
    // offset for a population with z-velocity e (source plane z - e)
    __device__ __forceinline__ R dr(int e) const { return e > 0 ? drm : (e < 0 ? drp : dr0); }
    __device__ __forceinline__ R dq(int e) const { return e > 0 ? dqm : (e < 0 ? dqp : dq0); }
};

// rate * x with rate = hi - lo (see StepConst::rate_hi)
template <typename R>
__device__ __forceinline__ R relax(R hi, R lo, R x) {
    return hi * x - lo * x;
}

template <typename R>
__device__ __forceinline__ ZRef<R> load_zref(const R *__restrict__ t, int z) {
    const R *p = t + kZRefStride * z;
    return ZRef<R>{__ldg(p),     __ldg(p + 1), __ldg(p + 2), __ldg(p + 3), __ldg(p + 4),
                   __ldg(p + 5), __ldg(p + 6), __ldg(p + 7), __ldg(p + 8)};
}

}  // namespace

// Kernel arguments shared by both step kernels.
template <typename T, typename R>
struct StepArgs {
    PopPtrs<T> pp;
    const R *phip;                    // phi', zero on both electrodes
    const double *ez00;               // mean-field Ez per plane
    const double *exa, *eya, *eza;    // uploaded E (first step after set_fields)
    R *qout, *rout, *uout, *vout, *wout;
    const R *zref;                    // reference table (load_zref)
    float2 *psum;                     // per-warp plane sums
    int *err;                         // set to 1 if a bounded wait gives up
};

// Pull of node (x, y, z) from global memory (the reference's stream and
// injection rule), as deviations ft_d = f_d - w_d rho_w(z), ht_d = g_d -
// w_d q_w(z).  local: the buffers hold each node's own pre-collision values.
template <typename T, typename R>
__device__ __forceinline__ void pull_global(R (&f)[Q], R (&h)[Q], const PopPtrs<T> &pp,
                                            const PullIdx &P, unsigned node, int z,
                                            const ZRef<R> &zr, const KConst<R> &c, bool local) {
#pragma unroll
    for (int d = 0; d < Q; ++d) {
        f[d] = pld(pp.fa[d] + (local ? node : pull_src(P, d))) +
               c.w[cls_of(d)] * zr.dr(local ? 0 : ez_of(d));
    }
    if (local) {
#pragma unroll
        for (int d = 0; d < Q; ++d) h[d] = pld(pp.ha[d] + node) + c.w[cls_of(d)] * zr.dq0;
    } else if (z == 0) {
        // g_d = -g_opp(d) + 2 q0 w_d (LBM.cu:1320-1348), on deviations
        h[0] = pld(pp.ha[0] + node) + c.w[0] * zr.dq0;
        const R inj = (R)2 * (c.q0 - zr.qref) - zr.dq0;
#pragma unroll
        for (int d = 1; d < Q; ++d)
            h[d] = -pld(pp.ha[opp_of(d)] + node) + inj * c.w[cls_of(d)];
    } else {
#pragma unroll
        for (int d = 0; d < Q; ++d)
            h[d] = pld(pp.ha[d] + pull_src(P, d)) + c.w[cls_of(d)] * zr.dq(ez_of(d));
    }
}

template <typename R>
struct Moments {
    R drho, dq, mx, my, mz, rho, charge;
};

template <typename R>
__device__ __forceinline__ Moments<R> moments(const R (&f)[Q], const R (&h)[Q], const ZRef<R> &zr) {
    Moments<R> m{0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int d = 0; d < Q; ++d) {
        m.drho += f[d];
        m.dq += h[d];
        if (ex_of(d)) m.mx += ex_of(d) > 0 ? f[d] : -f[d];
        if (ey_of(d)) m.my += ey_of(d) > 0 ? f[d] : -f[d];
        if (ez_of(d)) m.mz += ez_of(d) > 0 ? f[d] : -f[d];
    }
    m.rho = zr.rref + m.drho;
    m.charge = zr.qref + m.dq;
    return m;
}

// Warp sum of rho and q into psum[slot] (fixed order; all 32 lanes take part).
__device__ __forceinline__ void warp_plane_sum(float rho, float charge, float2 *psum, size_t slot) {
    float2 v = make_float2(rho, charge);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if ((threadIdx.x & 31) == 0) psum[slot] = v;
}

// ---- packed FP32x2 collision (sm_100 FFMA2): two opposite pairs of one weight
// class at once, the same algebra as the scalar loops of finish_node ----
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

struct PackF {
    float2 rp_hi, nrp_lo, rm_hi, nrm_lo, half, mone;
    float2 PK[4], QK[4], nhWR[4], nWR[4], nc1[4], nc2[4];
    float tux, tuy, tuz, fx, fy, fz;
};

template <int D1, int D2, typename T>
__device__ __forceinline__ void f_pair2(const float (&f)[Q], const PackF &p,
                                        const PopPtrs<T> &pp, unsigned node) {
    constexpr int K = cls_of(D1);
    static_assert(cls_of(D2) == K, "pairs of one weight class");
    const float2 fd = f2(f[D1], f[D2]), fo = f2(f[D1 + 1], f[D2 + 1]);
    const float2 cu = f2(dot_e(D1, p.tux, p.tuy, p.tuz), dot_e(D2, p.tux, p.tuy, p.tuz));
    const float2 eF = f2(dot_e(D1, p.fx, p.fy, p.fz), dot_e(D2, p.fx, p.fy, p.fz));
    float2 X = __ffma2_rn(p.half, __fadd2_rn(fd, fo), p.PK[K]);
    X = __ffma2_rn(__fmul2_rn(p.nhWR[K], cu), cu, X);
    float2 A = __ffma2_rn(p.nrp_lo, X, p.QK[K]);
    A = __ffma2_rn(p.rp_hi, X, A);
    A = __ffma2_rn(p.nc1[K], __fmul2_rn(cu, eF), A);
    const float2 D = __ffma2_rn(p.mone, fo, fd);
    const float2 Y = __ffma2_rn(p.half, D, __fmul2_rn(p.nWR[K], cu));
    float2 B = __ffma2_rn(p.nrm_lo, Y, __fmul2_rn(p.nc2[K], eF));
    B = __ffma2_rn(p.rm_hi, Y, B);
    const float2 od = __ffma2_rn(p.mone, __fadd2_rn(A, B), fd);
    const float2 oo = __ffma2_rn(p.mone, A, __fadd2_rn(fo, B));
    pst(pp.fb[D1] + node, od.x);
    pst(pp.fb[D2] + node, od.y);
    pst(pp.fb[D1 + 1] + node, oo.x);
    pst(pp.fb[D2 + 1] + node, oo.y);
}

struct PackG {
    float2 cp_hi, ncp_lo, cm_hi, ncm_lo, cm_lo, half, mone;
    float2 PQ[4], nhWQ[4], nWQ[4], twoWQ[4], wup[4];
    float tux, tuy, tuz;
    bool over;  // antisymmetric rate over-relaxed: hi = 2 exactly
};

template <int D1, int D2, typename T>
__device__ __forceinline__ void g_pair2(const float (&h)[Q], const PackG &p,
                                        const PopPtrs<T> &pp, unsigned node, unsigned nodeup,
                                        bool dup) {
    constexpr int K = cls_of(D1);
    static_assert(cls_of(D2) == K, "pairs of one weight class");
    const float2 hd = f2(h[D1], h[D2]), ho = f2(h[D1 + 1], h[D2 + 1]);
    const float2 cu = f2(dot_e(D1, p.tux, p.tuy, p.tuz), dot_e(D2, p.tux, p.tuy, p.tuz));
    float2 X = __ffma2_rn(p.half, __fadd2_rn(hd, ho), p.PQ[K]);
    X = __ffma2_rn(__fmul2_rn(p.nhWQ[K], cu), cu, X);
    const float2 Dd = __ffma2_rn(p.mone, ho, hd);
    const float2 Y = __ffma2_rn(p.half, Dd, __fmul2_rn(p.nWQ[K], cu));
    const float2 A = __ffma2_rn(p.cp_hi, X, __fmul2_rn(p.ncp_lo, X));
    float2 od, oo;
    if (p.over) {
        // with B = 2 Y - lo Y: hd - 2 Y = ho + 2 WQ cu and ho + 2 Y = hd - 2 WQ cu
        // exactly, so the outputs never form hd - B, which cancels when the
        // rate is close to 2
        const float2 t = __fmul2_rn(p.twoWQ[K], cu);
        od = __ffma2_rn(p.cm_lo, Y, __ffma2_rn(p.mone, A, __fadd2_rn(ho, t)));
        oo = __ffma2_rn(p.ncm_lo, Y, __ffma2_rn(p.mone, A, __ffma2_rn(p.mone, t, hd)));
    } else {
        const float2 B = __ffma2_rn(p.cm_hi, Y, __fmul2_rn(p.ncm_lo, Y));
        od = __ffma2_rn(p.mone, __fadd2_rn(A, B), hd);
        oo = __ffma2_rn(p.mone, A, __fadd2_rn(ho, B));
    }
    pst(pp.hb[D1] + node, od.x);
    pst(pp.hb[D2] + node, od.y);
    pst(pp.hb[D1 + 1] + node, oo.x);
    pst(pp.hb[D2 + 1] + node, oo.y);
    if (dup) {
        const float2 ud = __fadd2_rn(od, p.wup[K]), uo = __fadd2_rn(oo, p.wup[K]);
        pst(pp.hb[D1] + nodeup, ud.x);
        pst(pp.hb[D2] + nodeup, ud.y);
        pst(pp.hb[D1 + 1] + nodeup, uo.x);
        pst(pp.hb[D2 + 1] + nodeup, uo.y);
    }
}

// Everything after the moments: E, the injector override, the macroscopic
// outputs, the TRT collisions of f and g and the wall rules on store.
//
// Collision algebra (LBM.cu:519-1089 rewritten on deviations, per opposite
// pair d, o = d+1 of weight class k, s = f_d + f_o):
//   fp - feq+  = s/2 + P_k - (w_k rho / 2) cu^2,  P_k = w_k rho usq - w_k drho
//   fm - feq-  = (f_d - f_o)/2 - w_k rho cu
//   A = rate+ (fp - feq+) + dt sp (w_k/cs2) uF - dt sp w_k cflinv2 CFL cu eF
//   B = rate- (fm - feq-) - dt sm (w_k/cs2) cflinv eF
//   f_d' = f_d - A - B,  f_o' = f_o - A + B
// (e.u = cu cs2 CFL); the same with q, u + K E and no source for g.
template <typename T, typename R, bool MACROS>
__device__ __forceinline__ void finish_node(R (&f)[Q], R (&h)[Q], const Moments<R> &mo, int x,
                                            int y, int z, unsigned node, const ZRef<R> &zr,
                                            const StepArgs<T, R> &a, const KConst<R> &c,
                                            bool local, bool earr) {
    const int NX = c.nx, NY = c.ny, NZ = c.nz;
    const R drho = mo.drho, dq = mo.dq, mx = mo.mx, my = mo.my, mz = mo.mz;
    const R rho = mo.rho, charge = mo.charge;
    // ---- E at this node (and at z = 1 for the injector override) ----
    R Ex, Ey, Ez;
    const unsigned row = (unsigned)NX * ((unsigned)y + (unsigned)NY * z);
    const int xm = x == 0 ? NX - 1 : x - 1, xp = x == NX - 1 ? 0 : x + 1;
    const int ym = y == 0 ? NY - 1 : y - 1, yp = y == NY - 1 ? 0 : y + 1;
    const unsigned rym = (unsigned)NX * ((unsigned)ym + (unsigned)NY * z);
    const unsigned ryp = (unsigned)NX * ((unsigned)yp + (unsigned)NY * z);
    if (!earr) {
        // E = -grad(phi), central differences (gpu_efield, poisson.cu:44-60);
        // phi = phi00(z) + phi'(x,y,z) with phi' = 0 on both electrodes, and
        // Ez on the electrodes copied from the planes inside (gpu_bc,
        // poisson.cu:61-73).
        Ex = (__ldg(a.phip + row + xm) - __ldg(a.phip + row + xp)) * c.inv2dx;
        Ey = (__ldg(a.phip + rym + x) - __ldg(a.phip + ryp + x)) * c.inv2dy;
        const int zc = z < 1 ? 1 : (z > NZ - 2 ? NZ - 2 : z);
        const unsigned rzc = (unsigned)NX * ((unsigned)y + (unsigned)NY * zc);
        Ez = (R)__ldg(a.ez00 + zc) +
             (__ldg(a.phip + rzc - c.nxy + x) - __ldg(a.phip + rzc + c.nxy + x)) * c.inv2dz;
    } else {
        Ex = (R)__ldg(a.exa + node);
        Ey = (R)__ldg(a.eya + node);
        Ez = (R)__ldg(a.eza + node);
    }

    const R fx = charge * Ex + c.exf, fy = charge * Ey, fz = charge * Ez;
    const R rhoinv = (R)1 / rho;
    R ux = rhoinv * (mx * c.cflinv + fx * c.dt_half);
    R uy = rhoinv * (my * c.cflinv + fy * c.dt_half);
    R uz = rhoinv * (mz * c.cflinv + fz * c.dt_half);

    if (z == 0) {
        // LBM.cu:417-492
        const ZRef<R> z1 = load_zref(a.zref, 1);
        PullIdx P1;
        make_pull(P1, x, y, 1, NX, NY, NZ);
        const unsigned node1 = node + c.nxy;
        R dqm = pld(a.pp.ha[0] + node1) + c.w[0] * z1.dq0;
        R mxm = 0, mym = 0, mzm = 0;
#pragma unroll
        for (int d = 1; d < Q; ++d) {
            const unsigned s1 = local ? node1 : pull_src(P1, d);
            const int e = local ? 0 : ez_of(d);
            const R fm = pld(a.pp.fa[d] + s1) + c.w[cls_of(d)] * z1.dr(e);
            const R hm = pld(a.pp.ha[d] + s1) + c.w[cls_of(d)] * z1.dq(e);
            dqm += hm;
            if (ex_of(d)) mxm += ex_of(d) > 0 ? fm : -fm;
            if (ey_of(d)) mym += ey_of(d) > 0 ? fm : -fm;
            if (ez_of(d)) mzm += ez_of(d) > 0 ? fm : -fm;
        }
        const R chargem = z1.qref + dqm;
        R Exm, Eym, Ezm;
        if (!earr) {
            const unsigned row1 = row + c.nxy;
            Exm = (__ldg(a.phip + row1 + xm) - __ldg(a.phip + row1 + xp)) * c.inv2dx;
            Eym = (__ldg(a.phip + rym + c.nxy + x) - __ldg(a.phip + ryp + c.nxy + x)) * c.inv2dy;
            Ezm = (R)__ldg(a.ez00 + 1) +
                  (__ldg(a.phip + row + x) - __ldg(a.phip + row + 2 * c.nxy + x)) * c.inv2dz;
        } else {
            Exm = (R)__ldg(a.exa + node1);
            Eym = (R)__ldg(a.eya + node1);
            Ezm = (R)__ldg(a.eza + node1);
        }
        const R fxm = chargem * Exm + c.exf, fym = chargem * Eym, fzm = chargem * Ezm;
        ux = -rhoinv * (mxm * c.cflinv + fxm * c.dt_half);
        uy = -rhoinv * (mym * c.cflinv + fym * c.dt_half);
        uz = -rhoinv * (mzm * c.cflinv + fzm * c.dt_half);
    }

    a.qout[node] = charge;
    if (MACROS) {
        a.rout[node] = rho;
        a.uout[node] = ux;
        a.vout[node] = uy;
        a.wout[node] = uz;
    }

    // ---- f: collide (interior) or wall rule ----
    if (z == 0 || z == NZ - 1) {
        pst(a.pp.fb[0] + node, f[0]);
#pragma unroll
        for (int d = 1; d < Q; ++d) {
            R v = f[opp_of(d)];
            if (z == NZ - 1 && mw_sign_of(d) != 0) v += c.mw[d];
            pst(a.pp.fb[d] + node, v);
        }
    } else {
        const R rp_hi = c.rate_hi[0], rp_lo = c.rate_lo[0];
        const R rm_hi = c.rate_hi[1], rm_lo = c.rate_lo[1];
        const R usq = (R)0.5 * (ux * ux + uy * uy + uz * uz) * c.inv_cs2;
        const R tux = ux * c.inv_cs2cfl, tuy = uy * c.inv_cs2cfl, tuz = uz * c.inv_cs2cfl;
        const R uF = ux * fx + uy * fy + uz * fz;
        R WR[4], PK[4], QK[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            WR[k] = c.w[k] * rho;
            PK[k] = WR[k] * usq - c.w[k] * drho;
            QK[k] = c.c3[k] * uF;
        }
        pst(a.pp.fb[0] + node, f[0] - relax(rp_hi, rp_lo, f[0] + PK[0]) - QK[0]);
        if constexpr (sizeof(R) == 4) {
            PackF pk;
            pk.rp_hi = f2(rp_hi);
            pk.nrp_lo = f2(-rp_lo);
            pk.rm_hi = f2(rm_hi);
            pk.nrm_lo = f2(-rm_lo);
            pk.half = f2(0.5f);
            pk.mone = f2(-1.f);
#pragma unroll
            for (int k = 1; k < 4; ++k) {
                pk.PK[k] = f2(PK[k]);
                pk.QK[k] = f2(QK[k]);
                pk.nhWR[k] = f2(-0.5f * WR[k]);
                pk.nWR[k] = f2(-WR[k]);
                pk.nc1[k] = f2(-c.c1[k]);
                pk.nc2[k] = f2(-c.c2[k]);
            }
            pk.tux = tux;
            pk.tuy = tuy;
            pk.tuz = tuz;
            pk.fx = fx;
            pk.fy = fy;
            pk.fz = fz;
            f_pair2<1, 3>(f, pk, a.pp, node);
            f_pair2<7, 9>(f, pk, a.pp, node);
            f_pair2<11, 13>(f, pk, a.pp, node);
            f_pair2<15, 17>(f, pk, a.pp, node);
            f_pair2<19, 21>(f, pk, a.pp, node);
            f_pair2<23, 25>(f, pk, a.pp, node);
            {  // the fifth pair of class 1 alone
                constexpr int d = 5, o = 6, k = 1;
                const R cu = dot_e(d, tux, tuy, tuz);
                const R eF = dot_e(d, fx, fy, fz);
                const R X = (R)0.5 * (f[d] + f[o]) + PK[k] - (R)0.5 * WR[k] * cu * cu;
                const R A = relax(rp_hi, rp_lo, X) + QK[k] - c.c1[k] * cu * eF;
                const R Y = (R)0.5 * (f[d] - f[o]) - WR[k] * cu;
                const R B = relax(rm_hi, rm_lo, Y) - c.c2[k] * eF;
                pst(a.pp.fb[d] + node, f[d] - A - B);
                pst(a.pp.fb[o] + node, f[o] - A + B);
            }
        } else {
#pragma unroll
        for (int d = 1; d < Q; d += 2) {
            const int o = d + 1, k = cls_of(d);
            const R cu = dot_e(d, tux, tuy, tuz);
            const R eF = dot_e(d, fx, fy, fz);
            const R X = (R)0.5 * (f[d] + f[o]) + PK[k] - (R)0.5 * WR[k] * cu * cu;
            const R A = relax(rp_hi, rp_lo, X) + QK[k] - c.c1[k] * cu * eF;
            const R Y = (R)0.5 * (f[d] - f[o]) - WR[k] * cu;
            const R B = relax(rm_hi, rm_lo, Y) - c.c2[k] * eF;
            pst(a.pp.fb[d] + node, f[d] - A - B);
            pst(a.pp.fb[o] + node, f[o] - A + B);
        }
        }
    }

    // ---- g: collide (z <= NZ-2); the NZ-1 plane is written by z = NZ-2,
    // relative to q_ref(NZ-1) ----
    if (z != NZ - 1) {
        const R cp_hi = c.rate_hi[2], cp_lo = c.rate_lo[2];
        const R cm_hi = c.rate_hi[3], cm_lo = c.rate_lo[3];
        const R ucx = ux + c.K * Ex, ucy = uy + c.K * Ey, ucz = uz + c.K * Ez;
        const R usq = (R)0.5 * (ucx * ucx + ucy * ucy + ucz * ucz) * c.inv_cs2;
        const R tux = ucx * c.inv_cs2cfl, tuy = ucy * c.inv_cs2cfl, tuz = ucz * c.inv_cs2cfl;
        const bool dup = (z == NZ - 2);
        const unsigned nodeup = node + c.nxy;
        const R up = zr.up;  // q_w(z) - q_w(z+1)
        R WQ[4], PQ[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            WQ[k] = c.w[k] * charge;
            PQ[k] = WQ[k] * usq - c.w[k] * dq;
        }
        {
            const R out = h[0] - relax(cp_hi, cp_lo, h[0] + PQ[0]);
            pst(a.pp.hb[0] + node, z == 0 ? -out + (R)2 * (c.q0 - zr.qref) * c.w[0] : out);
            if (dup) pst(a.pp.hb[0] + nodeup, out + c.w[0] * up);
        }
        auto g_one = [&](auto dc) {
            constexpr int d = decltype(dc)::value, o = d + 1, k = cls_of(d);
            const R cu = dot_e(d, tux, tuy, tuz);
            const R X = (R)0.5 * (h[d] + h[o]) + PQ[k] - (R)0.5 * WQ[k] * cu * cu;
            const R Y = (R)0.5 * (h[d] - h[o]) - WQ[k] * cu;
            const R A = relax(cp_hi, cp_lo, X);
            R outd, outo;
            if (sizeof(R) == 4 && cm_hi == (R)2) {  // cancellation-free form, see g_pair2
                const R t = (R)2 * WQ[k] * cu;
                outd = (h[o] + t) - A + cm_lo * Y;
                outo = (h[d] - t) - A - cm_lo * Y;
            } else {
                const R B = relax(cm_hi, cm_lo, Y);
                outd = h[d] - A - B;
                outo = h[o] - A + B;
            }
            pst(a.pp.hb[d] + node, outd);
            pst(a.pp.hb[o] + node, outo);
            if (dup) {
                pst(a.pp.hb[d] + nodeup, outd + c.w[k] * up);
                pst(a.pp.hb[o] + nodeup, outo + c.w[k] * up);
            }
        };
        if constexpr (sizeof(R) == 4) {
            PackG pg;
            pg.cp_hi = f2(cp_hi);
            pg.ncp_lo = f2(-cp_lo);
            pg.cm_hi = f2(cm_hi);
            pg.ncm_lo = f2(-cm_lo);
            pg.cm_lo = f2(cm_lo);
            pg.over = cm_hi == 2.f;
            pg.half = f2(0.5f);
            pg.mone = f2(-1.f);
#pragma unroll
            for (int k = 1; k < 4; ++k) {
                pg.PQ[k] = f2(PQ[k]);
                pg.nhWQ[k] = f2(-0.5f * WQ[k]);
                pg.nWQ[k] = f2(-WQ[k]);
                pg.twoWQ[k] = f2(2.f * WQ[k]);
                pg.wup[k] = f2(c.w[k] * up);
            }
            pg.tux = tux;
            pg.tuy = tuy;
            pg.tuz = tuz;
            g_pair2<1, 3>(h, pg, a.pp, node, nodeup, dup);
            g_pair2<7, 9>(h, pg, a.pp, node, nodeup, dup);
            g_pair2<11, 13>(h, pg, a.pp, node, nodeup, dup);
            g_pair2<15, 17>(h, pg, a.pp, node, nodeup, dup);
            g_pair2<19, 21>(h, pg, a.pp, node, nodeup, dup);
            g_pair2<23, 25>(h, pg, a.pp, node, nodeup, dup);
            g_one(std::integral_constant<int, 5>{});
        } else {
#pragma unroll
            for (int d = 1; d < Q; d += 2) {
                const int o = d + 1, k = cls_of(d);
                const R cu = dot_e(d, tux, tuy, tuz);
                const R X = (R)0.5 * (h[d] + h[o]) + PQ[k] - (R)0.5 * WQ[k] * cu * cu;
                const R Y = (R)0.5 * (h[d] - h[o]) - WQ[k] * cu;
                const R A = relax(cp_hi, cp_lo, X);
                R outd, outo;
                if (sizeof(R) == 4 && cm_hi == (R)2) {  // cancellation-free form, see g_pair2
                    const R t = (R)2 * WQ[k] * cu;
                    outd = (h[o] + t) - A + cm_lo * Y;
                    outo = (h[d] - t) - A - cm_lo * Y;
                } else {
                    const R B = relax(cm_hi, cm_lo, Y);
                    outd = h[d] - A - B;
                    outo = h[o] - A + B;
                }
                pst(a.pp.hb[d] + node, outd);
                pst(a.pp.hb[o] + node, outo);
                if (dup) {
                    pst(a.pp.hb[d] + nodeup, outd + c.w[k] * up);
                    pst(a.pp.hb[o] + nodeup, outo + c.w[k] * up);
                }
            }
        }
    }
}

// The step of node (x, y, z) of the calling thread, its warp's plane sum into
// psum[slot()]; lanes that are not inside work on a valid node, so that the
// whole warp can take part in the plane sums, and store nothing.  (slot is
// called after the pull: a slot kept in registers over it costs loads in
// flight, 17 % of the step of 500 x 480 x 30 nodes in FP32.)
template <typename T, typename R, bool MACROS, typename S>
__device__ __forceinline__ void node_step(const StepArgs<T, R> &a, const KConst<R> &c, int x, int y,
                                          int z, bool inside, S slot, bool local, bool earr) {
    const unsigned node = (unsigned)x + (unsigned)c.nx * ((unsigned)y + (unsigned)c.ny * z);
    const ZRef<R> zr = load_zref(a.zref, z);
    PullIdx P;
    make_pull(P, x, y, z, c.nx, c.ny, c.nz);
    R f[Q], h[Q];
    pull_global<T, R>(f, h, a.pp, P, node, z, zr, c, local);
    const Moments<R> mo = moments(f, h, zr);
    warp_plane_sum(inside ? (float)mo.rho : 0.f, inside ? (float)mo.charge : 0.f, a.psum, slot());
    if (!inside) return;
    finish_node<T, R, MACROS>(f, h, mo, x, y, z, node, zr, a, c, local, earr);
}

// GENERAL = false: the steady-state step (pull, E from phi).  GENERAL = true
// adds two run-time switches used right after ehd_set_fields:
//   local_pops: the buffers hold the pre-collision populations of each node
//               (the reference's f1/h1 after init_equilibrium), so they are
//               read in place, without pull or injection rule;
//   e_arrays:   E comes from the uploaded FP64 arrays instead of phi.
// One thread per node, 128-thread blocks.
// One block of the per-node step: block (bxi, byi) of a gx x gy tiling of
// plane z (the grid indices are arguments so that a launch over several
// instances can map its blocks).
template <typename T, typename R, bool GENERAL, bool MACROS>
__device__ __forceinline__ void node_block(const StepArgs<T, R> &a, const KConst<R> &c, int bxi,
                                           int byi, int z, int gx, int gy, int local_pops,
                                           int e_arrays) {
    const bool local = GENERAL && local_pops;
    const bool earr = GENERAL && e_arrays;
    int x = bxi * blockDim.x + threadIdx.x;
    int y = byi * blockDim.y + threadIdx.y;
    const bool inside = x < c.nx && y < c.ny;
    if (!inside) {
        x = x < c.nx ? x : c.nx - 1;
        y = y < c.ny ? y : c.ny - 1;
    }
    node_step<T, R, MACROS>(
        a, c, x, y, z, inside,
        [&] {
            const int tid = threadIdx.x + blockDim.x * threadIdx.y;
            const int wpb = (blockDim.x * blockDim.y) >> 5;
            return (((size_t)z * gy + byi) * gx + bxi) * wpb + (tid >> 5);
        },
        local, earr);
}

template <typename T, typename R>
static StepArgs<T, R> make_step_args(const LbmArgs &la, const StepConst &c) {
    StepArgs<T, R> a;
    for (int d = 0; d < Q; ++d) {
        a.pp.fa[d] = (const typename PopT<T>::F *)la.fa + (size_t)d * c.n;
        a.pp.ha[d] = (const typename PopT<T>::G *)la.ha + (size_t)d * c.n;
        a.pp.fb[d] = (typename PopT<T>::F *)la.fb + (size_t)d * c.n;
        a.pp.hb[d] = (typename PopT<T>::G *)la.hb + (size_t)d * c.n;
    }
    a.phip = (const R *)la.phip;
    a.ez00 = la.ez00;
    a.exa = la.exa;
    a.eya = la.eya;
    a.eza = la.eza;
    a.qout = (R *)la.q;
    a.rout = (R *)la.rho;
    a.uout = (R *)la.u;
    a.vout = (R *)la.v;
    a.wout = (R *)la.w;
    a.zref = (const R *)la.zref;
    a.psum = la.psum;
    a.err = la.err;
    return a;
}

}  // namespace ehd
