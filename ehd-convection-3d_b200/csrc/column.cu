// column.cu -- steady-state steps of a 1 x 1 x NZ column (the hydrostatic
// start of every run, ehd_hydrostatic_column), many steps per launch.
//
// A column is a few dozen nodes stepped tens of thousands of times.  As six
// or seven launches a step (the per-node step, the plane means, the Poisson
// passes) it costs the launches alone: 24.9 us a step at NZ = 33 in FP64 on a
// B200, against well under a microsecond of arithmetic.  Here one block holds
// the whole state and runs any number of steps in one launch, so that a step
// costs its own chain of dependent operations.  Measured, FP64: a column of NZ = 33
// run 16,000 steps through ehd_hydrostatic_profile, its context's creation
// included, 388 -> 26 ms (24.3 -> 1.6 us a step; 30 ms with the moments as
// chains of additions and divisions by constants in the loop); 12 columns of
// NZ = 25 as one batch, 12,000 steps, 609 -> 38 ms (one block per column, side
// by side, where the batch's graph had held 84 launches a step).  With one
// multiprocessor busy the times scatter: other calls took up to 43 and 53 ms.
//
// Thread z of the first half of the block holds node z's flow populations f
// in registers, thread z of the second half its charge populations g (the two
// halves are whole warps), because the block is bound by the latency and the
// FP64 issue of one thread's arithmetic: two threads per node halve it.  With
// NX = NY = 1 the periodic x and y neighbours are the node itself, so only the
// 18 directions with e_z != 0 move, through shared memory.  A step has two
// block barriers: one after the moments (charge, momentum and the warps'
// partial sums of the Poisson solve are exchanged), one after the collisions.
//
// Poisson: on a column only the mean mode exists and phi' = 0.  With
// D_j = dz^2 s_j (s = -q / eps) and the edge differences
// s_i = phi_i - phi_{i+1}, the 3-point equation is s_i = s_{i-1} - D_i, so
//   s_i = s_0 - P_i,  P_i = D_1 + .. + D_i,
//   s_0 = (V + sum_j (n + 1 - j) D_j) / (n + 1)   (the drop over the gap is V)
// and Ez_i = (s_{i-1} + s_i) / (2 dz): one prefix sum and one weighted sum a
// step, in FP64.
//
// The state in global memory (populations, plane means, references, tables,
// fields) is read when the launch starts and written when it ends, as the
// per-step kernels leave it, so that every other entry point continues from
// it.  Collision algebra and rounding of the stored populations as in lbm.cu.
#include "column.h"
#include "common.cuh"

namespace ehd {

namespace {

// index of direction d among the 18 with e_z != 0 (in order of d), -1 else
__host__ __device__ constexpr int mov_of(int d) {
    int n = 0;
    for (int k = 0; k < d; ++k)
        if (ez_of(k) != 0) ++n;
    return ez_of(d) != 0 ? n : -1;
}
constexpr int kMov = 18;

// a value as it is stored in population type F
template <typename F, typename R>
__device__ __forceinline__ R stored(R v) {
    F s;
    pst(&s, v);
    return (R)plds(&s);
}

template <typename R>
__device__ __forceinline__ R relax_rate(R hi, R lo, R x) {
    return hi * x - lo * x;
}

template <typename R>
__device__ __forceinline__ R dot_dir(int d, R a, R b, R c) {
    R s = 0;
    if (ex_of(d)) s = ex_of(d) > 0 ? a : -a;
    if (ey_of(d)) s = ey_of(d) > 0 ? s + b : s - b;
    if (ez_of(d)) s = ez_of(d) > 0 ? s + c : s - c;
    return s;
}

// Sum of the products sign(d) v_d, sign in {-1, 0, 1}: in FP64 as a tree, a chain
// of 27 FP64 additions being the longest part of a step otherwise; in FP32 in the
// order of d, as the per-node kernel sums them (the tree's rounding took q, phi
// and E 7, 12 and 12 % further from the 64-bit run over 800 columns of 13 to 49
// planes, FP32 and mixed storage; in this order the distances are the per-node
// kernel's, and mostly its bits).
template <typename R, typename S>
__device__ __forceinline__ R dir_sum(const R (&v)[Q], S sign) {
    if constexpr (sizeof(R) == 4) {
        R a = 0;
#pragma unroll
        for (int d = 0; d < Q; ++d)
            if (sign(d) != 0) a += sign(d) > 0 ? v[d] : -v[d];
        return a;
    }
    R t[Q];
    int n = 0;
#pragma unroll
    for (int d = 0; d < Q; ++d)
        if (sign(d) != 0) t[n++] = sign(d) > 0 ? v[d] : -v[d];
#pragma unroll
    for (int w = 1; w < Q; w *= 2)
#pragma unroll
        for (int i = 0; i + w < Q; i += 2 * w)
            if (i + w < n) t[i] += t[i + w];
    return t[0];
}

}  // namespace

// dynamic shared memory, for nz nodes:
//   double wref[2][2 nz], mean[2][2 nz], ez[2][nz], wsum[2 * 32]
//   R mom[4][nz] (momentum x, y, z and rho), chg[nz]
//   R xf[18][nz], xg[18][nz], top[27] (the collector's stored g)
template <typename R>
static size_t column_smem(int nz) {
    return sizeof(double) * ((size_t)10 * nz + 64) + sizeof(R) * ((size_t)(5 + 2 * kMov) * nz + Q);
}

template <typename T, typename R, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
column_steps_kernel(const ColumnArgs a, const KConst<R> c, int nsteps) {
    using F = typename PopT<T>::F;
    using G = typename PopT<T>::G;
    extern __shared__ __align__(16) unsigned char column_raw[];
    const int nz = c.nz, n = nz - 2;
    double *wref = reinterpret_cast<double *>(column_raw);  // [parity][2 nz]
    double *mean = wref + 4 * nz;                           // [parity][2 nz]
    double *ezs = mean + 4 * nz;                            // [step & 1][nz]
    double *wsum = ezs + 2 * nz;                            // [warp][2]
    R *mom = reinterpret_cast<R *>(wsum + 64);              // [4][nz]
    R *chg = mom + 4 * nz;
    R *xf = chg + nz, *xg = xf + kMov * nz, *top = xg + kMov * nz;
    const int half = blockDim.x / 2;
    const bool flow = (int)threadIdx.x < half;
    const int z = flow ? (int)threadIdx.x : (int)threadIdx.x - half;
    const bool act = z < nz;
    const int lane = threadIdx.x & 31, gw = z >> 5;  // warp of this half
    const int zc = act ? z : nz - 1;
    const int zm = zc == 0 ? nz - 1 : zc - 1, zp = zc == nz - 1 ? 0 : zc + 1;
    // (no division in the loop but 1 / rho)
    const double kD = -(a.dz * a.dz) / a.eps, kN = 1.0 / (double)(n + 1), kE = 0.5 / a.dz;

    int p = a.parity;
    for (int i = threadIdx.x; i < 2 * nz; i += blockDim.x) {
        wref[i] = a.wref[0][i];
        wref[2 * nz + i] = a.wref[1][i];
        mean[i] = a.mean[0][i];
        mean[2 * nz + i] = a.mean[1][i];
    }
    // the stored populations of the thread's node (deviations from wref[p])
    R s[Q];
#pragma unroll
    for (int d = 0; d < Q; ++d) {
        R v;
        if (flow) v = (R)pld(reinterpret_cast<const F *>(a.f[p]) + (size_t)d * nz + zc);
        else v = (R)pld(reinterpret_cast<const G *>(a.h[p]) + (size_t)d * nz + zc);
        s[d] = v;
        if (act && mov_of(d) >= 0) (flow ? xf : xg)[mov_of(d) * nz + z] = v;
        if (!flow && z == nz - 1) top[d] = v;
    }
    // E of the first step: the mean field and what phi' the state came with
    // (zero after any Poisson solve); Ez of the electrodes from the planes inside
    if (!flow && act) {
        const R *ph = reinterpret_cast<const R *>(a.phip);
        const int e = z < 1 ? 1 : (z > n ? n : z);
        ezs[z] = (double)((R)a.ez00[e] + (ph[e - 1] - ph[e + 1]) * c.inv2dz);
    }
    __syncthreads();

    R rho = 0, charge = 0, ux = 0, uy = 0, uz = 0;
    R dev = 0;  // the half's zeroth moment before its reference is added
    R rref = 0, dr[3], qref = 0, dq[3];  // dr[e + 1]: source plane z - e
    double P = 0.0, D = 0.0, s0 = 0.0;
#pragma unroll 1
    for (int k = 0; k < nsteps; ++k) {
        const double *rd = wref + 2 * nz * p, *wr = wref + 2 * nz * (p ^ 1);
        const double *ez = ezs + nz * (k & 1);
        double *ez_next = ezs + nz * ((k & 1) ^ 1);
        // ---- pull and moments ----
        if (flow) {
            const double rw = wr[2 * zc];
            rref = (R)rw;
            dr[0] = (R)(rd[2 * zp] - rw);
            dr[1] = (R)(rd[2 * zc] - rw);
            dr[2] = (R)(rd[2 * zm] - rw);
#pragma unroll
            for (int d = 0; d < Q; ++d) {
                const int e = ez_of(d);
                const R v = e == 0 ? s[d] : xf[mov_of(d) * nz + (e > 0 ? zm : zp)];
                s[d] = v + c.w[cls_of(d)] * dr[e + 1];
            }
            dev = dir_sum(s, [](int) { return 1; });
            rho = rref + dev;
            if (act) {
                mom[z] = dir_sum(s, [](int d) { return ex_of(d); });
                mom[nz + z] = dir_sum(s, [](int d) { return ey_of(d); });
                mom[2 * nz + z] = dir_sum(s, [](int d) { return ez_of(d); });
                mom[3 * nz + z] = rho;
            }
        } else {
            const double qw = wr[2 * zc + 1];
            qref = (R)qw;
            dq[0] = (R)(rd[2 * zp + 1] - qw);
            dq[1] = (R)(rd[2 * zc + 1] - qw);
            dq[2] = (R)(rd[2 * zm + 1] - qw);
            if (z == nz - 1) {
#pragma unroll
                for (int d = 0; d < Q; ++d) s[d] = top[d];
            }
            if (z == 0) {
                // the injector: g_d = -g_opp(d) + 2 q0 w_d of its own values
                // (LBM.cu:1320-1348), on deviations
                const R inj = (R)2 * (c.q0 - qref) - dq[1];
                s[0] += c.w[0] * dq[1];
#pragma unroll
                for (int d = 1; d < Q; d += 2) {
                    const R t = s[d];
                    s[d] = -s[d + 1] + inj * c.w[cls_of(d)];
                    s[d + 1] = -t + inj * c.w[cls_of(d)];
                }
            } else {
#pragma unroll
                for (int d = 0; d < Q; ++d) {
                    const int e = ez_of(d);
                    const R v = e == 0 ? s[d] : xg[mov_of(d) * nz + (e > 0 ? zm : zp)];
                    s[d] = v + c.w[cls_of(d)] * dq[e + 1];
                }
            }
            dev = dir_sum(s, [](int) { return 1; });
            charge = qref + dev;
            if (act) chg[z] = charge;
            // the warp's prefix sum of D and sum of (n + 1 - z) D
            D = act && z >= 1 && z <= n ? (double)charge * kD : 0.0;
            P = D;
            double W = (double)(n + 1 - z) * D;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, P, o);
                if (lane >= o) P += t;
                W += __shfl_xor_sync(0xffffffffu, W, o);
            }
            if (lane == 31) {
                wsum[2 * gw] = P;
                wsum[2 * gw + 1] = W;
            }
        }
        __syncthreads();
        // ---- velocity (both halves), the next step's E (second half) ----
        const int zv = z == 0 ? 1 : zc;  // the injector mirrors the plane above it
        const R Ez = (R)ez[zc], Ev = (R)ez[zv];
        const R cv = chg[zv];
        if (!flow) rho = mom[3 * nz + zc];
        else charge = chg[zc];
        {
            const R fx = c.exf, fz = cv * Ev;
            const R sg = z == 0 ? (R)-1 : (R)1;
            const R rhoinv = sg / rho;
            ux = rhoinv * (mom[zv] * c.cflinv + fx * c.dt_half);
            uy = rhoinv * (mom[nz + zv] * c.cflinv);
            uz = rhoinv * (mom[2 * nz + zv] * c.cflinv + fz * c.dt_half);
        }
        if (flow) {
            if (act) {
                mean[2 * nz * (p ^ 1) + 2 * z] = (double)(float)rho;
                // the reference of the next write of this buffer: the means
                // of the state read now (the collector takes the plane below)
                wref[2 * nz * p + 2 * z] = mean[2 * nz * p + 2 * (z == nz - 1 ? nz - 2 : z)];
            }
            if (z == 0 || z == nz - 1) {
                // bounce-back, the moving upper wall
#pragma unroll
                for (int d = 1; d < Q; d += 2) {
                    const R t = s[d];
                    s[d] = s[d + 1];
                    s[d + 1] = t;
                    if (z == nz - 1) {
                        if (mw_sign_of(d) != 0) s[d] += c.mw[d];
                        if (mw_sign_of(d + 1) != 0) s[d + 1] += c.mw[d + 1];
                    }
                }
            } else {
                const R fx = c.exf, fz = charge * Ez;
                const R rp_hi = c.rate_hi[0], rp_lo = c.rate_lo[0];
                const R rm_hi = c.rate_hi[1], rm_lo = c.rate_lo[1];
                const R usq = (R)0.5 * (ux * ux + uy * uy + uz * uz) * c.inv_cs2;
                const R tux = ux * c.inv_cs2cfl, tuy = uy * c.inv_cs2cfl, tuz = uz * c.inv_cs2cfl;
                const R uF = ux * fx + uz * fz;
                R WR[4], PK[4], QK[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    WR[q] = c.w[q] * rho;
                    PK[q] = WR[q] * usq - c.w[q] * dev;
                    QK[q] = c.c3[q] * uF;
                }
                s[0] = s[0] - relax_rate(rp_hi, rp_lo, s[0] + PK[0]) - QK[0];
#pragma unroll
                for (int d = 1; d < Q; d += 2) {
                    const int o = d + 1, q = cls_of(d);
                    const R cu = dot_dir(d, tux, tuy, tuz);
                    const R eF = dot_dir(d, fx, (R)0, fz);
                    const R X = (R)0.5 * (s[d] + s[o]) + PK[q] - (R)0.5 * WR[q] * cu * cu;
                    const R Y = (R)0.5 * (s[d] - s[o]) - WR[q] * cu;
                    R od, oo;
                    if (sizeof(R) == 4 && d != 5) {  // in the order of f_pair2
                        const R A = fma(-c.c1[q], cu * eF, fma(rp_hi, X, fma(-rp_lo, X, QK[q])));
                        const R B = fma(rm_hi, Y, fma(-rm_lo, Y, -c.c2[q] * eF));
                        od = s[d] - (A + B);
                        oo = (s[o] + B) - A;
                    } else {
                        const R A = relax_rate(rp_hi, rp_lo, X) + QK[q] - c.c1[q] * cu * eF;
                        const R B = relax_rate(rm_hi, rm_lo, Y) - c.c2[q] * eF;
                        od = s[d] - A - B;
                        oo = s[o] - A + B;
                    }
                    s[d] = od;
                    s[o] = oo;
                }
            }
#pragma unroll
            for (int d = 0; d < Q; ++d) {
                s[d] = stored<F>(s[d]);
                if (mov_of(d) >= 0 && act) xf[mov_of(d) * nz + z] = s[d];
            }
        } else {
            const double up = wr[2 * zc + 1] - wr[2 * zp + 1];  // q_w(z) - q_w(z + 1)
            if (act) {
                mean[2 * nz * (p ^ 1) + 2 * z + 1] = (double)(float)charge;
                wref[2 * nz * p + 2 * z + 1] = mean[2 * nz * p + 2 * (z == nz - 1 ? nz - 2 : z) + 1];
            }
            {
                double W = 0.0, off = 0.0;
                for (int w = 0; w < (nz + 31) / 32; ++w) {
                    if (w < gw) off += wsum[2 * w];
                    W += wsum[2 * w + 1];
                }
                P += off;
                s0 = (a.voltage + W) * kN;
                const double e = (2.0 * s0 - 2.0 * P + D) * kE;
                if (z >= 1 && z <= n) ez_next[z] = e;
                if (z == 1) ez_next[0] = e;
                if (z == n) ez_next[nz - 1] = e;
            }
            if (z < nz - 1) {
                const R cp_hi = c.rate_hi[2], cp_lo = c.rate_lo[2];
                const R cm_hi = c.rate_hi[3], cm_lo = c.rate_lo[3];
                const R ucz = uz + c.K * Ez;
                const R usq = (R)0.5 * (ux * ux + uy * uy + ucz * ucz) * c.inv_cs2;
                const R tux = ux * c.inv_cs2cfl, tuy = uy * c.inv_cs2cfl, tuz = ucz * c.inv_cs2cfl;
                R WQ[4], PQ[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    WQ[q] = c.w[q] * charge;
                    PQ[q] = WQ[q] * usq - c.w[q] * dev;
                }
                const R out0 = s[0] - relax_rate(cp_hi, cp_lo, s[0] + PQ[0]);
                s[0] = z == 0 ? -out0 + (R)2 * (c.q0 - qref) * c.w[0] : out0;
#pragma unroll
                for (int d = 1; d < Q; d += 2) {
                    const int o = d + 1, q = cls_of(d);
                    const R cu = dot_dir(d, tux, tuy, tuz);
                    const R X = (R)0.5 * (s[d] + s[o]) + PQ[q] - (R)0.5 * WQ[q] * cu * cu;
                    const R Y = (R)0.5 * (s[d] - s[o]) - WQ[q] * cu;
                    const R A = relax_rate(cp_hi, cp_lo, X);
                    R od, oo;
                    if (sizeof(R) == 4 && cm_hi == (R)2) {  // cancellation-free form, see g_pair2
                        const R t = (R)2 * WQ[q] * cu;
                        od = (s[o] + t) - A + cm_lo * Y;
                        oo = (s[d] - t) - A - cm_lo * Y;
                    } else if (sizeof(R) == 4 && d != 5) {  // in the order of g_pair2
                        const R B = relax_rate(cm_hi, cm_lo, Y);
                        od = s[d] - (A + B);
                        oo = (s[o] + B) - A;
                    } else {
                        const R B = relax_rate(cm_hi, cm_lo, Y);
                        od = s[d] - A - B;
                        oo = s[o] - A + B;
                    }
                    s[d] = od;
                    s[o] = oo;
                }
                if (z == nz - 2) {
                    // the collector's g: a copy of this plane's, relative to
                    // its own reference (LBM.cu:1173-1200)
#pragma unroll
                    for (int d = 0; d < Q; ++d) {
                        const R v = stored<G>(s[d] + c.w[cls_of(d)] * (R)up);
                        top[d] = v;
                        if (mov_of(d) >= 0) xg[mov_of(d) * nz + z + 1] = v;
                    }
                }
#pragma unroll
                for (int d = 0; d < Q; ++d) {
                    s[d] = stored<G>(s[d]);
                    if (mov_of(d) >= 0) xg[mov_of(d) * nz + z] = s[d];
                }
            }
        }
        p ^= 1;
        __syncthreads();
    }

    // ---- the state as the per-step kernels leave it ----
    if (flow) {
        if (act) {
            F *f = reinterpret_cast<F *>(a.f[p]);
#pragma unroll
            for (int d = 0; d < Q; ++d) pst(f + (size_t)d * nz + z, s[d]);
            reinterpret_cast<R *>(a.rho)[z] = rho;
            reinterpret_cast<R *>(a.u)[z] = ux;
            reinterpret_cast<R *>(a.v)[z] = uy;
            reinterpret_cast<R *>(a.w)[z] = uz;
            if (z >= 1 && z <= n) reinterpret_cast<R *>(a.phip)[z] = (R)0;
        }
    } else if (act) {
        G *h = reinterpret_cast<G *>(a.h[p]);
#pragma unroll
        for (int d = 0; d < Q; ++d) pst(h + (size_t)d * nz + z, z == nz - 1 ? top[d] : s[d]);
        reinterpret_cast<R *>(a.q)[z] = charge;
        a.ez00[z] = ezs[nz * (nsteps & 1) + z];
        // phi_z = V - (s_0 + .. + s_{z-1})
        double ph = a.voltage, edge = s0;
        for (int i = 0; i < z; ++i) {
            if (i >= 1) edge -= (double)chg[i] * kD;
            ph -= edge;
        }
        a.phi00[z] = z == nz - 1 ? 0.0 : ph;
    }
    for (int i = threadIdx.x; i < 2 * nz; i += blockDim.x) {
        a.wref[0][i] = wref[i];
        a.wref[1][i] = wref[2 * nz + i];
        a.mean[0][i] = mean[i];
        a.mean[1][i] = mean[2 * nz + i];
    }
    // the step kernels' tables: reading buffer p and writing p ^ 1 next, and
    // the one of the last step
    if (act) {
        const double *rd = wref + 2 * nz * p, *wr = wref + 2 * nz * (p ^ 1);
        const int i = flow ? 0 : 1;
        R *kt = reinterpret_cast<R *>(a.ktab[p]) + 10 * z;
        R *kl = reinterpret_cast<R *>(a.ktab[p ^ 1]) + 10 * z;
        const double w0 = wr[2 * z + i];
        kt[i] = (R)w0;
        kt[2 + 3 * i] = (R)(rd[2 * zm + i] - w0);
        kt[3 + 3 * i] = (R)(rd[2 * z + i] - w0);
        kt[4 + 3 * i] = (R)(rd[2 * zp + i] - w0);
        kl[i] = flow ? rref : qref;
        kl[2 + 3 * i] = flow ? dr[2] : dq[2];
        kl[3 + 3 * i] = flow ? dr[1] : dq[1];
        kl[4 + 3 * i] = flow ? dr[0] : dq[0];
        if (flow) {
            kt[8] = (R)(wr[2 * z + 1] - wr[2 * zp + 1]);
            kt[9] = (R)0;
            kl[8] = (R)(rd[2 * z + 1] - rd[2 * zp + 1]);
            kl[9] = (R)0;
        }
    }
}

bool column_usable(int nx, int ny, int nz) {
    // two threads a node in one block of at most 512; the shared arrays of
    // 256 nodes in FP64 are 104 KB
    return nx == 1 && ny == 1 && nz <= 256;
}

namespace {
// 256 threads (NZ <= 128) leave each its 255 registers; above, 128
template <typename T, typename R>
cudaError_t column_prepare() {
    cudaError_t e = allow_max_dynamic_smem(column_steps_kernel<T, R, 256>);
    return e == cudaSuccess ? allow_max_dynamic_smem(column_steps_kernel<T, R, 512>) : e;
}
template <typename T, typename R>
cudaError_t column_launch(const ColumnArgs &a, const StepConst &c, int nsteps, cudaStream_t s) {
    const KConst<R> k = make_kconst<R>(c);
    const int threads = 2 * ((c.nz + 31) / 32 * 32);
    const size_t sm = column_smem<R>(c.nz);
    if (threads <= 256) column_steps_kernel<T, R, 256><<<1, threads, sm, s>>>(a, k, nsteps);
    else column_steps_kernel<T, R, 512><<<1, threads, sm, s>>>(a, k, nsteps);
    return cudaGetLastError();
}
}  // namespace

cudaError_t prepare_column(int prec) {
    switch (prec) {
        case 0: return column_prepare<double, double>();
        case 1: return column_prepare<float, float>();
        case 2: return column_prepare<__half, float>();
        case 3: return column_prepare<__nv_bfloat16, float>();
        default: return column_prepare<Mix16, float>();
    }
}

cudaError_t launch_column_steps(int prec, const ColumnArgs &a, const StepConst &c, int nsteps,
                                cudaStream_t s) {
    switch (prec) {
        case 0: return column_launch<double, double>(a, c, nsteps, s);
        case 1: return column_launch<float, float>(a, c, nsteps, s);
        case 2: return column_launch<__half, float>(a, c, nsteps, s);
        case 3: return column_launch<__nv_bfloat16, float>(a, c, nsteps, s);
        default: return column_launch<Mix16, float>(a, c, nsteps, s);
    }
}

}  // namespace ehd
