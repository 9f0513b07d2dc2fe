// lbm_pair.cu -- the steady-state step with two nodes per thread, for FP32
// compute with FP32 or FP16 flow populations (FP32, FP16 and mixed storage) on
// grids of even NX.
//
// With 2-byte populations the one-node-per-thread kernel is bound by the
// issue of its instructions, not by memory: about 1,400 a node, at 512 x 512 x
// 129 2.23 ms against 1.17 ms for its bytes at the copy bandwidth.  Here a
// thread owns the nodes x and x + 1 of a row (x even), and every operation
// from the loads to the stores is one instruction for both: a population pair
// is one 32-bit word (two, for the directions with e_x != 0, whose halves are
// put together by a byte permute), the arithmetic runs on packed FP32x2
// values, one per node, and a result pair is one conversion and one 32-bit
// store.  Planes are walked as runs of node pairs, so that no lane is idle at
// the end of a row.  That is 860 instructions a node; with the 168 registers
// of three blocks a multiprocessor (12 warps) the step of 512 x 512 x 129 in
// FP16 went 2.82 -> 2.16 ms (this kernel 1.66 ms; with two or four blocks,
// 255 or 128 registers, 2.62 and 2.66 ms), 256 x 256 x 129 in mixed storage
// 0.690 -> 0.586 ms (there against the row kernel), 302 x 266 x 38 mixed 333 ->
// 210 us for the LBM half.  What is left to the floor is load latency at that
// occupancy (2.3 of 5.7 cycles between issues).
//
// FP32 populations are 64-bit words: 760 instructions a node and 128 loads of
// a thread in flight, where the row kernel of lbm.cu spends about 1,340 and its
// warps wait on whole rows.  LBM half of a step in us, the kernel it replaced /
// this: 256 x 256 x 129 663 / 582 (6.62 TB/s of its 456 algorithmic bytes a node,
// 6.0 by the DRAM traffic), 128 x 128 x 65 96.5 / 83.2, 64 x 64 x 33 13.5 / 11.0,
// 200 x 200 x 65 241 / 193 (rows); 122 x 122 x 101 148 / 118, 302 x 266 x 38 301 /
// 232, 512 x 512 x 33 764 / 620, 38 x 38 x 40 9.2 / 7.5 (one node per thread).
//
// The injector plane z = 0 is stepped with one node per thread (node_step), by
// blocks of the same launch in FP32 and on small grids, in a launch of its own
// on large ones.  The pull, collision and wall rules are those of finish_node, on the
// same deviations and up to the plane sums in the same operations (rho and q of a
// step are the same bits).  (Rows through shared memory, as in lbm_rows_kernel, with
// g read twice to stay at 128 registers, took 2.53 ms where this takes 2.15.)
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "lbm_node.cuh"

namespace ehd {

namespace {

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// e_d . (a, b, c), the components of e_d in {-1, 0, 1}; m = (-1, -1)
__device__ __forceinline__ float2 dot2(int d, float2 a, float2 b, float2 c, float2 m) {
    float2 s = make_float2(0.f, 0.f);
    bool any = false;
    const int e[3] = {ex_of(d), ey_of(d), ez_of(d)};
    const float2 v[3] = {a, b, c};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (e[i] == 0) continue;
        if (!any) s = e[i] > 0 ? v[i] : neg2(v[i]);
        else s = e[i] > 0 ? add2(s, v[i]) : fma2(m, v[i], s);
        any = true;
    }
    return s;
}

// The pair (x + c, x + c + 1) of a direction's row, c = -e_x: from byte
// offsets of the words holding x - 2, x and x + 2 (wrapped in the row).
__device__ __forceinline__ float2 pull(const __half *p, unsigned om, unsigned o0, unsigned op, int ex) {
    const char *b = reinterpret_cast<const char *>(p);
    unsigned w = __ldg(reinterpret_cast<const unsigned *>(b + o0));
    if (ex > 0) w = __byte_perm(__ldg(reinterpret_cast<const unsigned *>(b + om)), w, 0x5432);
    if (ex < 0) w = __byte_perm(w, __ldg(reinterpret_cast<const unsigned *>(b + op)), 0x5432);
    return __half22float2(*reinterpret_cast<const __half2 *>(&w));
}
// the same for FP32 rows: twice the byte offsets
__device__ __forceinline__ float2 pull(const float *p, unsigned om, unsigned o0, unsigned op, int ex) {
    const char *b = reinterpret_cast<const char *>(p);
    if (ex == 0) return __ldg(reinterpret_cast<const float2 *>(b + 2 * o0));
    const float *q = reinterpret_cast<const float *>(b + 2 * o0);
    if (ex > 0) return make_float2(__ldg(reinterpret_cast<const float *>(b + 2 * om) + 1), __ldg(q));
    return make_float2(__ldg(q + 1), __ldg(reinterpret_cast<const float *>(b + 2 * op)));
}
__device__ __forceinline__ void put(__half *p, unsigned o, float2 v) {
    *reinterpret_cast<__half2 *>(reinterpret_cast<char *>(p) + o) = __float22half2_rn(v);
}
__device__ __forceinline__ void put(float *p, unsigned o, float2 v) {
    *reinterpret_cast<float2 *>(reinterpret_cast<char *>(p) + 2 * o) = v;
}

constexpr int kPairThreads = 128;

}  // namespace

template <typename T>
struct PairArgs {
    PopPtrs<T> pp;
    const float *phip;
    const double *ez00;
    float *qout, *rout, *uout, *vout, *wout;
    const float *zref;
    float2 *psum;  // [z][block][8]
};

// Block b of plane 0, one node per thread: two of them fill the eight plane-sum
// slots of a block of pairs.
template <typename T, bool MACROS>
__device__ __forceinline__ void plane0_block(const StepArgs<T, float> &a, const KConst<float> &c,
                                             int b) {
    const int i = b * kPairThreads + threadIdx.x;
    const bool in = i < c.nx * c.ny;
    const int y = in ? i / c.nx : c.ny - 1, x = in ? i - y * c.nx : c.nx - 1;
    node_step<T, float, MACROS>(
        a, c, x, y, 0, in, [&] { return b * (kPairThreads / 32) + (threadIdx.x >> 5); }, false,
        false);
}
template <typename T, bool MACROS>
__global__ void __launch_bounds__(kPairThreads, 4)
lbm_plane0_kernel(const StepArgs<T, float> a, const KConst<float> c) {
    step_enter();
    plane0_block<T, MACROS>(a, c, blockIdx.x);
}

// Planes z >= 1 (Args = PairArgs), or plane 0 as well (Args = StepArgs), as
// blockIdx.y = 0, 1 with twice as many blocks as a plane of pairs.
template <typename T, bool MACROS, typename Args>
__global__ void __launch_bounds__(kPairThreads, 3)
lbm_pair_kernel(const Args a, const KConst<float> c) {
    step_enter();
    constexpr bool kPlane0 = std::is_same<Args, StepArgs<T, float>>::value;
    const int NX = c.nx, NY = c.ny, NZ = c.nz, hx = NX / 2;
    const int pairs = hx * NY;
    if constexpr (kPlane0) {
        if (blockIdx.y < 2) {
            plane0_block<T, MACROS>(a, c, 2 * blockIdx.x + blockIdx.y);
            return;
        }
    }
    const int z = kPlane0 ? (int)blockIdx.y - 1 : 1 + (int)blockIdx.y;
    const int i = blockIdx.x * kPairThreads + threadIdx.x;
    // lanes past the plane work on its last pair (the whole warp takes part in
    // the plane sums) and store nothing
    const bool inside = i < pairs;
    const int ic = inside ? i : pairs - 1;
    const int y = ic / hx, xp2 = ic - y * hx;  // pair of the row
    const int ym = y == 0 ? NY - 1 : y - 1, yp = y == NY - 1 ? 0 : y + 1;
    const int zm = z - 1, zp = z == NZ - 1 ? 0 : z + 1;
    // byte offsets of 2-byte elements: word of the pair, of the pair before
    // and after it in the row
    const unsigned x0 = 4u * xp2, xm = xp2 == 0 ? 4u * (hx - 1) : x0 - 4u,
                   xq = xp2 == hx - 1 ? 0u : x0 + 4u;
    unsigned row[3][3];  // [e_y + 1][e_z + 1]: byte offset of row (y - e_y, z - e_z)
    {
        const int ys[3] = {yp, y, ym}, zs[3] = {zp, z, zm};
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
            for (int v = 0; v < 3; ++v)
                row[u][v] = 2u * (unsigned)NX * ((unsigned)ys[u] + (unsigned)NY * (unsigned)zs[v]);
    }
    float zr[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) zr[k] = __ldg(a.zref + 10 * z + k);
    const float2 mone = dup(-1.f), half = dup(0.5f);

    // ---- pull and moments ----
    float2 f[Q], h[Q];
    float2 drho = dup(0.f), dq = dup(0.f), mx = dup(0.f), my = dup(0.f), mz = dup(0.f);
#pragma unroll
    for (int d = 0; d < Q; ++d) {
        const unsigned r = row[ey_of(d) + 1][ez_of(d) + 1];
        f[d] = pull(a.pp.fa[d], r + xm, r + x0, r + xq, ex_of(d));
        h[d] = pull(a.pp.ha[d], r + xm, r + x0, r + xq, ex_of(d));
    }
    // To this step's references, in one rounding as in pull_global: w times the
    // shift, rounded before it is added, would be off by the same amount at every
    // node of a plane (FP32, 64 x 64 x 33, 100 steps, 24 starts: distance of u and
    // phi from the 64-bit run 1.012 and 1.006 times the per-node kernel's, 1.000
    // and 1.001 so).  256 x 256 x 129 in FP32 643 us a step, 640 with the rounded
    // products; 122 x 122 x 101 167 and 161.  16-bit f by e_z, which leaves the
    // kernel registers for more loads: 256 x 256 x 129 in FP16 499 us, in the order
    // of d 508.
    auto shift = [&](int d) {
        const float2 w = dup(c.w[cls_of(d)]);
        f[d] = fma2(w, dup(ez_of(d) > 0 ? zr[2] : (ez_of(d) < 0 ? zr[4] : zr[3])), f[d]);
        h[d] = fma2(w, dup(ez_of(d) > 0 ? zr[5] : (ez_of(d) < 0 ? zr[7] : zr[6])), h[d]);
    };
    if constexpr (std::is_same<T, float>::value) {
#pragma unroll
        for (int d = 0; d < Q; ++d) shift(d);
    } else {
#pragma unroll
        for (int e = -1; e <= 1; ++e)
#pragma unroll
            for (int d = 0; d < Q; ++d)
                if (ez_of(d) == e) shift(d);
    }
#pragma unroll
    for (int d = 0; d < Q; ++d) {
        drho = add2(drho, f[d]);
        dq = add2(dq, h[d]);
        if (ex_of(d)) mx = ex_of(d) > 0 ? add2(mx, f[d]) : fma2(mone, f[d], mx);
        if (ey_of(d)) my = ey_of(d) > 0 ? add2(my, f[d]) : fma2(mone, f[d], my);
        if (ez_of(d)) mz = ez_of(d) > 0 ? add2(mz, f[d]) : fma2(mone, f[d], mz);
    }
    const float2 rho = add2(dup(zr[0]), drho), charge = add2(dup(zr[1]), dq);
    {
        // FP32 sums of 32 nodes, as in the other step kernels: each half of the
        // warp has a slot
        float2 v = make_float2(inside ? rho.x + rho.y : 0.f, inside ? charge.x + charge.y : 0.f);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if ((threadIdx.x & 15) == 0)
            a.psum[((size_t)z * gridDim.x + blockIdx.x) * (kPairThreads / 16) +
                   (threadIdx.x >> 4)] = v;
    }
    if (!inside) return;

    // ---- E = -grad(phi), central differences (see finish_node) ----
    const unsigned node = row[1][1] / 2u + 2u * xp2;  // of the pair's first node
    float2 Ex, Ey, Ez;
    {
        auto pair_at = [&](unsigned o) { return __ldg(reinterpret_cast<const float2 *>(a.phip + o)); };
        const unsigned r = row[1][1] / 2u;
        const float2 p0 = pair_at(r + 2u * xp2);
        const float pm = __ldg(a.phip + r + xm / 2u + 1u), pp = __ldg(a.phip + r + xq / 2u);
        Ex = mul2(fma2(mone, make_float2(p0.y, pp), make_float2(pm, p0.x)), dup(c.inv2dx));
        // row[][1]: e_y = +1 is the row y - 1
        Ey = mul2(fma2(mone, pair_at(row[0][1] / 2u + 2u * xp2), pair_at(row[2][1] / 2u + 2u * xp2)),
                  dup(c.inv2dy));
        const int zc = z > NZ - 2 ? NZ - 2 : z;
        const unsigned nc = node - (unsigned)(z - zc) * c.nxy;
        Ez = fma2(fma2(mone, pair_at(nc + c.nxy), pair_at(nc - c.nxy)), dup(c.inv2dz),
                  dup((float)__ldg(a.ez00 + zc)));
    }
    const float2 fx = fma2(charge, Ex, dup(c.exf)), fy = mul2(charge, Ey), fz = mul2(charge, Ez);
    const float2 rinv = make_float2(1.f / rho.x, 1.f / rho.y);
    const float2 ci = dup(c.cflinv), dh = dup(c.dt_half);
    const float2 ux = mul2(rinv, fma2(mx, ci, mul2(fx, dh)));
    const float2 uy = mul2(rinv, fma2(my, ci, mul2(fy, dh)));
    const float2 uz = mul2(rinv, fma2(mz, ci, mul2(fz, dh)));
    *reinterpret_cast<float2 *>(a.qout + node) = charge;
    if (MACROS) {
        *reinterpret_cast<float2 *>(a.rout + node) = rho;
        *reinterpret_cast<float2 *>(a.uout + node) = ux;
        *reinterpret_cast<float2 *>(a.vout + node) = uy;
        *reinterpret_cast<float2 *>(a.wout + node) = uz;
    }
    const unsigned o = 2u * node;  // byte offset of 2-byte elements

    // ---- f: collision, or the wall rule of the collector plane ----
    if (z == NZ - 1) {
        put(a.pp.fb[0], o, f[0]);
#pragma unroll
        for (int d = 1; d < Q; ++d) {
            float2 v = f[opp_of(d)];
            if (mw_sign_of(d) != 0) v = add2(v, dup(c.mw[d]));
            put(a.pp.fb[d], o, v);
        }
        return;  // its g is written by the plane below
    }
    {
        const float2 usq = mul2(fma2(ux, ux, fma2(uy, uy, mul2(uz, uz))), dup(0.5f * c.inv_cs2));
        const float2 t = dup(c.inv_cs2cfl);
        const float2 tux = mul2(ux, t), tuy = mul2(uy, t), tuz = mul2(uz, t);
        const float2 uF = fma2(ux, fx, fma2(uy, fy, mul2(uz, fz)));
        const float2 rp_hi = dup(c.rate_hi[0]), nrp_lo = dup(-c.rate_lo[0]);
        const float2 rm_hi = dup(c.rate_hi[1]), nrm_lo = dup(-c.rate_lo[1]);
        float2 nWR[4], PK[4], QK[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            nWR[k] = mul2(dup(-c.w[k]), rho);
            PK[k] = fma2(neg2(nWR[k]), usq, mul2(dup(-c.w[k]), drho));
            QK[k] = mul2(dup(c.c3[k]), uF);
        }
        {
            const float2 X = add2(f[0], PK[0]);
            const float2 A = fma2(rp_hi, X, fma2(nrp_lo, X, QK[0]));
            put(a.pp.fb[0], o, fma2(mone, A, f[0]));
        }
#pragma unroll
        for (int d = 1; d < Q; d += 2) {
            const int k = cls_of(d);
            const float2 fd = f[d], fo = f[d + 1];
            const float2 cu = dot2(d, tux, tuy, tuz, mone), eF = dot2(d, fx, fy, fz, mone);
            const float2 wc = mul2(nWR[k], cu);
            float2 X = fma2(half, add2(fd, fo), PK[k]);
            X = fma2(mul2(half, wc), cu, X);
            float2 A = fma2(nrp_lo, X, QK[k]);
            A = fma2(rp_hi, X, A);
            A = fma2(dup(-c.c1[k]), mul2(cu, eF), A);
            const float2 Y = fma2(half, fma2(mone, fo, fd), wc);
            float2 B = fma2(nrm_lo, Y, mul2(dup(-c.c2[k]), eF));
            B = fma2(rm_hi, Y, B);
            put(a.pp.fb[d], o, fma2(mone, add2(A, B), fd));
            put(a.pp.fb[d + 1], o, fma2(mone, A, add2(fo, B)));
        }
    }

    // ---- g: collision; the plane below the collector writes the collector's
    // copy too, relative to its reference ----
    {
        const float2 Kd = dup(c.K);
        const float2 ucx = fma2(Kd, Ex, ux), ucy = fma2(Kd, Ey, uy), ucz = fma2(Kd, Ez, uz);
        const float2 usq = mul2(fma2(ucx, ucx, fma2(ucy, ucy, mul2(ucz, ucz))), dup(0.5f * c.inv_cs2));
        const float2 t = dup(c.inv_cs2cfl);
        const float2 tux = mul2(ucx, t), tuy = mul2(ucy, t), tuz = mul2(ucz, t);
        const float2 cp_hi = dup(c.rate_hi[2]), ncp_lo = dup(-c.rate_lo[2]);
        const float2 cm_hi = dup(c.rate_hi[3]), cm_lo = dup(c.rate_lo[3]);
        const bool over = c.rate_hi[3] == 2.f, top = z == NZ - 2;
        const unsigned ou = o + 2u * c.nxy;
        float2 nWQ[4], PQ[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            nWQ[k] = mul2(dup(-c.w[k]), charge);
            PQ[k] = fma2(neg2(nWQ[k]), usq, mul2(dup(-c.w[k]), dq));
        }
        {
            const float2 X = add2(h[0], PQ[0]);
            const float2 A = fma2(cp_hi, X, mul2(ncp_lo, X));
            const float2 out = fma2(mone, A, h[0]);
            put(a.pp.hb[0], o, out);
            if (top) put(a.pp.hb[0], ou, add2(out, dup(c.w[0] * zr[8])));
        }
#pragma unroll
        for (int d = 1; d < Q; d += 2) {
            const int k = cls_of(d);
            const float2 hd = h[d], ho = h[d + 1];
            const float2 cu = dot2(d, tux, tuy, tuz, mone);
            const float2 wc = mul2(nWQ[k], cu);
            float2 X = fma2(half, add2(hd, ho), PQ[k]);
            X = fma2(mul2(half, wc), cu, X);
            const float2 A = fma2(cp_hi, X, mul2(ncp_lo, X));
            const float2 Y = fma2(half, fma2(mone, ho, hd), wc);
            float2 od, oo;
            if (over) {
                // hd - B and ho + B without forming them (see g_pair2)
                const float2 t2 = add2(wc, wc);  // -2 WQ cu
                od = fma2(cm_lo, Y, fma2(mone, A, fma2(mone, t2, ho)));
                oo = fma2(neg2(cm_lo), Y, fma2(mone, A, add2(hd, t2)));
            } else {
                const float2 B = fma2(cm_hi, Y, mul2(neg2(cm_lo), Y));
                od = fma2(mone, add2(A, B), hd);
                oo = fma2(mone, A, add2(ho, B));
            }
            put(a.pp.hb[d], o, od);
            put(a.pp.hb[d + 1], o, oo);
            if (top) {
                const float2 up = dup(c.w[k] * zr[8]);
                put(a.pp.hb[d], ou, add2(od, up));
                put(a.pp.hb[d + 1], ou, add2(oo, up));
            }
        }
    }
}

int lbm_pair_slots(int nx, int ny) {
    const int pairs = nx / 2 * ny;
    return (pairs + kPairThreads - 1) / kPairThreads * (kPairThreads / 16);
}

// FP32, or FP16 f with FP16 or FP32 g; rows of whole pairs, 32-bit byte
// offsets of the 4-byte arrays, and NZ + 1 blocks along y where plane 0 goes
// with the pairs
bool lbm_pair_usable(int nx, int nz, long long n, int prec) {
    return (prec == 1 || prec == 2 || prec == 4) && nx % 2 == 0 && nz < 65535 && n < (1LL << 30);
}

// Up to so many blocks of pairs plane 0 goes with them: 64 x 64 x 33 in FP16
// (512 blocks) 30.7 us a step with a launch of its own, 25.6 without, 100 x
// 100 x 50 (2,000) 79.7 and 72.9; with many blocks the launch is nothing and the
// kernel without the extra branch is the faster one: 256 x 256 x 129 (32,768)
// 498 and 535.  In FP32 the branch costs nothing (122 x 122 x 101 160.6 us a
// step with it, 164.9 without; 256 x 256 x 129 639.5 and 642.2): always merged.
constexpr long long kMergeBlocks = 5000;

template <typename T>
static cudaError_t pair_launch(const LbmArgs &la, const StepConst &c, bool macros, cudaStream_t s) {
    const StepArgs<T, float> a = make_step_args<T, float>(la, c);
    const KConst<float> k = make_kconst<float>(c);
    const int pairs = c.nx / 2 * c.ny, nb = (pairs + kPairThreads - 1) / kPairThreads;
    if (std::is_same<T, float>::value || nb * (long long)(c.nz - 1) <= kMergeBlocks) {
        const dim3 grid(nb, c.nz + 1);
        if (macros) step_launch(lbm_pair_kernel<T, true, StepArgs<T, float>>, grid, kPairThreads, 0, s, a, k);
        else step_launch(lbm_pair_kernel<T, false, StepArgs<T, float>>, grid, kPairThreads, 0, s, a, k);
        return cudaGetLastError();
    }
    if constexpr (!std::is_same<T, float>::value) {
        PairArgs<T> p;
        p.pp = a.pp;
        p.phip = a.phip;
        p.ez00 = a.ez00;
        p.qout = a.qout;
        p.rout = a.rout;
        p.uout = a.uout;
        p.vout = a.vout;
        p.wout = a.wout;
        p.zref = a.zref;
        p.psum = a.psum;
        const dim3 grid(nb, c.nz - 1);
        if (macros) {
            step_launch(lbm_plane0_kernel<T, true>, 2 * nb, kPairThreads, 0, s, a, k);
            step_launch(lbm_pair_kernel<T, true, PairArgs<T>>, grid, kPairThreads, 0, s, p, k);
        } else {
            step_launch(lbm_plane0_kernel<T, false>, 2 * nb, kPairThreads, 0, s, a, k);
            step_launch(lbm_pair_kernel<T, false, PairArgs<T>>, grid, kPairThreads, 0, s, p, k);
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_lbm_pair(int prec, const LbmArgs &la, const StepConst &c, bool macros,
                            cudaStream_t s) {
    if (prec == 1) return pair_launch<float>(la, c, macros, s);
    return prec == 2 ? pair_launch<__half>(la, c, macros, s) : pair_launch<Mix16>(la, c, macros, s);
}

}  // namespace ehd
