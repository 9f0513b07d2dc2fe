// dft.cu -- the Poisson transforms along x and y for widths without
// compile-time FFT passes, as folded matrix products, and the z solve for any
// NZ.
//
// A transform of length n against a table of its cosines and sines is a
// matrix product.  Folding the input about its middle leaves half of it:
// with s_a = v_a + v_{n-a} and d_a = v_a - v_{n-a}, a = 0..n/2 (s alone for
// a = 0 and a = n/2),
//   sum_a v_a exp(-+ 2 pi i a b / n) = sum_a s_a C_ab -+ i sum_a d_a S_ab,
// and the outputs b and n - b share both sums.  For even n = 2 h a second
// folding halves it again: C_{a,h-b} = (-1)^a C_ab and S_{a,h-b} =
// -(-1)^a S_ab, so that the sums over even and over odd a, kept apart, give b
// and h - b.  Every pass below is the same product, over the values of a, of
// pairs (s, d) with pairs (C, S), two multiply-adds at a time (one packed
// FP32x2 instruction in FP32):
//   x forward   real rows: pair (s, d) of a row, out = (sum s C, -sum d S)
//   y           complex columns: pairs (s.x, d.x) and (s.y, d.y)
//   x inverse   half spectrum: the bin itself is the pair (re, im), scaled by
//               2 for the bins that stand for two;
//               phi_a = sum re C - sum im S, phi_{n-a} = sum re C + sum im S
// That is n / 2 (even n: n / 4) multiply-adds of pairs per row point and
// pass.  Run-time radix passes through shared memory do fewer, but spend their
// time on index arithmetic, bank conflicts and serial chains (prime factors
// above all: 122 = 2 x 61).
//
// Tiles: 32 rows (x) or 32 columns (y) per block of 128 threads and 16 (8)
// times TN outputs, TN chosen for the least padding (dft_tile); 16 values of a
// at a time in two shared-memory stages, the next stage's global loads in
// flight during the products.  A thread holds 4 rows x TN outputs (2 complex
// columns x TN), which keeps shared-memory reads below the multiply-adds'
// time; small blocks, because 122 x 122 x 101 has 12,078 rows for 148
// multiprocessors.
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace ehd {

namespace {

constexpr int kKC = 16;  // table rows per stage

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}

template <typename R2>
__device__ __forceinline__ R2 zero2() {
    R2 z;
    z.x = 0;
    z.y = 0;
    return z;
}

// four consecutive pairs from shared memory, 16-byte aligned
__device__ __forceinline__ void ld4(float2 (&v)[4], const float2 *p) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 2);
    v[0] = make_float2(a.x, a.y);
    v[1] = make_float2(a.z, a.w);
    v[2] = make_float2(b.x, b.y);
    v[3] = make_float2(b.z, b.w);
}
__device__ __forceinline__ void ld4(double2 (&v)[4], const double2 *p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = p[i];
}

constexpr int kM = 32;          // rows (x) or columns (y) of a block
constexpr int kXPad = 2;        // of a staged row of pairs, 16-byte aligned
constexpr int kXU = 16, kYU = 8;  // outputs of a block per TN, x and y
constexpr int kThreads = 128;

template <typename R, int TN>
constexpr size_t rows_smem() {
    return sizeof(typename Cplx<R>::T) * 2 * kKC * (size_t)(kM + kXPad + kXU * TN);
}
template <typename R, int TN>
constexpr size_t cols_smem() {
    return sizeof(typename Cplx<R>::T) * 2 * kKC * (size_t)(2 * kM + kYU * TN);
}
// resident blocks the compiler should leave registers for
template <typename R>
constexpr int min_blocks() { return sizeof(R) == 8 ? 2 : 3; }

// The values of a in the order of the table's rows: all of them (odd n), or
// the even ones, then the odd ones, each padded to whole stages.  The inverse passes
// (INV) take each of these runs from its end: their inputs are the modes of phi',
// which fall off as a^-2, and a sum that adds the large ones last rounds at their
// size once or twice instead of n / 4 times (E_x of a noisy charge in FP32, distance
// from a 64-bit solve: 160 x 160 x 33 5.6e-6 the other way, 1.8e-6 so, radix passes
// 2.7e-6; 360 x 90 x 20 9.2e-6, 2.1e-6 and 3.3e-6).
template <bool EVEN, bool INV>
struct Order {
    int n, te, ts;  // length, stages of the even values, all stages
    __device__ __forceinline__ explicit Order(int n_) : n(n_) {
        const int h = n / 2;
        te = EVEN ? (h / 2 + 1 + kKC - 1) / kKC : (h + 1 + kKC - 1) / kKC;
        ts = EVEN ? te + ((h + 1) / 2 + kKC - 1) / kKC : te;
    }
    // table row of row r of stage t, its value, and whether it exists
    __device__ __forceinline__ int row(int t, int r) const {
        if (INV) {
            t = t < te ? te - 1 - t : te + ts - 1 - t;
            r = kKC - 1 - r;
        }
        return kKC * t + r;
    }
    __device__ __forceinline__ int at(int t, int r) const {
        const int i = row(t, r);
        if (!EVEN) return i;
        return i < kKC * te ? 2 * i : 2 * (i - kKC * te) + 1;
    }
    __device__ __forceinline__ bool in(int a) const { return 2 * a <= n; }
    __device__ __forceinline__ bool pair(int a) const { return a > 0 && 2 * a < n; }
};

// One stage of the x products: thread (tk, tr) accumulates rows 4 tr + i and
// outputs tk + 16 j.
template <int TN, typename R2>
__device__ __forceinline__ void rows_stage(const R2 *As, const R2 *Bs, int tk, int tr,
                                           R2 (&acc)[4][TN]) {
#pragma unroll
    for (int x = 0; x < kKC; ++x) {
        R2 a[4], b[TN];
        ld4(a, As + x * (kM + kXPad) + 4 * tr);
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = Bs[x * kXU * TN + tk + kXU * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
    }
}
// One stage of the y products: thread (tm, tn) accumulates columns tm + 16 i
// and outputs TN tn + j, ax the pairs of real parts, ay of imaginary parts.
template <int TN, typename R2>
__device__ __forceinline__ void cols_stage(const R2 *A1, const R2 *A2, const R2 *Bs, int tm, int tn,
                                           R2 (&ax)[2][TN], R2 (&ay)[2][TN]) {
#pragma unroll
    for (int y = 0; y < kKC; ++y) {
        R2 a[2], c[2], b[TN];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            a[i] = A1[y * kM + tm + 16 * i];
            c[i] = A2[y * kM + tm + 16 * i];
        }
        if constexpr (TN == 4) {
            ld4(b, Bs + y * kYU * TN + TN * tn);
        } else {
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[y * kYU * TN + TN * tn + j];
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                ax[i][j] = fma2(a[i], b[j], ax[i][j]);
                ay[i][j] = fma2(c[i], b[j], ay[i][j]);
            }
    }
}

// One stage of the table: its 16 rows, BN columns from n0
template <int BN, typename R2>
struct TableStage {
    static constexpr int kV = kKC * BN / kThreads;
    R2 v[kV];
    template <typename O>
    __device__ __forceinline__ void load(const R2 *__restrict__ tab, int tp, const O &ord, int t,
                                         int n0) {
#pragma unroll
        for (int i = 0; i < kV; ++i) {
            const int e = threadIdx.x + kThreads * i, x = e / BN, k = e - x * BN;
            v[i] = tab[(size_t)ord.row(t, x) * tp + n0 + k];
        }
    }
    __device__ __forceinline__ void store(R2 *Bs) const {
#pragma unroll
        for (int i = 0; i < kV; ++i) Bs[threadIdx.x + kThreads * i] = v[i];
    }
};

template <int A, int B, typename R2>
__device__ __forceinline__ void clear(R2 (&v)[A][B]) {
#pragma unroll
    for (int i = 0; i < A; ++i)
#pragma unroll
        for (int j = 0; j < B; ++j) v[i][j] = zero2<R2>();
}
// the sums at h - b from those over even and over odd a at b
template <typename R2>
__device__ __forceinline__ R2 mirrored(R2 e, R2 o) {
    R2 r;
    r.x = e.x - o.x;
    r.y = o.y - e.y;
    return r;
}
template <typename R2>
__device__ __forceinline__ R2 add2(R2 a, R2 b) {
    a.x += b.x;
    a.y += b.y;
    return a;
}

}  // namespace

// K1: s' = -(q - q_m)/eps on the planes z = 1..NZ-2 (odd_extension's interior
// rows, poisson.cu:96-106), transformed along x; half spectrum out, FP64 row
// sums from the blocks of the first outputs.  The interior rows of all planes
// are one run of rows.
template <typename R, int TN, bool EVEN>
__global__ void __launch_bounds__(kThreads, min_blocks<R>())
dft_rows_fwd(const R *__restrict__ q, typename Cplx<R>::T *__restrict__ spec,
             double *__restrict__ rowsum, const typename Cplx<R>::T *__restrict__ tab, int tp,
             const double *__restrict__ qmean, int nx, int ny, int rows, int pitch,
             double eps, const PoissonPtrs *__restrict__ grp) {
    step_enter();
    if (grp) {  // one instance of a group launch per blockIdx.z
        const PoissonPtrs &gp = grp[blockIdx.z];
        q = (const R *)gp.q;
        spec = (typename Cplx<R>::T *)gp.spec;
        rowsum = gp.rowsum;
        qmean = gp.qmean;
    }
    using R2 = typename Cplx<R>::T;
    constexpr int BN = kXU * TN, SA = kKC * (kM + kXPad), SB = kKC * BN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2 *As = reinterpret_cast<R2 *>(smem_raw);  // [2][kKC][kM + kXPad]
    R2 *Bs = As + 2 * SA;                       // [2][kKC][BN]
    const int tid = threadIdx.x;
    const int r0 = blockIdx.x * kM, n0 = blockIdx.y * BN;
    const bool sums = blockIdx.y == 0;
    const R ieps = (R)(1.0 / eps);
    const Order<EVEN, false> ord(nx);
    q += (size_t)nx * ny;  // plane 1
    // staging: table row tid % 16 of the rows tid / 16 + 8 i
    const int xs = tid & 15, rs = tid >> 4;
    R qm[4];
    double sum[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + rs + 8 * i;
        qm[i] = r < rows ? (R)qmean[2 * (r / ny + 1) + 1] : (R)0;
        sum[i] = 0.0;
    }
    R lo[4], hi[4];
    TableStage<BN, R2> tb;
    auto load = [&](int t) {
        const int x = ord.at(t, xs);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + rs + 8 * i;
            const R *row = q + (size_t)nx * r;
            const bool in = r < rows && ord.in(x);
            // (a = 0 and a = n / 2 stand alone: their partner counts as q_m)
            lo[i] = in ? row[x] : qm[i];
            hi[i] = in && ord.pair(x) ? row[nx - x] : qm[i];
        }
        tb.load(tab, tp, ord, t, n0);
    };
    auto store = [&](int s, int t) {
        R2 *a = As + s * SA;
        const bool pair = ord.pair(ord.at(t, xs));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const R u = -(lo[i] - qm[i]) * ieps, v = -(hi[i] - qm[i]) * ieps;
            if (sums) sum[i] += ((double)lo[i] - (double)qm[i]) + ((double)hi[i] - (double)qm[i]);
            R2 p;
            p.x = u + v;
            p.y = pair ? u - v : (R)0;
            a[xs * (kM + kXPad) + rs + 8 * i] = p;
        }
        tb.store(Bs + s * SB);
    };
    const int tk = tid & 15, tr = tid >> 4;
    R2 acc[4][TN], odd[4][EVEN ? TN : 1];
    clear(acc);
    clear(odd);
    load(0);
    store(0, 0);
    __syncthreads();
    for (int t = 0; t < ord.te; ++t) {
        const int s = t & 1;
        if (t + 1 < ord.ts) load(t + 1);
        rows_stage<TN>(As + s * SA, Bs + s * SB, tk, tr, acc);
        if (t + 1 < ord.ts) store(s ^ 1, t + 1);
        __syncthreads();
    }
    if constexpr (EVEN)
        for (int t = ord.te; t < ord.ts; ++t) {
            const int s = t & 1;
            if (t + 1 < ord.ts) load(t + 1);
            rows_stage<TN>(As + s * SA, Bs + s * SB, tk, tr, odd);
            if (t + 1 < ord.ts) store(s ^ 1, t + 1);
            __syncthreads();
        }
    const int h = nx / 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + 4 * tr + i;
        if (r >= rows) continue;
        R2 *o = spec + (size_t)pitch * r;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int k = n0 + tk + kXU * j;
            R2 v = acc[i][j];
            if constexpr (EVEN) {
                if (2 * k < h) {
                    R2 w = mirrored(acc[i][j], odd[i][j]);
                    w.y = -w.y;
                    o[h - k] = w;
                }
                v = add2(acc[i][j], odd[i][j]);
            }
            v.y = -v.y;
            if (EVEN ? 2 * k <= h : k <= h) o[k] = v;
        }
    }
    if (sums) {  // FP64 row sums: the 16 threads of a row, fixed order
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
            const int r = r0 + rs + 8 * i;
            if (xs == 0 && r < rows) rowsum[r] = -sum[i] / eps;
        }
    }
}

// K4: phi' = Re of the inverse transform along x, over NX NY (odd_extract,
// poisson.cu:154-167, for the interior planes).  The imaginary parts of the
// bins 0 and NX / 2, which a real row ignores, meet the zeros of S.
template <typename R, int TN, bool EVEN>
__global__ void __launch_bounds__(kThreads, min_blocks<R>())
dft_rows_inv(const typename Cplx<R>::T *__restrict__ spec, R *__restrict__ phip,
             const typename Cplx<R>::T *__restrict__ tab, int tp, int nx, int ny, int rows,
             int pitch, const PoissonPtrs *__restrict__ grp) {
    step_enter();
    if (grp) {  // one instance of a group launch per blockIdx.z
        const PoissonPtrs &gp = grp[blockIdx.z];
        spec = (const typename Cplx<R>::T *)gp.spec;
        phip = (R *)gp.phip;
    }
    using R2 = typename Cplx<R>::T;
    constexpr int BN = kXU * TN, SA = kKC * (kM + kXPad), SB = kKC * BN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2 *As = reinterpret_cast<R2 *>(smem_raw);
    R2 *Bs = As + 2 * SA;
    const int tid = threadIdx.x;
    const int r0 = blockIdx.x * kM, n0 = blockIdx.y * BN;
    const Order<EVEN, true> ord(nx);
    const int ks = tid & 15, rs = tid >> 4;
    R2 v[4];
    TableStage<BN, R2> tb;
    auto load = [&](int t) {
        const int k = ord.at(t, ks);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + rs + 8 * i;
            v[i] = r < rows && ord.in(k) ? spec[(size_t)pitch * r + k] : zero2<R2>();
        }
        tb.load(tab, tp, ord, t, n0);
    };
    auto store = [&](int s, int t) {
        R2 *a = As + s * SA;
        const R two = ord.pair(ord.at(t, ks)) ? (R)2 : (R)1;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i].x *= two;
            v[i].y *= two;
            a[ks * (kM + kXPad) + rs + 8 * i] = v[i];
        }
        tb.store(Bs + s * SB);
    };
    const int tk = tid & 15, tr = tid >> 4;
    R2 acc[4][TN], odd[4][EVEN ? TN : 1];
    clear(acc);
    clear(odd);
    load(0);
    store(0, 0);
    __syncthreads();
    for (int t = 0; t < ord.te; ++t) {
        const int s = t & 1;
        if (t + 1 < ord.ts) load(t + 1);
        rows_stage<TN>(As + s * SA, Bs + s * SB, tk, tr, acc);
        if (t + 1 < ord.ts) store(s ^ 1, t + 1);
        __syncthreads();
    }
    if constexpr (EVEN)
        for (int t = ord.te; t < ord.ts; ++t) {
            const int s = t & 1;
            if (t + 1 < ord.ts) load(t + 1);
            rows_stage<TN>(As + s * SA, Bs + s * SB, tk, tr, odd);
            if (t + 1 < ord.ts) store(s ^ 1, t + 1);
            __syncthreads();
        }
    const R norm = (R)(1.0 / ((double)nx * (double)ny));
    const int h = nx / 2;
    phip += (size_t)nx * ny;  // plane 1
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + 4 * tr + i;
        if (r >= rows) continue;
        R *row = phip + (size_t)nx * r;
        auto emit = [&](int x, R2 s) {
            row[x] = (s.x - s.y) * norm;
            if (ord.pair(x)) row[nx - x] = (s.x + s.y) * norm;
        };
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int x = n0 + tk + kXU * j;
            if constexpr (EVEN) {
                if (2 * x <= h) emit(x, add2(acc[i][j], odd[i][j]));
                if (2 * x < h) emit(h - x, mirrored(acc[i][j], odd[i][j]));
            } else {
                if (x <= h) emit(x, acc[i][j]);
            }
        }
    }
}

// K2: transform along y of the kx columns of plane blockIdx.y, from `in` to
// `out` ([z-1][ky][kx], the blocks of different outputs read the same columns,
// so not in place); S = -1 forward (spec to spec2), +1 inverse (back).  The
// forward pass also reduces the FP64 plane sum.
template <typename R, int S, int TN, bool EVEN>
__global__ void __launch_bounds__(kThreads, min_blocks<R>())
dft_cols(const typename Cplx<R>::T *__restrict__ in, typename Cplx<R>::T *__restrict__ out,
         const typename Cplx<R>::T *__restrict__ tab, int tp, int ny, int nxh, int pitch, int mtiles,
         const double *__restrict__ rowsum, double *__restrict__ planesum,
         const PoissonPtrs *__restrict__ grp) {
    step_enter();
    if (grp) {  // one instance of a group launch per blockIdx.z
        const PoissonPtrs &gp = grp[blockIdx.z];
        rowsum = gp.rowsum;
        planesum = gp.planesum;
        in = (const typename Cplx<R>::T *)(S < 0 ? gp.spec : gp.spec2);
        out = (typename Cplx<R>::T *)(S < 0 ? gp.spec2 : gp.spec);
    }
    using R2 = typename Cplx<R>::T;
    constexpr int BN = kYU * TN, SA = kKC * kM, SB = kKC * BN;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2 *A1 = reinterpret_cast<R2 *>(smem_raw);  // [2][kKC][kM] pairs (s.x, d.x)
    R2 *A2 = A1 + 2 * SA;                       // pairs (s.y, d.y)
    R2 *Bs = A2 + 2 * SA;                       // [2][kKC][BN]
    const int tid = threadIdx.x;
    const int m0 = (blockIdx.x % mtiles) * kM, n0 = (blockIdx.x / mtiles) * BN;
    const Order<EVEN, (S > 0)> ord(ny);
    const size_t plane = (size_t)blockIdx.y * ny * pitch;
    in += plane;
    out += plane;
    // staging: column tid % 32 of the table rows tid / 32 + 4 i
    const int cs = tid & 31, ys = tid >> 5;
    const bool cin = m0 + cs < nxh;
    R2 lo[4], hi[4];
    TableStage<BN, R2> tb;
    auto load = [&](int t) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int y = ord.at(t, ys + 4 * i);
            const bool ok = cin && ord.in(y);
            lo[i] = ok ? in[(size_t)pitch * y + m0 + cs] : zero2<R2>();
            hi[i] = ok && ord.pair(y) ? in[(size_t)pitch * (ny - y) + m0 + cs] : zero2<R2>();
        }
        tb.load(tab, tp, ord, t, n0);
    };
    auto store = [&](int s, int t) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool pair = ord.pair(ord.at(t, ys + 4 * i));
            R2 p, w;
            p.x = lo[i].x + hi[i].x;
            p.y = pair ? lo[i].x - hi[i].x : (R)0;
            w.x = lo[i].y + hi[i].y;
            w.y = pair ? lo[i].y - hi[i].y : (R)0;
            A1[s * SA + (ys + 4 * i) * kM + cs] = p;
            A2[s * SA + (ys + 4 * i) * kM + cs] = w;
        }
        tb.store(Bs + s * SB);
    };
    const int tm = tid & 15, tn = tid >> 4;
    R2 ax[2][TN], ay[2][TN], ox[2][EVEN ? TN : 1], oy[2][EVEN ? TN : 1];
    clear(ax);
    clear(ay);
    clear(ox);
    clear(oy);
    load(0);
    store(0, 0);
    if (S < 0 && blockIdx.x == 0 && tid < 32) {  // fixed order, one warp
        double sum = 0.0;
        for (int y = tid; y < ny; y += 32) sum += rowsum[(size_t)blockIdx.y * ny + y];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (tid == 0) planesum[blockIdx.y + 1] = sum;
    }
    __syncthreads();
    for (int t = 0; t < ord.te; ++t) {
        const int s = t & 1;
        if (t + 1 < ord.ts) load(t + 1);
        cols_stage<TN>(A1 + s * SA, A2 + s * SA, Bs + s * SB, tm, tn, ax, ay);
        if (t + 1 < ord.ts) store(s ^ 1, t + 1);
        __syncthreads();
    }
    if constexpr (EVEN)
        for (int t = ord.te; t < ord.ts; ++t) {
            const int s = t & 1;
            if (t + 1 < ord.ts) load(t + 1);
            cols_stage<TN>(A1 + s * SA, A2 + s * SA, Bs + s * SB, tm, tn, ox, oy);
            if (t + 1 < ord.ts) store(s ^ 1, t + 1);
            __syncthreads();
        }
    const int h = ny / 2;
    // A = (x.x, y.x), B = (x.y, y.y); out_ky = A + S i B, out_{ny-ky} = A - S i B
    auto emit = [&](int ky, int k, R2 x, R2 y) {
        const R bx = S > 0 ? -y.y : y.y, by = S > 0 ? x.y : -x.y;
        R2 o;
        o.x = x.x + bx;
        o.y = y.x + by;
        out[(size_t)pitch * ky + k] = o;
        if (ord.pair(ky)) {
            o.x = x.x - bx;
            o.y = y.x - by;
            out[(size_t)pitch * (ny - ky) + k] = o;
        }
    };
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int ky = n0 + TN * tn + j;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = m0 + tm + 16 * i;
            if (k >= nxh) continue;
            if constexpr (EVEN) {
                if (2 * ky <= h) emit(ky, k, add2(ax[i][j], ox[i][j]), add2(ay[i][j], oy[i][j]));
                if (2 * ky < h)
                    emit(h - ky, k, mirrored(ax[i][j], ox[i][j]), mirrored(ay[i][j], oy[i][j]));
            } else {
                if (ky <= h) emit(ky, k, ax[i][j], ay[i][j]);
            }
        }
    }
}

namespace {
// The mean mode of a tall column, x_i = -((n + 1 - i) A_i + i B_i) / (n + 1) / nxy
// with A_i = sum_{j < i} j rhs_j and B_i = sum_{j >= i} (n + 1 - j) rhs_j (i, j = 1..n),
// by the block of 128 threads: a run of planes each, the sums before and after
// it from one scan.  The n terms of every plane, each a dependent FP64 step, would
// be the solve's longest chain: 4 x 4 x 1729 in FP32 287 us a step with them,
// 208 so; up to kTallMean planes they hide behind the modes.
constexpr int kTallMean = 512;
__device__ __noinline__ void tall_mean(const double *mrhs, double *mphi, double *phi00, int nz,
                                       double nxy, double voltage) {
    // (not static shared memory: the columns of the other blocks would move off
    // their 128-byte lines)
    double *wa = mphi + nz, *wb = wa + 4;
    const int n = nz - 2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = (n + 127) / 128;
    const int i0 = 1 + tid * c < n + 1 ? 1 + tid * c : n + 1, i1 = i0 + c < n + 1 ? i0 + c : n + 1;
    double a = 0.0, b = 0.0;
    for (int i = i0; i < i1; ++i) {
        a += (double)i * mrhs[i - 1];
        b += (double)(n + 1 - i) * mrhs[i - 1];
    }
    // sums of a over the threads before, of b over those after
    double sa = a, sb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double ta = __shfl_up_sync(0xffffffffu, sa, o), tb = __shfl_down_sync(0xffffffffu, sb, o);
        if (lane >= o) sa += ta;
        if (lane + o < 32) sb += tb;
    }
    if (lane == 31) wa[warp] = sa;
    if (lane == 0) wb[warp] = sb;
    double A = __shfl_up_sync(0xffffffffu, sa, 1), B = __shfl_down_sync(0xffffffffu, sb, 1);
    if (lane == 0) A = 0.0;
    if (lane == 31) B = 0.0;
    __syncthreads();
    for (int w = 0; w < 4; ++w) {
        if (w < warp) A += wa[w];
        if (w > warp) B += wb[w];
    }
    for (int i = i0; i < i1; ++i) {
        mphi[i] = (double)(n + 1 - i) * A;
        A += (double)i * mrhs[i - 1];
    }
    for (int i = i1 - 1; i >= i0; --i) {
        B += (double)(n + 1 - i) * mrhs[i - 1];
        const double x = -(mphi[i] + (double)i * B) / (double)(n + 1) / nxy;
        mphi[i] = x;
        phi00[i] = x;
    }
    if (tid == 0) {
        mphi[0] = phi00[0] = voltage;
        mphi[nz - 1] = phi00[nz - 1] = 0.0;
    }
}
}  // namespace

// K3 for any NZ whose columns fit in shared memory: the tridiagonal system of
// poisson_zsolve per mode (kx, ky), phi(z-1) - beta phi(z) + phi(z+1) =
// dz^2 s(z), beta = 2 + (kx^2 + ky^2) dz^2, phi = 0 on the electrodes, solved
// from both ends at once, in place.  One lane eliminates the upper half of the
// planes downwards, the lane 16 apart the lower half upwards, with the same
// FP64 pivots (the matrix is symmetric Toeplitz; the first (NZ - 2) / 2 rows
// of the context's table), they meet in the middle and each substitutes back
// over its half.  Arithmetic in FP64, the columns in the compute type.
//
// The chain of about NZ dependent FP64 steps is what the kernel waits for, so
// it runs on 2 modes x 16 lanes a warp over mb = 16 or 32 modes a block: many
// small blocks, whose columns arrive (cp.async, every load in flight at once)
// and leave while others' chains run.  Block 0 solves the (0,0)
// mode in closed form beside the others (see poisson_zdst); the (0,0) mode of
// the fluctuation is 0.  The bound of two blocks a multiprocessor leaves the
// compiler registers for whole batches of loads (FP64 90 instead of 72: 16 x 16 x
// 865 194 -> 180 us a step).
template <typename R>
__global__ void __launch_bounds__(128, 2)
poisson_zmeet(typename Cplx<R>::T *__restrict__ spec, const double *__restrict__ cpt,
              const double *__restrict__ planesum, const double *__restrict__ qmean,
              double *__restrict__ phi00, double *__restrict__ ez00, int nx, int ny, int nz,
              int nxh, int pitch, int mb, double dz, double eps, double voltage, double kx0,
              double ky0, const PoissonPtrs *__restrict__ grp) {
    step_enter();
    if (grp) {  // one instance of a group launch per blockIdx.z
        const PoissonPtrs &gp = grp[blockIdx.z];
        spec = (typename Cplx<R>::T *)gp.spec;
        planesum = gp.planesum;
        qmean = gp.qmean;
        phi00 = gp.phi00;
        ez00 = gp.ez00;
    }
    using R2 = typename Cplx<R>::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = nz - 2;
    const double dz2 = dz * dz;
    if (blockIdx.x == 0) {
        double *mrhs = reinterpret_cast<double *>(smem_raw), *mphi = mrhs + n;
        const double nxy = (double)nx * (double)ny;
        for (int i = tid; i < n; i += 128) {
            double d = planesum[i + 1] + nxy * (-(double)(R)qmean[2 * (i + 1) + 1] / eps);
            if (i == 0) d += -voltage / dz2 * nxy;  // poisson.cu:97
            mrhs[i] = d * dz2;
        }
        __syncthreads();
        if (nz > kTallMean) {
            tall_mean(mrhs, mphi, phi00, nz, nxy, voltage);
        } else for (int i = tid; i < nz; i += 128) {
            double x = 0.0;
            if (i == 0) {
                x = voltage;
            } else if (i < nz - 1) {
                for (int jz = 1; jz <= n; ++jz) {
                    const int l = i < jz ? i : jz, h = i < jz ? jz : i;
                    x -= (double)(l * (n + 1 - h)) * mrhs[jz - 1];
                }
                x = x / (double)(n + 1) / nxy;
            }
            mphi[i] = x;
            phi00[i] = x;
        }
        __syncthreads();
        for (int z = tid; z < nz; z += 128) {
            const int zc = z < 1 ? 1 : (z > nz - 2 ? nz - 2 : z);
            ez00[z] = 0.5 * (mphi[zc - 1] - mphi[zc + 1]) / dz;
        }
        return;
    }
    R2 *col = reinterpret_cast<R2 *>(smem_raw);  // [n][mb]
    const int modes = nxh * ny;
    const int m0 = ((int)blockIdx.x - 1) * mb;
    const size_t plane = (size_t)ny * pitch;
    // thread tid moves mode tid % mb of the planes tid / mb + (128 / mb) i
    const int ct = tid % mb, zt = tid / mb, zs = 128 / mb;
    const bool cin = m0 + ct < modes;
    const int cky = cin ? (m0 + ct) / nxh : 0;
    R2 *g = spec + (size_t)cky * pitch + (cin ? m0 + ct - cky * nxh : 0);
    if (cin)
        for (int z = zt; z < n; z += zs) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(col + z * mb + ct);
            if (sizeof(R) == 4)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst),
                             "l"(g + (size_t)z * plane)
                             : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst),
                             "l"(g + (size_t)z * plane)
                             : "memory");
        }
    // the block's pivots into L2, by 32-byte pieces: where the state is larger
    // than L2 they are gone from one step to the next, and the chain would wait
    // for each batch of them (16 x 16 x 865 in FP64 203 -> 194 us a step)
    {
        const int per = mb / 4 + 1;
        for (int i = tid; i < (n / 2) * per; i += 128) {
            const int k = i / per, m = m0 + 4 * (i - k * per);
            asm volatile("prefetch.global.L2 [%0];" ::"l"(
                cpt + (size_t)k * modes + (m < modes ? m : modes - 1)));
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (16 * warp < mb) {
        constexpr int kB = 8;
        const int c = 16 * warp + (lane & 15), side = lane >> 4;
        const int mode = m0 + c < modes ? m0 + c : modes - 1;
        R2 *x = col + c;
        const double *pc = cpt + mode;
        const int m = n / 2;  // planes of each half
        auto at = [&](int k) { return (side ? n - 1 - k : k) * mb; };
        // the (0,0) mode takes part (its system is regular) and is stored as 0
        const R keep = m0 + c == 0 ? (R)0 : (R)1;
        double dr = 0.0, di = 0.0, cl = 0.0;
#pragma unroll 1
        for (int k0 = 0; k0 < m; k0 += kB) {
            R2 sv[kB];
            double cv[kB];
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int k = k0 + u < m ? k0 + u : m - 1;
                sv[u] = x[at(k)];
                cv[u] = __ldg(pc + (size_t)k * modes);
            }
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                if (k0 + u < m) {
                    dr = ((double)sv[u].x * dz2 - dr) * cv[u];
                    di = ((double)sv[u].y * dz2 - di) * cv[u];
                    R2 o;
                    o.x = (R)dr;
                    o.y = (R)di;
                    x[at(k0 + u)] = o;
                    cl = cv[u];
                }
            }
        }
        const double or_ = __shfl_xor_sync(0xffffffffu, dr, 16);
        const double oi = __shfl_xor_sync(0xffffffffu, di, 16);
        double xr, xi;
        int last = m - 1;  // the first plane of the substitution
        if (n & 1) {
            const int ky = mode / nxh, kx = mode - ky * nxh;
            const double wx = kx * kx0, wy = (ky <= ny / 2 ? ky : ky - ny) * ky0;
            const double mu = 1.0 / (-(2.0 + (wx * wx + wy * wy) * dz2) - 2.0 * cl);
            const R2 sm = x[m * mb];
            xr = ((double)sm.x * dz2 - dr - or_) * mu;
            xi = ((double)sm.y * dz2 - di - oi) * mu;
            __syncwarp();
            if (side == 0) {
                R2 o;
                o.x = (R)xr * keep;
                o.y = (R)xi * keep;
                x[m * mb] = o;
            }
        } else {
            // x_{m-1} + c x_m = d, x_m + c x_{m-1} = d of the other side
            const double f = 1.0 / (1.0 - cl * cl);
            xr = (dr - cl * or_) * f;
            xi = (di - cl * oi) * f;
            R2 o;
            o.x = (R)xr * keep;
            o.y = (R)xi * keep;
            x[at(m - 1)] = o;
            last = m - 2;
        }
#pragma unroll 1
        for (int k1 = last; k1 >= 0; k1 -= kB) {
            R2 dv[kB];
            double cv[kB];
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int k = k1 - u >= 0 ? k1 - u : 0;
                dv[u] = x[at(k)];
                cv[u] = __ldg(pc + (size_t)k * modes);
            }
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                if (k1 - u >= 0) {
                    xr = (double)dv[u].x - cv[u] * xr;
                    xi = (double)dv[u].y - cv[u] * xi;
                    R2 o;
                    o.x = (R)xr * keep;
                    o.y = (R)xi * keep;
                    x[at(k1 - u)] = o;
                }
            }
        }
    }
    __syncthreads();
    if (cin)
        for (int z = zt; z < n; z += zs) g[(size_t)z * plane] = col[z * mb + ct];
}

// ---- launchers ----

namespace {
// outputs b that a pass forms (the others share their sums), table rows
int dft_outputs(int n) { return n % 2 == 0 ? n / 4 + 1 : n / 2 + 1; }
int dft_stages(int n) {
    const int h = n / 2;
    auto st = [](int m) { return (m + kKC - 1) / kKC; };
    return n % 2 == 0 ? st(h / 2 + 1) + st((h + 1) / 2) : st(h + 1);
}
// TN for an axis: the least padded outputs, weighed by what a narrower tile
// costs in shared-memory reads per product; FP64 accumulators leave room for 3
int dft_tile(int n, int unit, size_t rsize) {
    const int nb = dft_outputs(n);
    int best = 2;
    double cost = 0.0;
    for (int tn = 2; tn <= (rsize == 8 ? 3 : 5); ++tn) {
        const int w = unit * tn;
        const double c = (double)((nb + w - 1) / w * w) * (1.0 + 0.6 / tn);
        if (tn == 2 || c < cost) {
            cost = c;
            best = tn;
        }
    }
    return best;
}
}  // namespace

int dft_table_pitch(int n, bool y, size_t rsize) {
    const int w = (y ? kYU : kXU) * dft_tile(n, y ? kYU : kXU, rsize);
    return (dft_outputs(n) + w - 1) / w * w;
}
size_t dft_table_elems(int n, bool y, size_t rsize) {
    return (size_t)kKC * dft_stages(n) * dft_table_pitch(n, y, rsize);
}
void dft_table(int n, bool y, size_t rsize, double *t) {
    const int tp = dft_table_pitch(n, y, rsize), h = n / 2;
    const int te = n % 2 == 0 ? (h / 2 + 1 + kKC - 1) / kKC : dft_stages(n);
    std::vector<double> cs(n), sn(n);
    for (int m = 0; m < n; ++m) {
        cs[m] = std::cos(2.0 * M_PI * (double)m / (double)n);
        // exact zeros of the sine
        sn[m] = m == 0 || 2 * m == n ? 0.0 : std::sin(2.0 * M_PI * (double)m / (double)n);
    }
    for (int r = 0; r < kKC * dft_stages(n); ++r) {
        int a = r;
        if (n % 2 == 0) a = r < kKC * te ? 2 * r : 2 * (r - kKC * te) + 1;
        for (int b = 0; b < tp; ++b) {
            const bool in = a <= h && b < dft_outputs(n);
            const int m = (int)((long long)a * b % n);
            t[2 * ((size_t)r * tp + b)] = in ? cs[m] : 0.0;
            t[2 * ((size_t)r * tp + b) + 1] = in ? sn[m] : 0.0;
        }
    }
}

// Folded products or run-time radix passes (FFT in shared memory): whichever
// an estimate in picoseconds per point and pass says is faster, fitted to
// Poisson solves on a B200.  The products cost a fixed part (staging) and a
// part per padded product, w = table rows x outputs / n; a radix pass about
// the same for every factor up to 5, a direct pass of prime p in proportion
// to p.  Solves with the same z solve, products / radix passes, us:
// FP32 160 x 160 x 65 (w = 29) 76 / 107, 360 x 360 x 33 (w = 51) 175 / 239,
// 400 x 400 x 33 (w = 72) 258 / 254, 768 x 48 x 33 (x only, w = 125) 104 / 82;
// FP64 160 x 160 x 65 152 / 131, 240 x 240 x 33 (w = 34) 158 / 146,
// 400 x 400 x 33 588 / 319.  Large primes are the products' (FP32, with the z
// solve of this file): 122 x 122 x 101 57 / 175, 349 x 183 x 20 88 / 303.
// Short axes come with small grids, where what counts is a kernel's own
// latency: 24 x 24 x 17 28 / 34.
bool dft_usable(int n, bool y, size_t rsize) {
    if (n > kDftMax) return false;
    const double w = (double)dft_table_elems(n, y, rsize) / n;
    const bool f64 = rsize == 8;
    const double products = f64 ? 9.7 + 0.25 * w : 4.0 + 0.118 * w;
    double passes = 0.0;
    int m = n;
    for (int f : {4, 2, 3, 5})
        for (; m % f == 0; m /= f) passes += f64 ? 3.7 : 2.7;
    for (int f = 7; m > 1; f += 2)
        for (; m % f == 0; m /= f) passes += f64 ? 3.7 + 0.5 * f : 2.7 + 0.36 * f;
    return n <= 64 || products < passes;
}

namespace {
// calls f(TN, EVEN) with the axis's tile as compile-time values
template <typename R, typename F>
cudaError_t with_tile(int n, int unit, F f) {
    const int tn = dft_tile(n, unit, sizeof(R));
    auto go = [&](auto even) -> cudaError_t {
        if (tn == 2) return f(std::integral_constant<int, 2>{}, even);
        if (tn == 3) return f(std::integral_constant<int, 3>{}, even);
        if constexpr (sizeof(R) == 4) {
            if (tn == 4) return f(std::integral_constant<int, 4>{}, even);
            return f(std::integral_constant<int, 5>{}, even);
        }
        return cudaErrorInvalidValue;
    };
    return n % 2 == 0 ? go(std::true_type{}) : go(std::false_type{});
}
}  // namespace

template <typename R>
cudaError_t prepare_zmeet() {
    return allow_max_dynamic_smem(poisson_zmeet<R>);
}

template <typename R>
cudaError_t prepare_dft(int nx, int ny) {
    cudaError_t e = with_tile<R>(nx, kXU, [&](auto tn, auto even) {
        cudaError_t r = allow_max_dynamic_smem(dft_rows_fwd<R, decltype(tn)::value, decltype(even)::value>);
        return r == cudaSuccess
                   ? allow_max_dynamic_smem(dft_rows_inv<R, decltype(tn)::value, decltype(even)::value>)
                   : r;
    });
    if (e == cudaSuccess)
        e = with_tile<R>(ny, kYU, [&](auto tn, auto even) {
            cudaError_t r = allow_max_dynamic_smem(dft_cols<R, -1, decltype(tn)::value, decltype(even)::value>);
            return r == cudaSuccess
                       ? allow_max_dynamic_smem(dft_cols<R, 1, decltype(tn)::value, decltype(even)::value>)
                       : r;
        });
    return e == cudaSuccess ? prepare_zmeet<R>() : e;
}

template <typename R>
cudaError_t launch_dft_rows_fwd(const PoissonArgs &a, cudaStream_t s) {
    using R2 = typename Cplx<R>::T;
    const int rows = a.ny * (a.nz - 2), tp = dft_table_pitch(a.nx, false, sizeof(R));
    return with_tile<R>(a.nx, kXU, [&](auto tn, auto even) {
        constexpr int TN = decltype(tn)::value;
        const dim3 grid((rows + kM - 1) / kM, tp / (kXU * TN), a.ngrp);
        auto kern = dft_rows_fwd<R, TN, decltype(even)::value>;
        cudaError_t e = set_smem(kern, rows_smem<R, TN>(), s);
        if (e != cudaSuccess) return e;
        step_launch(kern, grid, kThreads, rows_smem<R, TN>(), s, (const R *)a.q, (R2 *)a.spec,
                    a.rowsum, (const R2 *)a.tabx, tp, a.qmean, a.nx, a.ny, rows, a.pitch, a.eps,
                    a.grp);
        return cudaGetLastError();
    });
}
template <typename R>
cudaError_t launch_dft_rows_inv(const PoissonArgs &a, cudaStream_t s) {
    using R2 = typename Cplx<R>::T;
    const int rows = a.ny * (a.nz - 2), tp = dft_table_pitch(a.nx, false, sizeof(R));
    return with_tile<R>(a.nx, kXU, [&](auto tn, auto even) {
        constexpr int TN = decltype(tn)::value;
        const dim3 grid((rows + kM - 1) / kM, tp / (kXU * TN), a.ngrp);
        auto kern = dft_rows_inv<R, TN, decltype(even)::value>;
        cudaError_t e = set_smem(kern, rows_smem<R, TN>(), s);
        if (e != cudaSuccess) return e;
        step_launch(kern, grid, kThreads, rows_smem<R, TN>(), s, (const R2 *)a.spec, (R *)a.phip,
                    (const R2 *)a.tabx, tp, a.nx, a.ny, rows, a.pitch, a.grp);
        return cudaGetLastError();
    });
}
template <typename R>
cudaError_t launch_dft_cols(const PoissonArgs &a, int sign, cudaStream_t s) {
    using R2 = typename Cplx<R>::T;
    const int mtiles = (a.nxh + kM - 1) / kM, tp = dft_table_pitch(a.ny, true, sizeof(R));
    return with_tile<R>(a.ny, kYU, [&](auto tn, auto even) {
        constexpr int TN = decltype(tn)::value;
        const dim3 grid(mtiles * (tp / (kYU * TN)), a.nz - 2, a.ngrp);
        auto kern = sign < 0 ? dft_cols<R, -1, TN, decltype(even)::value>
                             : dft_cols<R, 1, TN, decltype(even)::value>;
        cudaError_t e = set_smem(kern, cols_smem<R, TN>(), s);
        if (e != cudaSuccess) return e;
        step_launch(kern, grid, kThreads, cols_smem<R, TN>(), s,
                    (const R2 *)(sign < 0 ? a.spec : a.spec2), (R2 *)(sign < 0 ? a.spec2 : a.spec), (const R2 *)a.taby, tp, a.ny, a.nxh, a.pitch, mtiles, a.rowsum, a.planesum, a.grp);
        return cudaGetLastError();
    });
}

// 32 modes a block where two such blocks share a multiprocessor, 16 up to
// what one block may use, 0: the columns do not fit
int zmeet_modes(int nz, size_t rsize) {
    const size_t col = 2 * rsize * (size_t)(nz - 2);
    if (32 * col <= 100 * 1024) return 32;
    return 16 * col <= 220 * 1024 ? 16 : 0;
}
template <typename R>
cudaError_t launch_zmeet(const PoissonArgs &a, cudaStream_t s) {
    using R2 = typename Cplx<R>::T;
    const int mb = zmeet_modes(a.nz, sizeof(R)), modes = a.nxh * a.ny;
    // (at least the mean mode's two FP64 arrays and partial sums)
    const size_t cols = sizeof(R2) * (size_t)mb * (a.nz - 2),
                 mean = sizeof(double) * (2 * (size_t)a.nz + 8);
    const size_t sm = cols > mean ? cols : mean;
    cudaError_t e = set_smem(poisson_zmeet<R>, sm, s);
    if (e != cudaSuccess) return e;
    step_launch(poisson_zmeet<R>, dim3((modes + mb - 1) / mb + 1, 1, a.ngrp), 128, sm, s,
                (R2 *)a.spec, a.cpt, a.planesum, a.qmean, a.phi00, a.ez00, a.nx, a.ny, a.nz,
                a.nxh, a.pitch, mb, a.dz, a.eps, a.voltage, 2.0 * M_PI / a.lx, 2.0 * M_PI / a.ly,
                a.grp);
    return cudaGetLastError();
}

#define EHD_INST_DFT(R)                                                       \
    template cudaError_t prepare_zmeet<R>();                                 \
    template cudaError_t prepare_dft<R>(int, int);                           \
    template cudaError_t launch_dft_rows_fwd<R>(const PoissonArgs &, cudaStream_t); \
    template cudaError_t launch_dft_rows_inv<R>(const PoissonArgs &, cudaStream_t); \
    template cudaError_t launch_dft_cols<R>(const PoissonArgs &, int, cudaStream_t); \
    template cudaError_t launch_zmeet<R>(const PoissonArgs &, cudaStream_t);
EHD_INST_DFT(float)
EHD_INST_DFT(double)

}  // namespace ehd
