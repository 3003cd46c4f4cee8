// fednl_refmode.cuh -- the round in the reference's own operation order (desc.arith_order = 1).
//
// The reference's AVX2 build (dopt SUPPORT_CPU_AVX_256_bits=1, SUPPORT_CPU_FMA_EXT=0, no FMA
// contraction) fixes the order of every floating-point operation of a round.  The kernels here
// perform the same IEEE operations in the same order, so a round reproduces the reference's values
// bit for bit given the same inputs:
//   * margins: one Vec4d accumulator, attribute j < 4 floor(d/4) into lane j mod 4, reduced as
//     (c0 + c2) + (c1 + c3), the remaining attributes added in order
//     (MatrixNMD_SIMD_double.h:1256-1430);
//   * sigmoid: the vectorclass exp in SIMD lanes (exp_d<Vec4d>, vectormath_exp.h:141-230) for
//     samples s < 8 floor(n/8); libm's exp on the scalar tail, here the correctly rounded exp
//     (glibc returns the other neighbour for a few inputs in ten thousand);
//   * ||diff||_F from the upper part (MatrixNMD_SIMD_double.h:1068-1253): eight lane accumulators
//     shared by all columns, a scalar for each column's tail rows and one for the diagonal;
//   * TopLEK's window numerators one by one in heap-array and then extraction order
//     (SpecialMathRoutinesForMatrix.h:435-503), in k_select;
//   * Cholesky (CholeskyFactorization.h:153-272) and the two triangular solves
//     (ElementarySolvers.h:71-224) with two-Vec4d dot products: element k < 8 floor(n/8) into lane
//     k mod 8, lanes reduced as (0 + h(c0..c3)) + h(c4..c7), h(c) = (c0 + c2) + (c1 + c3), the tail
//     summed in order from 0 and added last (LightVector_SIMD_double.h:233-380);
//   * the objective's loss with the vectorclass log in lanes (log_d<Vec4d>, vectormath_exp.h:947-1003).
#pragma once

#include "fednl_kernels.cuh"

namespace fednl {
namespace refo {

// ---- scalar restatements of the reference's lane arithmetic -------------------------------------

// exp_d<Vec4d, 0, 0> of one lane, without FMA (mul_add(a, b, c) = a b + c, nmul_add(a, b, c) = c - a b)
__device__ __forceinline__ double exp_vcl(double x0)
{
    if (x0 != x0) return x0;
    if (!(fabs(x0) < 708.39)) return x0 < 0.0 ? 0.0 : __longlong_as_double(0x7ff0000000000000ll);
    const double p2 = 0x1p-1, p3 = 0x1.5555555555555p-3, p4 = 0x1.5555555555555p-5, p5 = 0x1.1111111111111p-7;
    const double p6 = 0x1.6c16c16c16c17p-10, p7 = 0x1.a01a01a01a01ap-13, p8 = 0x1.a01a01a01a01ap-16;
    const double p9 = 0x1.71de3a556c734p-19, p10 = 0x1.27e4fb7789f5cp-22, p11 = 0x1.ae64567f544e4p-26;
    const double p12 = 0x1.1eed8eff8d898p-29, p13 = 0x1.6124613a86d09p-33;
    const double ln2d_hi = 0.693145751953125, ln2d_lo = 1.42860682030941723212E-6;
    const double r = rint(__dmul_rn(x0, 1.44269504088896340736));
    double x = __dsub_rn(x0, __dmul_rn(r, ln2d_hi));
    x = __dsub_rn(x, __dmul_rn(r, ln2d_lo));
    const double x2 = __dmul_rn(x, x), x4 = __dmul_rn(x2, x2), x8 = __dmul_rn(x4, x4);
    const double hi = __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(p13, x), p12), x4),
                                __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(p11, x), p10), x2), __dadd_rn(__dmul_rn(p9, x), p8)));
    const double lo = __dadd_rn(
        __dmul_rn(__dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(p7, x), p6), x2), __dadd_rn(__dmul_rn(p5, x), p4)), x4),
        __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(p3, x), p2), x2), x));
    const double z = __dadd_rn(__dmul_rn(hi, x8), lo);
    return __dmul_rn(__dadd_rn(z, 1.0), pow2i((int)r));
}

struct dd {
    double hi, lo;
};

__device__ __forceinline__ dd dd_norm(double s, double e)
{
    const double t = __dadd_rn(s, e);
    return dd{t, __dsub_rn(e, __dsub_rn(t, s))};
}

__device__ __forceinline__ dd dd_add(dd a, dd b)
{
    double s, e;
    two_sum(a.hi, b.hi, s, e);
    e = __dadd_rn(e, __dadd_rn(a.lo, b.lo));
    return dd_norm(s, e);
}

__device__ __forceinline__ dd dd_mul(dd a, dd b)
{
    const double p = __dmul_rn(a.hi, b.hi);
    double e = __fma_rn(a.hi, b.hi, -p);
    e = __dadd_rn(e, __dadd_rn(__dmul_rn(a.hi, b.lo), __dmul_rn(a.lo, b.hi)));
    return dd_norm(p, e);
}

// Correctly rounded exp (own method): x = k ln2 + r with ln2 in three parts (30-bit head: k L1 and
// x - k L1 exact), r as a double-double; exp(r 2^-10) by its Taylor series to degree 9 in
// double-double arithmetic, squared ten times; one rounding of hi + lo; exact scaling by 2^k.
// Below 2^-90 relative error before the rounding: the correctly rounded result for normal results.
__device__ __forceinline__ double exp_cr(double x)
{
    if (x != x) return x;
    if (x > 709.782712893384) return __longlong_as_double(0x7ff0000000000000ll);
    if (x < -745.1332191019412) return 0.0;
    const double L1 = 0x1.62e42fe8p-1, L2 = 0x1.e8e7bcd5e4f1ep-31, L3 = -0x1.8cff81a12a17ep-85;
    const double fh[10] = {1.0, 1.0, 0x1p-1, 0x1.5555555555555p-3, 0x1.5555555555555p-5, 0x1.1111111111111p-7,
                           0x1.6c16c16c16c17p-10, 0x1.a01a01a01a01ap-13, 0x1.a01a01a01a01ap-16, 0x1.71de3a556c734p-19};
    const double fl[10] = {0.0, 0.0, 0.0, 0x1.5555555555555p-57, 0x1.5555555555555p-59, 0x1.1111111111111p-63,
                           -0x1.f49f49f49f49fp-65, 0x1.a01a01a01a01ap-73, 0x1.a01a01a01a01ap-76, -0x1.c154f8ddc6c00p-73};
    const double kd = rint(__dmul_rn(x, 0x1.71547652b82fep+0));
    const double r1 = __dsub_rn(x, __dmul_rn(kd, L1));
    const double p2 = __dmul_rn(kd, L2);
    const double p2e = __fma_rn(kd, L2, -p2);
    double s, e;
    two_sum(r1, -p2, s, e);
    e = __dsub_rn(__dsub_rn(e, p2e), __dmul_rn(kd, L3));
    dd y = dd_norm(s, e);
    y.hi = __dmul_rn(y.hi, 0x1p-10);
    y.lo = __dmul_rn(y.lo, 0x1p-10);
    dd t{fh[9], fl[9]};
#pragma unroll
    for (int n = 8; n >= 0; --n) t = dd_add(dd_mul(t, y), dd{fh[n], fl[n]});
#pragma unroll
    for (int q = 0; q < 10; ++q) t = dd_mul(t, t);
    const double p = __dadd_rn(t.hi, t.lo);
    const int k = (int)kd;
    if (k > 1000) return __dmul_rn(__dmul_rn(p, pow2i(k - 1000)), pow2i(1000));
    if (k < -1000) return __dmul_rn(__dmul_rn(p, pow2i(k + 1000)), pow2i(-1000));
    return __dmul_rn(p, pow2i(k));
}

// log_d<Vec4d, 0> of one lane, without FMA, for positive normal inputs (zero -> -inf, +inf -> +inf)
__device__ __forceinline__ double log_vcl(double x1)
{
    if (x1 != x1 || x1 < 0.0) return __longlong_as_double(0x7ff8000000000000ll);
    if (x1 == 0.0) return __longlong_as_double((long long)0xfff0000000000000ull);
    if (x1 == __longlong_as_double(0x7ff0000000000000ll)) return x1;
    const double ln2_hi = 0.693359375, ln2_lo = -2.121944400546905827679E-4;
    const double P0 = 7.70838733755885391666E0, P1 = 1.79368678507819816313E1, P2 = 1.44989225341610930846E1;
    const double P3 = 4.70579119878881725854E0, P4 = 4.97494994976747001425E-1, P5 = 1.01875663804580931796E-4;
    const double Q0 = 2.31251620126765340583E1, Q1 = 7.11544750618563894466E1, Q2 = 8.29875266912776603211E1;
    const double Q3 = 4.52279145837532221105E1, Q4 = 1.12873587189167450590E1;
    const unsigned long long b = (unsigned long long)__double_as_longlong(x1);
    double x = __longlong_as_double((long long)((b & 0x000FFFFFFFFFFFFFull) | 0x3FE0000000000000ull));
    double fe = __dsub_rn((double)(long long)(b >> 52), 1023.0);
    if (x > __dmul_rn(1.41421356237309504880, 0.5)) fe = __dadd_rn(fe, 1.0);
    else x = __dadd_rn(x, x);
    x = __dsub_rn(x, 1.0);
    const double xx2 = __dmul_rn(x, x), xx4 = __dmul_rn(xx2, xx2);
    double px = __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(P3, x), P2), xx2),
                          __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(P5, x), P4), xx4), __dadd_rn(__dmul_rn(P1, x), P0)));
    const double x2 = __dmul_rn(x, x);
    px = __dmul_rn(px, __dmul_rn(x, x2));
    const double qx = __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(Q3, x), Q2), xx2),
                                __dadd_rn(__dmul_rn(__dadd_rn(Q4, x), xx4), __dadd_rn(__dmul_rn(Q1, x), Q0)));
    double res = __ddiv_rn(px, qx);
    res = __dadd_rn(__dmul_rn(fe, ln2_lo), res);
    res = __dadd_rn(res, __dsub_rn(x, __dmul_rn(x2, 0.5)));
    res = __dadd_rn(__dmul_rn(fe, ln2_hi), res);
    return res;
}

// the reference's sigmoid of sample sl of a client with n samples (elementwiseSigmoid,
// VectorND_Raw_SIMD_double.h:1596-1650)
__device__ __forceinline__ double sigmoid_at(double m, int sl, int n)
{
    const double e = (sl < (n & ~7)) ? exp_vcl(-m) : exp_cr(-m);
    return __ddiv_rn(1.0, __dadd_rn(1.0, e));
}

// -log sigma of the loss (logisticUnweightedLossFromMarginSigmoid, :1464-1532): vectorclass log in
// the lanes, the own log on the tail (the reference takes libm's there)
__device__ __forceinline__ double negloss_at(double sig, int sl, int n)
{
    return (sl < (n & ~7)) ? -log_vcl(sig) : -fednl_log(sig);
}

// (0 + h(c0..c3)) + h(c4..c7) with h(c) = (c0 + c2) + (c1 + c3): the two-Vec4d reduction
__device__ __forceinline__ double lanes8(const double* c)
{
    double fin = __dadd_rn(0.0, __dadd_rn(__dadd_rn(c[0], c[2]), __dadd_rn(c[1], c[3])));
    return __dadd_rn(fin, __dadd_rn(__dadd_rn(c[4], c[6]), __dadd_rn(c[5], c[7])));
}

// two-Vec4d dot product of a[i] b[i], i < n, by one thread
__device__ __forceinline__ double dot8_seq(const double* a, const double* b, int n)
{
    double c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int items = n & ~7;
    int i = 0;
    for (; i < items; i += 8)
#pragma unroll
        for (int l = 0; l < 8; ++l) c[l] = __dadd_rn(c[l], __dmul_rn(a[i + l], b[i + l]));
    double rest = 0.0;
    for (; i < n; ++i) rest = __dadd_rn(rest, __dmul_rn(a[i], b[i]));
    return __dadd_rn(lanes8(c), rest);
}

// the same by the 32 lanes of a warp: lanes 0-7 take the Vec4d lanes, lane 8 the tail; the result
// is valid in lane 0
__device__ __forceinline__ double dot8_warp(const double* a, const double* b, int n)
{
    const int lane = threadIdx.x & 31;
    const int items = n & ~7;
    double acc = 0.0;
    if (lane < 8) {
        for (int i = lane; i < items; i += 8) acc = __dadd_rn(acc, __dmul_rn(a[i], b[i]));
    } else if (lane == 8) {
        for (int i = items; i < n; ++i) acc = __dadd_rn(acc, __dmul_rn(a[i], b[i]));
    }
    double c[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) c[l] = __shfl_sync(0xffffffffu, acc, l);
    const double rest = __shfl_sync(0xffffffffu, acc, 8);
    return __dadd_rn(lanes8(c), rest);
}

}  // namespace refo

// ---- 1r. margins, sigmoid and per-sample weights in the reference's order ---------------------
// Binary features: the nonzero products are +-x_j (labels +-1), zero products leave a lane
// unchanged, so a lane sums x over the sample's set attributes of its residue class; the label
// multiplies the finished sum (negation commutes with round-to-nearest).
__device__ __forceinline__ void margin_weights_ref(const Dev& P, int s, double m)
{
    const int c = P.client_of[s];
    const int n = P.ns[c], sl = s - P.soff[c];
    const double sig = refo::sigmoid_at(m, sl, n);
    const double inv_m = 1.0 / (double)n;
    const double z1 = __dsub_rn(1.0, sig);
    const double b = P.lab[s];
    P.Dv[s] = __dmul_rn(inv_m, __dmul_rn(z1, sig));
    const double q = __dmul_rn(z1, -inv_m);
    P.qb[s] = (P.A != nullptr || b == 1.0) ? q : __dmul_rn(-1.0, q);   // dense: the label enters through u
    if (P.fmode) P.fterm[s] = refo::negloss_at(sig, sl, n);
}

__device__ __forceinline__ double margin_binary_ref(const Dev& P, const double* x, int s)
{
    const int cb = P.d & ~3;
    double c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
    int t = P.rowptr[s];
    const int t1 = P.rowptr[s + 1];
    for (; t < t1; ++t) {
        const int j = P.colidx[t];
        if (j >= cb) break;
        const double v = x[j];
        switch (j & 3) {
        case 0: c0 = __dadd_rn(c0, v); break;
        case 1: c1 = __dadd_rn(c1, v); break;
        case 2: c2 = __dadd_rn(c2, v); break;
        default: c3 = __dadd_rn(c3, v); break;
        }
    }
    double acc = __dadd_rn(__dadd_rn(c0, c2), __dadd_rn(c1, c3));
    for (; t < t1; ++t) acc = __dadd_rn(acc, x[P.colidx[t]]);
    return (P.lab[s] == 1.0) ? acc : -acc;
}

__device__ __forceinline__ double margin_dense_ref(const Dev& P, const double* x, int s)
{
    const int d = P.d, cb = d & ~3;
    const double b = P.lab[s];
    const double* a = P.A + (size_t)s * d;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    int j = 0;
    for (; j < cb; j += 4)
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const double u = (b == 1.0) ? a[j + l] : __dmul_rn(a[j + l], -1.0);
            c[l] = __dadd_rn(c[l], __dmul_rn(u, x[j + l]));
        }
    double acc = __dadd_rn(__dadd_rn(c[0], c[2]), __dadd_rn(c[1], c[3]));
    for (; j < d; ++j) {
        const double u = (b == 1.0) ? a[j] : __dmul_rn(a[j], -1.0);
        acc = __dadd_rn(acc, __dmul_rn(u, x[j]));
    }
    return acc;
}

__global__ void k_margin_ref(Dev P, int S)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const double m = (P.A == nullptr) ? margin_binary_ref(P, P.x, s) : margin_dense_ref(P, P.x, s);
    margin_weights_ref(P, s, m);
}

// FedNL-LS trial point: -log sigma_s only
__global__ void k_ls_margin_ref(Dev P, int S)
{
    if (P.ls[2] != 0.0) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const double m = (P.A == nullptr) ? margin_binary_ref(P, P.x, s) : margin_dense_ref(P, P.x, s);
    const int c = P.client_of[s];
    const int n = P.ns[c], sl = s - P.soff[c];
    P.fterm[s] = refo::negloss_at(refo::sigmoid_at(m, sl, n), sl, n);
}

// ---- 3r. ||diff||_F^2 from the packed upper part, per processed client ----------------------
// For the compressors without a selection kernel (TopK / TopLEK: select_frob_ref, in k_select).
// One CTA per client.  The ten running sums of the reference's loop are chains of dependent FP64
// adds (eight lane accumulators shared by all columns: column j, rows i < 8 floor(j/8) with
// i mod 8 = lane; one scalar for rows 8 floor(j/8) .. j-1; one for the diagonal), and a dependent
// FP64 add costs about 64 cycles on this part, so everything else is taken off those chains: warps
// 1..7 stage the squares of the coming columns into a ring of shared-memory buffers while warp 0's
// lanes 0..9 add one column's squares to their sums.
constexpr int kFrobRefThreads = 256;
constexpr int kFrobRing = 4;                       // ring buffers: a column is added 3 steps after staging

__global__ void __launch_bounds__(kFrobRefThreads) k_frob_ref(Dev P)
{
    extern __shared__ double s_sq[];               // [kFrobRing][d]
    const int c = P.act ? P.act[blockIdx.x] : blockIdx.x;
    const double* v = P.diff + (size_t)c * P.ustr;
    const int d = P.d, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double acc = 0.0;
    // step j0: warps 1..7 stage column j0 into buffer j0 % kFrobRing; warp 0 adds column
    // j0 - (kFrobRing - 1), staged kFrobRing - 1 barriers earlier, from its buffer (a different one)
    for (int j0 = 0; j0 < d + kFrobRing - 1; ++j0) {
        if (warp > 0 && j0 < d) {
            double* buf = s_sq + (size_t)(j0 % kFrobRing) * d;
            const double* col = v + (size_t)j0 * (j0 + 1) / 2;
            for (int i = tid - 32; i <= j0; i += kFrobRefThreads - 32) buf[i] = __dmul_rn(col[i], col[i]);
        }
        const int j = j0 - (kFrobRing - 1);
        if (warp == 0 && j >= 0) {
            const double* buf = s_sq + (size_t)(j % kFrobRing) * d;
            const int items = j & ~7;
            if (lane < 8) {
                for (int i = lane; i < items; i += 8) acc = __dadd_rn(acc, buf[i]);
            } else if (lane == 8) {
                for (int i = items; i < j; ++i) acc = __dadd_rn(acc, buf[i]);
            } else if (lane == 9) {
                acc = __dadd_rn(acc, buf[j]);
            }
        }
        __syncthreads();
    }
    if (warp == 0) {
        double c8[8];
#pragma unroll
        for (int l = 0; l < 8; ++l) c8[l] = __shfl_sync(0xffffffffu, acc, l);
        const double rest = __shfl_sync(0xffffffffu, acc, 8);
        const double diag = __shfl_sync(0xffffffffu, acc, 9);
        if (lane == 0) {
            double out = refo::lanes8(c8);
            out = __dadd_rn(out, rest);
            const double f = __dadd_rn(__dadd_rn(out, out), diag);
            P.F[c] = f;
            if (!P.pp) P.lk[c] = sqrt(f);
        }
    }
}

// ---- 8cr. objective values ------------------------------------------------------------------
// f_i = loss + (lambda / 2) ||x||^2 (evaluateFunction(x, margin, sigmoid), logistic_regression.h:
// 119-123): the loss's lanes over the client's samples, its tail, (fin + rest) / n; one warp per
// client; skipped once the line search has finished (gate = P.ls)
__global__ void k_fclient_ref(Dev P, const double* x, const double* gate)
{
    if (gate && gate[2] != 0.0) return;
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (c >= P.nc) return;
    const int lane = threadIdx.x & 31;
    const int n = P.ns[c];
    const double* ft = P.fterm + P.soff[c];
    const int items = n & ~7;
    double acc = 0.0;
    if (lane < 8) {
        for (int i = lane; i < items; i += 8) acc = __dadd_rn(acc, ft[i]);
    } else if (lane == 8) {
        for (int i = items; i < n; ++i) acc = __dadd_rn(acc, ft[i]);
    }
    double c8[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) c8[l] = __shfl_sync(0xffffffffu, acc, l);
    const double rest = __shfl_sync(0xffffffffu, acc, 8);
    const double loss = __ddiv_rn(__dadd_rn(refo::lanes8(c8), rest), (double)n);
    const double xs = refo::dot8_warp(x, x, P.d);
    if (lane == 0) P.fi[c] = __dadd_rn(loss, __dmul_rn(__ddiv_rn(P.lambda, 2.0), xs));
}

// master: f = (f_0 + f_1 + ... in client order) / n (function_aggregation, TrainLoop.h:1511-1541)
__device__ __forceinline__ double client_mean_ref(const Dev& P)
{
    double s = 0.0;
    for (int c = 0; c < P.nc; ++c) s = __dadd_rn(s, P.fi[c]);
    return __dmul_rn(s, P.inv_n);
}

__global__ void k_fmaster_ref(Dev P, double* out)
{
    if (threadIdx.x == 0) *out = client_mean_ref(P);
}

// FedNL-LS: t = 1, -(dx . g) as the reference's dot product, x_k kept
__global__ void k_ls_init_ref(Dev P)
{
    for (int i = threadIdx.x; i < P.d; i += blockDim.x) P.xprev[i] = P.x[i];
    if (threadIdx.x < 32) {
        const double dg = refo::dot8_warp(P.dx, P.g, P.d);
        if (threadIdx.x == 0) {
            P.ls[0] = 1.0;
            P.ls[1] = -dg;
            P.ls[2] = P.ls[4] != 0.0 ? 0.0 : 1.0;
            P.ls[3] = 0.0;
        }
    }
}

__global__ void k_ls_check_ref(Dev P, double c, double gamma)
{
    if (P.ls[2] != 0.0) return;
    if (threadIdx.x == 0) {
        const double fr = client_mean_ref(P);
        P.ls[3] = __dadd_rn(P.ls[3], 1.0);
        const double t = P.ls[0];
        if (fr <= __dadd_rn(P.stats[2], __dmul_rn(__dmul_rn(c, t), P.ls[1]))) P.ls[2] = 1.0;
        else P.ls[0] = __dmul_rn(t, gamma);
    }
}

// ---- 8r. Option-B solve in the reference's order -------------------------------------------
// choleskyFactorization<.., true, true> computes column i of R (= L^T) row by row:
// R_ji = (1 / R_jj)(H_ji - R[0:j, i] . R[0:j, j]) for j < i, then R_ii = sqrt((H_ii + l) -
// ||R[0:i, i]||^2); forwardSubstitutionWithATranspose gives y_j = (g_j - R[0:j, j] . y[0:j]) / R_jj,
// backwardSubstitutionWithATranspose x_i = (y_i - R[i, i+1:d] . x[i+1:d]) / R_ii, all dot products
// in the two-Vec4d order.  In the dot of entry (j, i) over k < j, row k goes to lane k mod 8 when
// k < 8 floor(j/8) and to the in-order tail otherwise; the terms of each lane and of the tail are
// added in increasing k, which is the order in which the rows of R are finished.  So the kernel runs
// right-looking with eight lane accumulators per entry of the augmented matrix [H | g] (g as column d,
// whose entries become y), in panels of 32 rows:
//   1. every CTA finishes the panel's 32 x 32 block redundantly (no barrier) and, behind it, its own
//      share of the columns to the right, all in shared memory, 8 rows at a time: the rows' lane sums are
//      reduced (L); warp 0 runs the pivots' chain one row ahead (tail, square root and reciprocal by
//      integer arithmetic); warp 1 forms the 8 x 8 block's rows, a lane per entry; warp 3 the block's
//      columns right of it and warps 2 and 5-7 the own columns follow warp 1 row by row; then all warps
//      add the 8 rows to the lanes of the panel's later rows;
//   2. grid barrier; the CTAs add the panel's rows to the lanes of the trailing entries in tiles, four rows
//      a lane; grid barrier.
// The backward substitution runs in CTA 0.  Row i's lane q starts with x[i + 1 + q], the value found q
// rows earlier, so when x[t] is known, lane q of warp 0 forms lane q of row t - 1 - q, all from x[t],
// x[t + 8], ...; lane 0 completes row t - 1.  Other warps form the next step's products and the row's
// finished partial sums, so warp 0 issues one dependent add per product and the row's last operations.
// Every value equals the reference's.
// Bound by these chains (a dependent FP64 add takes 64 cycles): 1260 cycles a row of the factorisation
// and 1440 + 8 (d - i) a row of the substitution.  d = 301: 2735 -> 783 us (before: one CTA finishing 8
// rows at a time from lanes in global memory, a substitution whose products waited for their loads).
constexpr int kRefCholThreads = 256;
constexpr int kRefNB = 32;                                       // panel rows
constexpr int kRefSlab = 16;                                     // panel columns of a CTA per pass
constexpr int kRefBlock = kRefNB * (kRefNB + 1) / 2;             // block entries (j, i), j <= i
constexpr int kRefSmemD = 8192;

__device__ __forceinline__ size_t apos(int j, int i) { return (size_t)i * (i + 1) / 2 + j; }

// columns a CTA holds at once, and its dynamic shared memory: lanes [8][E], H [E], L [8][64], the rows
// [32][65] (block columns 0..31, own columns 32..63); the substitution reuses it: products
// [2][8 ceil(d / 8)] and x [d] (larger d keeps them in global memory)
__host__ __device__ inline int ref_slab(int d, int G) { return d / G + 1 < kRefSlab ? d / G + 1 : kRefSlab; }
__host__ __device__ inline size_t ref_chol_smem(int d, int G)
{
    const size_t E = kRefBlock + (size_t)kRefNB * ref_slab(d, G);
    const size_t fac = (9 * E + 8 * 64 + kRefNB * 65) * 8;
    const size_t sub = d <= kRefSmemD ? (2 * (size_t)((d + 7) & ~7) + d) * 8 : 0;
    return fac > sub ? fac : sub;
}

__device__ __forceinline__ double plus_zero(double v)        // 0.0 + v without the FP64 pipe
{
    return __double_as_longlong(v) == (long long)0x8000000000000000ull ? 0.0 : v;
}

// RN(a / b) from inv = RN(1 / b): two Markstein steps (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000", 1990): the first leaves a faithful quotient, the second, its
// remainder exact, rounds it correctly.  Five operations, about half the cycles of the division; operands
// and quotients near the ends of the exponent range (tested beside the operations) take the division.
__device__ __forceinline__ double div_by(double a, double b, double inv)
{
    double q = __dmul_rn(a, inv);
    q = __fma_rn(__fma_rn(-q, b, a), inv, q);
    q = __fma_rn(__fma_rn(-q, b, a), inv, q);
    const int ea = (int)((unsigned long long)__double_as_longlong(a) >> 52) & 0x7ff;
    const int eb = (int)((unsigned long long)__double_as_longlong(b) >> 52) & 0x7ff;
    if ((unsigned)(ea - 200) > 1600u || (unsigned)(eb - 200) > 1600u || (unsigned)(ea - eb + 800) > 1600u)
        q = __ddiv_rn(a, b);
    return q;
}

__global__ void __launch_bounds__(kRefCholThreads, 1) k_chol_ref(Dev P, const double* __restrict__ Hin,
                                                                 const double* lptr, double lval,
                                                                 const double* __restrict__ gin, double* dxout,
                                                                 double* xupd, int record)
{
    extern __shared__ double s_ref[];
    GridSync gs(P.bar, gridDim.x);
    __shared__ double s_r[kRefNB], s_inv[kRefNB], s_num1[8], s_tl[8], s_ls[16][8], s_part[2][2], s_last[80], s_ent[4][12];
    __shared__ int s_bad, s_neg[8];       // a pivot of the factorisation / row k of the 8 was negative
    const int d = P.d, D = d + 1, tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int G = gridDim.x, bid = blockIdx.x;
    const size_t Ua = (size_t)D * (d + 2) / 2;
    double* R = P.rref;                       // [Ua] R, column d = y
    double* acc = P.racc;                     // [8][Ua] lanes of the entries right of and below the panel
    double* rinv = P.work;                    // [d] 1 / R_kk
    const double l = lptr ? *lptr : lval;
    const int slab = ref_slab(d, G), E = kRefBlock + kRefNB * slab;
    double* AL = s_ref;                       // [8][E]
    double* HV = AL + 8 * (size_t)E;          // [E]
    double(*Lr)[64] = reinterpret_cast<double(*)[64]>(HV + E);
    double(*RB)[65] = reinterpret_cast<double(*)[65]>(HV + E + 8 * 64);
    if (P.ls && bid == 0 && tid == 0) P.ls[4] = 0.0;
    if (record && bid == G - 1 && warp == 7) {      // ||g||, for the round's statistics
        const double gsq = refo::dot8_warp(gin, gin, d);
        if (lane == 0) P.stats[0] = sqrt(gsq);
    }
    if (tid == 0) s_bad = 0;
    for (int c0 = 0; c0 < d; c0 += kRefNB) {
        const int nb = min(kRefNB, d - c0), c1 = c0 + nb;
        const int ntot = D - c1 > bid ? (D - c1 - bid + G - 1) / G : 0;     // own columns c1 + bid + s G
        // own columns in passes of `slab` (one pass unless d > 32 G); the block is redone in each
        for (int base = 0; base == 0 || base < ntot; base += slab) {
            const int ns = max(0, min(slab, ntot - base));
            const int col0 = c1 + bid + base * G;                            // global column of own column 0
            __syncthreads();
            // entries of the panel: block (j, i) at i (i + 1) / 2 + j, own column s at kRefBlock + 32 s + j
            for (int e = tid; e < kRefBlock + kRefNB * ns; e += nthr) {
                int j, i;
                if (e < kRefBlock) {
                    upper_ij(e, j, i);
                    if (i >= nb) continue;
                    i += c0;
                } else {
                    j = (e - kRefBlock) & (kRefNB - 1);
                    if (j >= nb) continue;
                    i = col0 + ((e - kRefBlock) / kRefNB) * G;
                }
                j += c0;
                double v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = c0 ? acc[q * Ua + apos(j, i)] : 0.0;
                const double h = i < d ? Hin[up_pos(j, i)] : gin[j];
#pragma unroll
                for (int q = 0; q < 8; ++q) AL[q * (size_t)E + e] = v[q];
                HV[e] = i == j ? __dadd_rn(h, l) : h;
            }
            __syncthreads();
            for (int r0 = 0; r0 < nb; r0 += 8) {
                const int nr = min(8, nb - r0), r1 = r0 + 8, m = nb - r1;     // rows of the panel after them
                // L of the 8 rows: a warp per block row, then the own columns' entries
                for (int t = tid; t < 8 * kRefNB + 8 * ns; t += nthr) {
                    const bool blk = t < 8 * kRefNB;
                    const int q = blk ? t >> 5 : (t - 8 * kRefNB) / ns, j = r0 + q;
                    const int s = blk ? t & 31 : (t - 8 * kRefNB) - q * ns;
                    if (q >= nr || (blk && (s < j || s >= nb))) continue;
                    const int e = blk ? s * (s + 1) / 2 + j : kRefBlock + kRefNB * s + j;
                    double c8[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) c8[u] = AL[u * (size_t)E + e];
                    Lr[q][blk ? s : 32 + s] = refo::lanes8(c8);
                }
                __syncthreads();
                if (warp == 0) {
                    // the pivots: sq = L + tail, a = (H + l) - sq, r = sqrt(a), 1 / r
                    const auto pivot = [&](int k, double sq) {
                        const int j = r0 + k;
                        const double a = __dsub_rn(HV[j * (j + 1) / 2 + j], sq);
                        double inv;
                        const double r = sqrt_rcp_rn_int(a, inv);
                        if (lane == 0) {
                            s_r[j] = r;
                            s_inv[j] = inv;
                            s_neg[k] = a < 0.0 ? 1 : 0;
                            if (a < 0.0) s_bad = 1;
                        }
                        return inv;
                    };
                    double inv = pivot(0, Lr[0][r0]);
                    for (int k = 0; k < nr; ++k) {
                        named_sync<64>(1);      // row k's pivot, warp 1's exports
                        if (s_neg[k]) break;
                        if (k + 1 < nr) {
                            const double rk = __dmul_rn(inv, s_num1[k]);
                            const double tl = __dadd_rn(s_tl[k], __dmul_rn(rk, rk));
                            inv = pivot(k + 1, __dadd_rn(Lr[k + 1][r0 + k + 1], tl));
                        }
                    }
                } else if (warp == 1) {
                    // the 8 x 8 block's entries (j, i), 1 <= j <= i < 8, a lane each, in the order of j; row k
                    // is formed by the lanes of row k (lanes 28.. those of row 0)
                    int j = 1, i = 1;
                    {
                        int e = lane < 28 ? lane : 0;
                        while (e >= 8 - j) {
                            e -= 8 - j;
                            ++j;
                        }
                        i = j + e;
                    }
                    const bool on = lane < 28 && i < nr;
                    double tail = 0.0, h = 0.0, L = 0.0;
                    if (on) {
                        const int bi = r0 + i;
                        h = HV[bi * (bi + 1) / 2 + r0 + j];
                        L = Lr[j][bi];
                    }
                    double num0 = 0.0;       // row 0: lane i holds column i (1..7)
                    if (lane >= 1 && lane < nr) {
                        const int bi = r0 + lane;
                        num0 = __dsub_rn(HV[bi * (bi + 1) / 2 + r0], Lr[0][bi]);
                    }
                    if (lane == 1) {
                        s_num1[0] = num0;
                        s_tl[0] = 0.0;
                    }
                    for (int k = 0; k < nr; ++k) {
                        named_sync<64>(1);      // row k's pivot
                        if (s_neg[k]) {
                            named_arrive<192>(3 + k);
                            break;
                        }
                        const double inv = s_inv[r0 + k];
                        if (k == 0) {
                            const double r = __dmul_rn(inv, num0);
                            if (lane < nr) RB[r0][r0 + lane] = lane == 0 ? s_r[r0] : r;
                        } else {
                            const double r = __dmul_rn(inv, num0);
                            if (on && j == k) RB[r0 + k][r0 + i] = i == k ? s_r[r0 + k] : r;
                        }
                        __threadfence_block();
                        named_arrive<192>(3 + k);
                        if (k + 1 < nr) {
                            const bool later = on && j > k;
                            const double rj = later ? RB[r0 + k][r0 + j] : 0.0, ri = later ? RB[r0 + k][r0 + i] : 0.0;
                            const double nt = __dadd_rn(tail, __dmul_rn(rj, ri));
                            tail = later ? nt : tail;
                            num0 = __dsub_rn(h, __dadd_rn(L, tail));       // of use for row k + 1
                            if (on && j == k + 1 && i == k + 2) s_num1[k + 1] = num0;
                            if (on && j == k + 2 && i == k + 2) s_tl[k + 1] = tail;      // for pivot k + 2
                        }
                    }
                } else if (warp == 3) {
                    // the block's columns right of the 8, a lane each, row by row behind warp 1
                    const int i = r0 + 8 + lane;
                    const bool on = i < nb;
                    double tail[8], h[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        tail[q] = 0.0;
                        h[q] = on ? HV[i * (i + 1) / 2 + r0 + q] : 0.0;
                    }
                    double num = on ? __dsub_rn(h[0], Lr[0][i]) : 0.0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        if (k >= nr) break;
                        named_sync<192>(3 + k);
                        if (s_neg[k]) break;
                        if (m <= 0) continue;
                        const double r = __dmul_rn(s_inv[r0 + k], num);
                        if (on) RB[r0 + k][i] = r;
#pragma unroll
                        for (int q = k + 1; q < 8; ++q) {        // the row joins the tails of the 8 rows after it
                            tail[q] = __dadd_rn(tail[q], __dmul_rn(RB[r0 + k][r0 + q], r));
                            if (q == k + 1) num = __dsub_rn(h[q], __dadd_rn(on ? Lr[q][i] : 0.0, tail[q]));
                        }
                    }
                } else if (warp != 4) {
                    // own columns, four a warp, a lane per column and row: lane 8 c + q holds row q's tail
                    const int s = (warp == 2 ? 0 : warp - 4) * 4 + (lane >> 3), q = lane & 7;
                    const bool on = s < ns && q < nr, isd = col0 + s * G == d;
                    const double h = on ? HV[kRefBlock + kRefNB * s + r0 + q] : 0.0, L = on ? Lr[q][32 + s] : 0.0;
                    const bool any = (s & ~3) < ns;              // the warp has columns
                    double tail = 0.0, num = __dsub_rn(h, L);
                    for (int k = 0; k < nr; ++k) {
                        named_sync<192>(3 + k);
                        if (s_neg[k]) break;
                        if (!any) continue;
                        double r = __dmul_rn(s_inv[r0 + k], num);
                        if (isd && q == k && on) r = div_by(num, s_r[r0 + k], s_inv[r0 + k]);
                        r = __shfl_sync(0xffffffffu, r, (lane & ~7) + k);
                        if (on && q == k) RB[r0 + k][32 + s] = r;
                        if (k + 1 < nr) {
                            const double rj = q > k && q < nr ? RB[r0 + k][r0 + q] : 0.0;
                            const double nt = __dadd_rn(tail, __dmul_rn(rj, r));
                            tail = q > k ? nt : tail;
                            num = __dsub_rn(h, __dadd_rn(L, tail));        // of use for row k + 1
                        }
                    }
                }
                __syncthreads();
                if (s_bad) break;
                // the 8 rows join the lanes of the panel's later rows
                if (m > 0) {
                    const int tb = m * (m + 1) / 2;
                    for (int t = tid; t < tb + m * ns; t += nthr) {
                        int j, i, e;
                        if (t < tb) {
                            upper_ij(t, j, i);
                            j += r1;
                            i += r1;
                            e = i * (i + 1) / 2 + j;
                        } else {
                            const int s = (t - tb) / m;
                            j = r1 + (t - tb) - s * m;
                            i = 32 + s;
                            e = kRefBlock + kRefNB * s + j;
                        }
                        double v[8], u[8], w[8];      // loaded before the first store
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            v[q] = AL[q * (size_t)E + e];
                            u[q] = RB[r0 + q][j];
                            w[q] = RB[r0 + q][i];
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q) AL[q * (size_t)E + e] = __dadd_rn(v[q], __dmul_rn(u[q], w[q]));
                    }
                }
                __syncthreads();
            }
            if (s_bad) break;
            if (bid == 0 && base == 0 && tid < nb) rinv[c0 + tid] = s_inv[tid];
            if (bid == 0 && base == 0)
                for (int e = tid; e < kRefBlock; e += nthr) {
                    int j, i;
                    upper_ij(e, j, i);
                    if (i < nb) R[apos(c0 + j, c0 + i)] = RB[j][i];
                }
            for (int t = tid; t < nb * ns; t += nthr) {
                const int s = t / nb, j = t - s * nb;
                R[apos(c0 + j, col0 + s * G)] = RB[j][32 + s];
            }
        }
        if (s_bad) {      // the same decision in every CTA
            if (bid == 0 && tid == 0) {
                *P.status = -4;
                if (record) *P.round_ctr += 1;
            }
            gs.finish();
            return;
        }
        if (!gs.sync()) goto timeout;
        if (c1 < d) {     // then nb = 32: four rows join each lane of the trailing entries
            // tiles of TS x TS entries, their 2 TS columns of the panel's rows in shared memory; a thread
            // forms (entry, lane) pairs, so a small trailing triangle still fills the warps.  A tile of 16
            // takes about three times as long as one of 8 (FP64 pipe against latency): the size whose
            // rounds over the CTAs are shorter
            const int m = D - c1, n16 = (m + 15) / 16, n8 = (m + 7) / 8;
            const int rounds16 = (n16 * (n16 + 1) / 2 + G - 1) / G, rounds8 = (n8 * (n8 + 1) / 2 + G - 1) / G;
            const int TS = 3 * rounds16 <= rounds8 ? 16 : 8, nt = TS == 16 ? n16 : n8, sh = TS == 16 ? 4 : 3;
            double* A = s_ref;                        // [32][TS + 1] columns j
            double* B = A + kRefNB * (TS + 1);        // [32][TS + 1] columns i
            for (int tile = bid; tile < nt * (nt + 1) / 2; tile += G) {
                int tj, ti;
                upper_ij(tile, tj, ti);
                const int j0 = c1 + tj * TS, i0 = c1 + ti * TS;
                __syncthreads();
                for (int t = tid; t < kRefNB * TS; t += nthr) {
                    const int k = t & (kRefNB - 1), u = t / kRefNB;
                    A[k * (TS + 1) + u] = j0 + u <= d ? R[apos(c0 + k, j0 + u)] : 0.0;
                    B[k * (TS + 1) + u] = i0 + u <= d ? R[apos(c0 + k, i0 + u)] : 0.0;
                }
                __syncthreads();
                for (int t = tid; t < 8 * TS * TS; t += nthr) {
                    const int ju = t & (TS - 1), iu = (t >> sh) & (TS - 1), q = t >> (2 * sh);
                    const int j = j0 + ju, i = i0 + iu;
                    if (j > i || i > d) continue;
                    double* ap = acc + q * Ua + apos(j, i);
                    double a = c0 ? *ap : 0.0;
#pragma unroll
                    for (int k = 0; k < kRefNB; k += 8)
                        a = __dadd_rn(a, __dmul_rn(A[(k + q) * (TS + 1) + ju], B[(k + q) * (TS + 1) + iu]));
                    *ap = a;
                }
            }
            if (!gs.sync()) goto timeout;
        }
    }
    if (bid != 0) {
        gs.finish();
        return;
    }
    {
        // Backward substitution.  Step t: x[t] is known; lane q of warp 0 forms lane q of row t - 1 - q.
        const int pst = (d + 7) & ~7;                     // products per buffer: [m][q], element t + 8 m
        double* prod = d <= kRefSmemD ? s_ref : acc;      // [2][pst]; the lanes are no longer needed
        double* x = d <= kRefSmemD ? s_ref + 2 * (size_t)pst : P.ybuf;
        double* rest = P.rinv;                            // [d] the rows' tails
        auto elems = [&](int i) { return (d - 1 - i) >> 3; };      // of each of row i's lanes
        const int first = max(0, d - 8);                  // rows first .. d-1: fewer than 8 elements, all tail
        __syncthreads();
        // the first rows' entries, y and diagonal in shared memory
        if (tid < 80) {
            const int i = first + tid / 10, c = tid % 10;
            if (i < d) s_last[tid] = c < 8 ? (first + c < d && first + c >= i ? R[apos(i, first + c)] : 0.0)
                                           : c == 8 ? R[apos(i, d)] : rinv[i];
        }
        __syncthreads();
        if (warp == 0) {
            for (int i = d - 1; i >= first; --i) {
                const double* ri = s_last + (i - first) * 10;
                double sum = 0.0;
                for (int t = i + 1; t < d; ++t) sum = __dadd_rn(sum, __dmul_rn(ri[t - first], x[t]));
                const double v = div_by(__dsub_rn(ri[8], __dadd_rn(0.0, sum)), ri[i - first], ri[9]);
                if (lane == 0) x[i] = v;
                __syncwarp();
            }
        }
        __syncthreads();
        for (int i = tid; i < first; i += nthr) {         // tails: at most seven elements, of the rows known now
            const int u0 = i + 1 + 8 * elems(i);
            double v[7], sum = 0.0;
#pragma unroll
            for (int u = 0; u < 7; ++u) v[u] = u0 + u < d ? R[apos(i, u0 + u)] : 0.0;
#pragma unroll
            for (int u = 0; u < 7; ++u)
                if (u0 + u < d) sum = __dadd_rn(sum, __dmul_rn(v[u], x[u0 + u]));
            rest[i] = sum;
        }
        // The products of a step, elements m >= 1: u = 8 m + q, row t - 1 - q, column t + 8 m, by warps 2, 3
        // and 5-7.
        // R is loaded two steps ahead of the products' use (four a thread; more at large d in line).
        constexpr int kAhead = 4;
        double rv[kAhead];
        const int pt = warp < 4 ? tid - 64 : tid - 96, pn = nthr - 96;
        auto entry = [&](int t, int u, int& c) {
            const int q = u & 7, mm = u >> 3, i = t - 1 - q;
            c = t + 8 * mm;
            return t >= 1 && mm >= 1 && i >= 0 && mm < elems(i) ? (long long)apos(i, c) : -1ll;
        };
        auto fetch = [&](int t) {
#pragma unroll
            for (int v = 0; v < kAhead; ++v) {
                int c;
                const long long at = entry(t, pt + v * pn, c);
                rv[v] = at >= 0 ? R[at] : 0.0;
            }
        };
        auto products = [&](int t) {
            double* pr = prod + (size_t)(t & 1) * pst;
#pragma unroll
            for (int v = 0; v < kAhead; ++v) {
                int c;
                if (entry(t, pt + v * pn, c) >= 0) pr[pt + v * pn] = __dmul_rn(rv[v], x[c]);
            }
            for (int u = pt + kAhead * pn; u < pst; u += pn) {
                int c;
                const long long at = entry(t, u, c);
                if (at >= 0) pr[u] = __dmul_rn(R[at], x[c]);
            }
        };
        if (warp >= 2 && warp != 4) fetch(d - 2);       // step d - 1 has no element m >= 1
        // warp 0's entries of a step, brought to shared memory by warp 1 a step ahead: R of the newest element
        // (lane q < 8), the row's y (8), diagonal (9), its reciprocal (10) and the row's tail (11)
        auto ahead = [&](int t) {
            const int i = t - 1 - lane;
            double v = 0.0;
            if (t >= 1) {
                if (lane < 8 && i >= 0) v = R[apos(i, t)];
                else if (lane == 8) v = R[apos(t - 1, d)];
                else if (lane == 9) v = R[apos(t - 1, t - 1)];
                else if (lane == 10) v = rinv[t - 1];
                else if (lane == 11 && t - 1 < first) v = rest[t - 1];
            }
            return v;
        };
        if (warp == 1 && lane < 12) s_ent[(d - 1) & 3][lane] = ahead(d - 1);
        __syncthreads();
        // One barrier a step, after the chain: it hands warp 0 the row's partial sums and the next step's
        // products, and the others the lanes' sums.  The newest x goes on in warp 0's registers; the others
        // use an x seven barriers after it is stored at the earliest.
        double xt = x[d - 1], en = warp == 0 ? s_ent[(d - 1) & 3][lane & 7] : 0.0;
        for (int t = d - 1; t >= 1; --t) {
            const int row = t - 1;
            const bool finish = row < first;               // the step completes row t - 1
            if (warp == 0) {
                const int i = t - 1 - lane;
                const bool on = lane < 8 && i >= 0 && i < first;
                const double* pr = prod + (size_t)(t & 1) * pst + (lane & 7);
                const int M = on ? elems(i) : 0;
                const int M0 = (d - t) >> 3;               // lane 0's elements; the others have as many or one more
                double c = plus_zero(__dmul_rn(en, xt));
#pragma unroll 8
                for (int m = 1; m < M0; ++m) c = __dadd_rn(c, pr[8 * m]);
                if (M0 >= 1 && M > M0) c = __dadd_rn(c, pr[8 * M0]);
                if (on && M > 0 && lane > 0) s_ls[i & 15][lane] = c;
                __syncthreads();
                const double* et = s_ent[t & 3];
                en = s_ent[(t - 1) & 3][lane & 7];
                if (finish) {
                    const double* pa = s_part[t & 1];
                    double v = __dadd_rn(__dadd_rn(c, s_ls[row & 15][2]), pa[0]);
                    v = __dadd_rn(plus_zero(v), pa[1]);
                    v = __dadd_rn(v, et[11]);
                    v = div_by(__dsub_rn(et[8], v), et[9], et[10]);
                    if (lane == 0) x[row] = v;
                    xt = __shfl_sync(0xffffffffu, v, 0);
                } else {
                    xt = x[row];
                }
            } else {
                if (warp == 1) {
                    const double nx = ahead(t - 1);
                    if (finish) {
                        const double* c = s_ls[row & 15];
                        const double p0 = __dadd_rn(c[1], c[3]);
                        const double p1 = __dadd_rn(__dadd_rn(c[4], c[6]), __dadd_rn(c[5], c[7]));
                        if (lane == 0) {
                            s_part[t & 1][0] = p0;
                            s_part[t & 1][1] = p1;
                        }
                    }
                    if (lane < 12) s_ent[(t - 1) & 3][lane] = nx;
                } else if (warp != 4) {
                    products(t - 1);
                    fetch(t - 2);
                }
                __syncthreads();
            }
        }
        __syncthreads();
        for (int i = tid; i < d; i += nthr) {
            const double dxi = x[i];
            if (dxout) dxout[i] = dxi;
            if (xupd) xupd[i] = __dsub_rn(xupd[i], dxi);
        }
        if (record && tid == 0) {
            const int r = *P.round_ctr;
            if (r < P.hist_cap) P.hist[r] = P.stats[0];
            *P.round_ctr = r + 1;
        }
        if (P.ls && tid == 0) P.ls[4] = 1.0;
    }
    gs.finish();
    return;
timeout:
    if (bid == 0 && threadIdx.x == 0) {
        *P.status = -5;
        if (record) *P.round_ctr += 1;
    }
}

}  // namespace fednl
