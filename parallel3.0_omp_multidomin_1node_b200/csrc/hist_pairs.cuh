// History blocks of a (source, field element) pair for all steps k at once
// (included by assemble.cu): ComputeT2Block / T1Block / UBlock,
// DBEM1/multidomain.cpp:1739-1813, over the rules of quad.cuh.
//
// What bounds it: FP64 arithmetic.  Evaluating the point kernels per step (one
// launch per k, each point's geometry, distance powers and tensors computed
// again with about twenty divisions) took 707 ms on a 2,058-element bar.  But a
// quadrature point's part in step m is
//   U   = alpha q + beta I,   T = A q + B n (x) R + C (R (x) n + (R.n) I),
// q = R (x) R, with factors alpha .. C that alone depend on m, and it is nonzero
// only while the point's waves pass: m from n1 (the P front, floor(r / C1 Dt)) to
// n2 (the S front).  So a warp computes each point's distance and fronts once
// per pair, and a step costs a point its factors and some 70 multiply-adds.
// Field elements' points are tabulated per CTA, which takes one field element
// and a range of sources.
#pragma once

#include "quad.cuh"

namespace tdbem {
namespace {

constexpr int kPairWarps = 8, kPairSources = 64;  // warps and sources per CTA
constexpr int kPwPoints = kNumPW2 * 9, kRegPoints = 16, kPairPoints = kPwPoints + kRegPoints;

// A field element's quadrature points: patch-wise rule, then regular rule.
struct PairTable {
    double x[3][kPairPoints], n[3][kPairPoints], w[kPairPoints];
};

// Per warp: the points' distances from the pair's source, fronts (n1, n2) and
// steps in which they count (first, last: patches are skipped outside their
// windows), and the sums of a step.
template <class S>
struct PairWarp {
    double r[kPairPoints], ir[kPairPoints];
    short4 span[kPairPoints];  // n1, n2, first, last
    short2 patch[kNumPW2];
    S sum[32];                 // T1 (9), T2 of the next step (9), U (6: 00 01 02 11 12 22)
    S t2[9], reg[9], regu[6];  // T2 carried from the step before; regular rule: T1 + T2, U
    S out[18];                 // stored blocks, for readers of all nine values
};

__device__ __forceinline__ void fill_table(PairTable& tb, const QuadRules& q, const double* cc)
{
    for (int it = threadIdx.x; it < kPairPoints; it += blockDim.x) {
        double s1, s2, wt;
        if (it < kPwPoints) {
            const int p = it / 9, j = it - 9 * p;
            s1 = q.lpospw[p][j][0];
            s2 = q.lpospw[p][j][1];
            wt = q.pwgv[p][j];
        } else {
            s1 = q.rp[it - kPwPoints][0];
            s2 = q.rp[it - kPwPoints][1];
            wt = q.nrgv0[it - kPwPoints];
        }
        double pt[3], nor[3], jac;
        q_from_local(cc, s1, s2, pt);
        q_normal_jacobi(cc, s1, s2, nor, &jac);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            tb.x[c][it] = pt[c];
            tb.n[c][it] = nor[c];
        }
        tb.w[it] = wt * jac;
    }
}

// The n with n dt <= t < n dt + dt (the wave-front indicator Fai's condition,
// q_fai), clamped to what the step loop can reach.
__device__ __forceinline__ int front_step(double t, double dt)
{
    if (!(t < 30000.0 * dt)) return 30000;
    int n = (int)(t / dt);
    while (n > 0 && t < n * dt) --n;
    while (t >= n * dt + dt) ++n;
    return n;
}

// Wave-front classification of (field element, source point) for time index m: 0
// skip, 1 patch-wise rule, 2 regular rule (NeedCal,
// DBEM1/dsquareelement.cpp:1156-1201), with its distances taken once.
struct PairClass {
    double a1, a2, b1, b2, dt;
    template <class MT>
    __device__ __forceinline__ PairClass(const MT& M, const double* center, double radius, const double* src)
    {
        const double r = q_dist(center, src), rmax = r + radius;
        double rmin = r - radius;
        if (rmin < 0.0) rmin = 0.0;
        a1 = rmax / qv(M.C1);
        a2 = rmax / qv(M.C2);
        b1 = rmin / qv(M.C1);
        b2 = rmin / qv(M.C2);
        dt = M.Dt;
    }
    __device__ __forceinline__ int operator()(int m) const
    {
        const double ndt = m * dt, np1dt = (m + 1) * dt;
        if (ndt >= a2 || np1dt <= b1) return 0;
        if (ndt <= b1 && (np1dt >= a1 && np1dt <= b2)) return 2;
        if (ndt <= b1 && np1dt >= a2) return 2;
        if (ndt >= a1 && np1dt <= b2) return 2;
        if ((ndt >= a1 && ndt <= b2) && np1dt >= a2) return 2;
        return 1;
    }
};

// Factors of a point at step m: T1(m) and T2(m + 1) (evaluated at m) as A, B, C;
// U(m) as alpha, beta.  q_dyna_u and q_dyna_t, gathered by tensor.
template <class S>
struct PointFactors {
    S a1, b1, c1, a2, b2, c2, al, be;
};
template <class MT, class S = typename MT::Scalar>
__device__ __forceinline__ PointFactors<S> point_factors(const MT& M, int m, int n1, int n2, double r, double ir, double rn)
{
    PointFactors<S> f{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double n = m, ndt = n * M.Dt, np1dt = ndt + M.Dt;
    const double ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2, k4 = kOneOver4Pi;
    const double t2 = k4 / M.Dt;
    const S k0 = M.OneOverFourPaiRou;
    if (m == n1) {
        const double c1 = (4.0 * M.C2_2OverC1_2 - 1.0) * ir3, c2 = M.C2_2OverC1_2 * 12.0 * rn * ir5,
                     c3 = M.C2_2OverC1_2 * 2.0 * ir3;
        const S g1 = M.C2_2OverC1_3 * (-2.0 * rn * ir2 * ir2), g2 = 1.0 / M.C1 * ((2.0 * M.C2_2OverC1_2 - 1.0) * ir2);
        const S x = r / M.C1Dt, t = k4 * ((n + 1.0) - x), u = k4 * (x - n);
        f.a1 += t * (-c2) + g1 * t2;
        f.b1 += t * c1 + g2 * t2;
        f.c1 += t * c3;
        f.a2 += u * (-c2) - g1 * t2;
        f.b2 += u * c1 - g2 * t2;
        f.c2 += u * c3;
        f.al += M.OneOverC1_2 * k0 * ir3;
    }
    if (m == n2) {
        const double e1 = 12.0 * rn * ir5, e2 = 2.0 * ir3, e3 = 3.0 * ir3;
        const S ic2 = 1.0 / M.C2, h1 = ic2 * (2.0 * rn * ir2 * ir2), h2 = ic2 * (-ir2);
        const S x = r / M.C2Dt, t = k4 * ((n + 1.0) - x), u = k4 * (x - n);
        f.a1 += t * e1 + h1 * t2;
        f.b1 += t * (-e2);
        f.c1 += t * (-e3) + h2 * t2;
        f.a2 += u * e1 - h1 * t2;
        f.b2 += u * (-e2);
        f.c2 += u * (-e3) - h2 * t2;
        const S c = M.OneOverC2_2 * k0;
        f.al += c * (-ir3);
        f.be += c * ir;
    }
    S ri, rj;
    if (m > n1 && m < n2) {
        ri = (n + 0.5) * M.Dt_2 * ir2;
        rj = (n * n + n + 0.33333333333333333) * (M.Dt_3 * ir3);
    } else if (m == n1 && m < n2) {
        const double t = np1dt * ir;
        ri = 0.5 * (t * t - M.OneOverC1_2);
        rj = 0.33333333333333 * (t * t * t - M.OneOverC1_3);
    } else if (m == n1) {
        ri = M.Half_1OC22_1OC12;
        rj = M.Third_1OC23_1OC13;
    } else {
        const double t = ndt * ir;
        ri = 0.5 * (M.OneOverC2_2 - t * t);
        rj = 0.333333333333333 * (M.OneOverC2_3 - t * t * t);
    }
    const S rjt = rj * (r / M.Dt), t = k4 * (ri * (n + 1.0) - rjt), u = k4 * (rjt - ri * n);
    const S f1 = M.C2_2 * -6.0;
    const S ft = f1 * t, fu = f1 * u;
    const double f2 = 5.0 * rn * ir5;
    f.a1 += ft * f2;
    f.b1 += ft * (-ir3);
    f.c1 += ft * (-ir3);
    f.a2 += fu * f2;
    f.b2 += fu * (-ir3);
    f.c2 += fu * (-ir3);
    const S kr = k0 * ri;
    f.al += kr * (3.0 * ir3);
    f.be += kr * (-ir);
    return f;
}

// v += w (A q + B n (x) R + C (R (x) n + (R.n) I)), row-major
template <class S>
__device__ __forceinline__ void add_traction(S (&v)[32], int at, const double* R, const double* N, double rn, S a, S b, S c,
                                             double w)
{
    a = a * w;
    b = b * w;
    c = c * w;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            v[at + 3 * i + j] += a * (R[i] * R[j]) + b * (R[j] * N[i]) + c * (i == j ? R[i] * N[j] + rn : R[i] * N[j]);
}
template <class S>
__device__ __forceinline__ void add_displacement(S (&v)[32], int at, const double* R, S al, S be, double w)
{
    al = al * w;
    be = be * w;
    v[at] += al * (R[0] * R[0]) + be;
    v[at + 1] += al * (R[0] * R[1]);
    v[at + 2] += al * (R[0] * R[2]);
    v[at + 3] += al * (R[1] * R[1]) + be;
    v[at + 4] += al * (R[1] * R[2]);
    v[at + 5] += al * (R[2] * R[2]) + be;
}

__device__ __forceinline__ double lane_swap(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ QDual lane_swap(const QDual& v, int o) { return {lane_swap(v.v, o), lane_swap(v.e, o)}; }

// The warp's sums of v[0..n): lane l returns that of v[l] (l < 32).  Each
// exchange halves what a lane keeps: 31 shuffles for up to 32 values.
template <class S>
__device__ __forceinline__ S warp_sums(S (&v)[32], int lane)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i >= o) break;
            const S send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + lane_swap(send, o);
        }
    }
    return v[0];
}

// Walks the steps m = ka - 1 .. kb of one pair; for every k = m >= ka calls
// block(k, c2, c1, t2, t1, u): the classes of the T2 and T1 / U parts (0: none;
// c2 = 3: the singular T2 block of a self pair at k = 1, which the caller has)
// and their 9 / 9 / 6 values in shared memory, the same for the whole warp.
template <class MT, class Block, class S = typename MT::Scalar>
__device__ __forceinline__ void pair_steps(const MT& M, const PairTable& tb, PairWarp<S>& pw, const QElem& e,
                                           const double* src, bool self, int ka, int kb, Block block)
{
    const int lane = threadIdx.x & 31;
    const PairClass cls(M, e.center, e.radius, src);
    const double c1dt = qv(M.C1Dt), c2dt = qv(M.C2Dt);
    // patch windows (q_pw_need_cal): m counts unless (r - rpw) >= (m + 1) C1 Dt or
    // (r + rpw) < m C2 Dt
    for (int p = lane; p < kNumPW2; p += 32) {
        const double r = q_dist(e.rcen + 3 * p, src), a = r - e.rpw, b = r + e.rpw;
        int f = a > 0.0 ? min((int)(a / c1dt), 30000) : 0, l = b > 0.0 ? min((int)(b / c2dt), 30000) : -1;
        while (f > 0 && !(a >= f * c1dt)) --f;
        while (f < 30000 && a >= (f + 1) * c1dt) ++f;
        while (l >= 0 && b < l * c2dt) --l;
        while (l < 30000 && !(b < (l + 1) * c2dt)) ++l;
        pw.patch[p] = make_short2((short)f, (short)l);
    }
    __syncwarp();
    for (int it = lane; it < kPairPoints; it += 32) {
        const double dx = tb.x[0][it] - src[0], dy = tb.x[1][it] - src[1], dz = tb.x[2][it] - src[2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        const int n1 = front_step(r / qv(M.C1), M.Dt), n2 = front_step(r / qv(M.C2), M.Dt);
        int f = n1, l = n2;
        if (it < kPwPoints) {
            const short2 w = pw.patch[it / 9];
            f = max(f, (int)w.x);
            l = min(l, (int)w.y);
        }
        pw.r[it] = r;
        pw.ir[it] = 1.0 / r;
        pw.span[it] = make_short4((short)n1, (short)n2, (short)f, (short)l);
    }
    __syncwarp();
    int before = 0;  // class of m - 1
#pragma unroll 1
    for (int m = ka - 1; m <= kb; ++m) {
        const int now = cls(m);
        if (now == 1) {
            S v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.0;
#pragma unroll 1
            for (int it = lane; it < kPwPoints; it += 32) {
                const short4 sp = pw.span[it];
                if (m < sp.z || m > sp.w) continue;
                const double R[3] = {tb.x[0][it] - src[0], tb.x[1][it] - src[1], tb.x[2][it] - src[2]};
                const double N[3] = {tb.n[0][it], tb.n[1][it], tb.n[2][it]}, w = tb.w[it];
                const double rn = R[0] * N[0] + R[1] * N[1] + R[2] * N[2];
                const PointFactors<S> f = point_factors(M, m, sp.x, sp.y, pw.r[it], pw.ir[it], rn);
                add_traction<S>(v, 0, R, N, rn, f.a1, f.b1, f.c1, w);
                add_traction<S>(v, 9, R, N, rn, f.a2, f.b2, f.c2, w);
                add_displacement<S>(v, 18, R, f.al, f.be, w);
            }
            const S t = warp_sums<S>(v, lane);
            if (lane < 24) pw.sum[lane] = t;
        }
        const bool self_k = self && m == 1;
        if (m >= ka && (now == 2 || (before == 2 && !self_k))) {
            // regular rule: T1(m) + T2(m) at every point, whatever the block's
            // type (IntDynaTij(typeT, ..., T_ID), DBEM1/dsquareelement.cpp:2233-2290)
            S v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.0;
            if (lane < kRegPoints) {
                const int it = kPwPoints + lane;
                const short4 sp = pw.span[it];
                const double R[3] = {tb.x[0][it] - src[0], tb.x[1][it] - src[1], tb.x[2][it] - src[2]};
                const double N[3] = {tb.n[0][it], tb.n[1][it], tb.n[2][it]}, w = tb.w[it];
                const double rn = R[0] * N[0] + R[1] * N[1] + R[2] * N[2];
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const int mm = m - h;
                    if (mm < sp.x || mm > sp.y) continue;
                    const PointFactors<S> f = point_factors(M, mm, sp.x, sp.y, pw.r[it], pw.ir[it], rn);
                    add_traction<S>(v, 0, R, N, rn, h ? f.a2 : f.a1, h ? f.b2 : f.b1, h ? f.c2 : f.c1, w);
                    if (h == 0) add_displacement<S>(v, 9, R, f.al, f.be, w);
                }
            }
            const S t = warp_sums<S>(v, lane);
            if (lane < 9) pw.reg[lane] = t;
            else if (lane < 15) pw.regu[lane - 9] = t;
        }
        __syncwarp();
        if (m >= ka) {
            const int c2 = self_k ? 3 : before;
            block(m, c2, now, c2 == 2 ? pw.reg : pw.t2, now == 2 ? pw.reg : pw.sum, now == 2 ? pw.regu : pw.sum + 18);
            __syncwarp();
        }
        if (now == 1 && lane < 9) pw.t2[lane] = pw.sum[9 + lane];
        before = now;
        __syncwarp();
    }
}

// 3x3 index of a U value among its six
__device__ __forceinline__ int sym6(int i) { return i < 3 ? i : i == 3 ? 1 : i == 4 ? 3 : i == 5 ? 4 : i == 6 ? 2 : i == 7 ? 4 : 5; }

// The stored blocks of step k of a pair from its values (history_pair's
// builder rules, DBEM1/multidomain.cpp:1120-1144, decided on the values): lane l
// < 9 returns its element of MTS (T2, then T1 accumulated) and MGS, transposed
// and signed; flags bit0 MTS, bit1 MGS.
template <class S>
__device__ __forceinline__ int stored_blocks(int lane, int c2, int c1, const S* t2, const S* t1, const S* u, double su,
                                             double st, S& mts, S& mgs)
{
    const int l = lane < 9 ? lane : 0, tr = (l % 3) * 3 + l / 3;
    const unsigned nine = 0x1FFu;
    // all-zero, near-zero (<= 1e-14) and non-finite blocks are skipped
    auto admitted = [&](const S& b) {
        const double v = fabs(qv(b));
        const unsigned big = __ballot_sync(0xffffffffu, v > 1.0e-14), bad = __ballot_sync(0xffffffffu, !(v <= 1.7976931348623157e308));
        return (big & nine) != 0 && (bad & nine) == 0;
    };
    auto above = [&](const S& b) { return (__ballot_sync(0xffffffffu, fabs(qv(b)) > 1.0e-14) & nine) != 0; };
    int fl = 0;
    mts = 0.0;
    mgs = 0.0;
    bool present = false;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const S b = part == 0 ? t2[tr] : t1[tr];
        if ((part == 0 ? c2 : c1) != 0 && su != 0.0 && admitted(b)) {
            mts += su * b;
            present = true;
            if (!above(mts)) {
                present = false;
                mts = 0.0;
            }
        }
    }
    if (present) fl |= 1;
    if (c1) {
        const S b = u[sym6(tr)];
        if (st != 0.0 && admitted(b)) {
            mgs = st * b;
            if (above(mgs)) fl |= 2;
        }
    }
    return fl;
}

}  // namespace
}  // namespace tdbem
