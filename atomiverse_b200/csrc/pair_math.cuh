// pair_math.cuh -- numerics shared by the pair kernels (pair.cu and
// pair_general.cu): approximate FP32 special functions, this library's FP64
// exp and reciprocal, the erfcx polynomial, per-row constants and sums, and
// the fixed-point flush of energies and virials.
#pragma once

#include "atvb_common.cuh"
#include "atvb_kernels.cuh"
#include "erfcx_coef.h"

namespace atvb {

constexpr double kMinPair2 = 1e-20; // lj_kernel.cuh:15 kMinPairDist^2

struct PairAcc {
    double fx, fy, fz, elj, ec;
    double v[6];
};

// ---- approximate FP32 special functions (PTX .approx instructions) -------
ATVB_DEV float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
ATVB_DEV float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
ATVB_DEV float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// exp(-z) for z >= 0 in FP64, table-driven (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15 (1989) 144-157): n = rint(-z 64/ln2), r =
// -z - n ln2/64 (ln2/64 split into a head whose products with n are exact
// and a tail), |r| <= ln2/128, and exp(-z) = 2^(n div 64) 2^((n mod 64)/64)
// exp(r) with 2^(j/64) from a 64-entry table and exp(r) by its Taylor
// series to degree 5 (truncation < 4e-17).  z is clamped at 708 (the result
// is then ~1e-308, far below anything the callers keep).
// exp(w) for -708 <= w <= 0, no clamp (the pair kernels' arguments
// -alpha^2 r^2 stay above -(alpha rlist)^2 >= -676, checked at setup)
ATVB_DEV double exp_neg64_small(double w) {
    const double n = rint(w * kExp64ByLn2);
    double r = fma(-n, kExpLn2By64Hi, w);
    r = fma(-n, kExpLn2By64Lo, r);
    double p = 1.0 / 120.0;
    p = fma(p, r, 1.0 / 24.0);
    p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    const int ni = (int)n;
    const double t = __ldg(kExp2Tab + (ni & 63));
    const long long e = (long long)((ni >> 6) + 1023) << 52; // ni >> 6 >= -1022
    return (t * p) * __longlong_as_double(e);
}

ATVB_DEV double exp_neg64(double z) { return exp_neg64_small(-fmin(z, 708.0)); }

// 1 / v for 1 <= v <= 4 in FP64: FP32 estimate, two Newton steps
// (relative error 2^-22 -> 2^-44 -> below one FP64 ulp).
ATVB_DEV double rcp64(double v) {
    double t = (double)rcp_approx((float)v);
    t = fma(t, fma(-v, t, 1.0), t);
    return fma(t, fma(-v, t, 1.0), t);
}

// 1 / sqrt(v) in FP64 for v in the FP32 normal range: FP32 estimate
// (rsqrt.approx), then two Newton steps y <- y (3/2 - (v/2) y^2) (relative
// error 2^-22 -> 2^-45 -> rounding level).
ATVB_DEV double rsqrt64(double v) {
    double y = (double)rsqrt_approx((float)v);
    const double h = 0.5 * v;
    y = y * fma(-h, y * y, 1.5);
    return y * fma(-h, y * y, 1.5);
}

// erfcx(x) for 0 <= x <= 6 from the universal polynomial of erfcx_coef.h,
// given t = 1 / (1 + kErfcxP x).  Coefficients are compile-time constants.
// FP64: the even and odd coefficients as two Horner chains in u^2 (half
// the dependency depth of one chain, one more operation), p = E + u O
ATVB_DEV double erfcx_of_t(double t) {
    const double u = fma(kErfcxA, t, kErfcxB);
    const double v = u * u;
    constexpr int NE = (kErfcxD_N + 1) / 2, NO = kErfcxD_N / 2;
    double e = kErfcxD[2 * (NE - 1)];
    double o = kErfcxD[2 * (NO - 1) + 1];
#pragma unroll
    for (int k = NE - 2; k >= 0; --k)
        e = fma(e, v, kErfcxD[2 * k]);
#pragma unroll
    for (int k = NO - 2; k >= 0; --k)
        o = fma(o, v, kErfcxD[2 * k + 1]);
    return fma(u, o, e);
}
// the short-range FP64 set (systems with alpha * cutoff <= kErfcxSXmax):
// t = 1 / (1 + kErfcxSP x), five fewer terms
ATVB_DEV double erfcx_short_of_t(double t) {
    const double u = fma(kErfcxSA, t, kErfcxSB);
    const double v = u * u;
    constexpr int NE = (kErfcxS_N + 1) / 2, NO = kErfcxS_N / 2;
    double e = kErfcxS[2 * (NE - 1)];
    double o = kErfcxS[2 * (NO - 1) + 1];
#pragma unroll
    for (int k = NE - 2; k >= 0; --k)
        e = fma(e, v, kErfcxS[2 * k]);
#pragma unroll
    for (int k = NO - 2; k >= 0; --k)
        o = fma(o, v, kErfcxS[2 * k + 1]);
    return fma(u, o, e);
}
ATVB_DEV float erfcx_of_t(float t) {
    const float u = fmaf((float)kErfcxA, t, (float)kErfcxB);
    float p = kErfcxF[kErfcxF_N - 1];
#pragma unroll
    for (int k = kErfcxF_N - 2; k >= 0; --k)
        p = fmaf(p, u, kErfcxF[k]);
    return p;
}

// Per-row constants of one system, hoisted out of the pair loop.
template <typename T>
struct RowConst {
    // shifted LJ with folded constants (r6 = 1/r^6): F/r = r6 (lj1 r6 - lj2) / r^2,
    // E = r6 (lj3 r6 - lj4) - shift; lj1 = 48 eps sigma^12, lj2 = 24 eps sigma^6,
    // lj3 = 4 eps sigma^12, lj4 = 4 eps sigma^6
    T lj_rc2, lj1, lj2, lj3, lj4, shift;
    T sig6, eps4, eps24; // the unfolded form (FP32 build)
    T c_rc2, alpha, alpha2; // alpha2: alpha^2 (FP64) or alpha^2 log2(e) (FP32)
    T kqi;
    T band_lj, band_c; // FP32 only: error band of r^2 around each cutoff
};

template <typename T>
struct RowSums {
    T fx = 0, fy = 0, fz = 0, elj = 0, ec = 0;
    T v[6] = {0, 0, 0, 0, 0, 0};
    // mixed build: force components summed in 64-bit fixed point, units of
    // kForceFix^-1 eV/A (range +-2e9 eV/A), so the row sum is exact and
    // independent of summation order
    long long fq[3] = {0, 0, 0};
    // mixed build: the row's smallest r^2 (a pair closer than
    // SysParams::force_r2_safe may carry a force beyond the fixed point)
    T rmin = T(1e30);
};
constexpr float kForceFix = 4294967296.0f;  // 2^32
constexpr double kForceFixInv = 1.0 / 4294967296.0;

template <typename T>
ATVB_DEV void finish_row(const RowSums<T>& r, PairAcc& a, bool vir) {
    if constexpr (sizeof(T) == 4) {
        // multiples of 2^-32 below 2^21 in magnitude: every later FP64 sum of
        // the lanes' values is exact, so the force is order-independent
        a.fx = (double)r.fq[0] * kForceFixInv;
        a.fy = (double)r.fq[1] * kForceFixInv;
        a.fz = (double)r.fq[2] * kForceFixInv;
    } else {
        a.fx = (double)r.fx;
        a.fy = (double)r.fy;
        a.fz = (double)r.fz;
    }
    a.elj = (double)r.elj;
    a.ec = (double)r.ec;
    if (vir)
        for (int k = 0; k < 6; ++k)
            a.v[k] = (double)r.v[k];
}

// What a block reads of a system, once per system it works on (a row of 78
// entries shared by four lanes spent a quarter of its loads on SysParams);
// the mixed rows use the pointers only.
template <typename T>
struct PairSys {
    using Pos = typename std::conditional<sizeof(T) == 4, int4, double4>::type;
    const Pos* pos;
    const int* nbr;
    const int* nnbr;
    double4* f4;
    int n, cap;
    bool lj, co, vir;
    T step[3]; // length of one fixed-point position step per axis
    RowConst<T> c;
};

template <typename T>
ATVB_DEV RowConst<T> row_const(const SysParams& P, double qi) {
    RowConst<T> c;
    c.lj_rc2 = (T)P.lj_rc2;
    c.lj1 = (T)(2.0 * P.lj_eps24 * P.lj_sig6 * P.lj_sig6);
    c.lj2 = (T)(P.lj_eps24 * P.lj_sig6);
    c.lj3 = (T)(P.lj_eps4 * P.lj_sig6 * P.lj_sig6);
    c.lj4 = (T)(P.lj_eps4 * P.lj_sig6);
    c.shift = (T)P.lj_shift;
    c.sig6 = (T)P.lj_sig6;
    c.eps4 = (T)P.lj_eps4;
    c.eps24 = (T)P.lj_eps24;
    c.c_rc2 = (T)P.coul_rc2;
    c.alpha = (T)P.coul_alpha;
    c.alpha2 = sizeof(T) == 4 ? (T)(P.coul_alpha2 * 1.4426950408889634) : (T)P.coul_alpha2;
    c.kqi = (T)(kQqr2e * qi);
    c.band_lj = (T)P.mix_band_lj;
    c.band_c = (T)P.mix_band_c;
    return c;
}

template <typename T>
ATVB_DEV PairSys<T> pair_sys(const SysParams& P) {
    PairSys<T> S;
    S.pos = reinterpret_cast<const typename PairSys<T>::Pos*>(P.pos4);
    S.nbr = P.nbr;
    S.nnbr = P.nnbr;
    S.f4 = P.f4;
    S.n = P.n;
    S.cap = P.cap;
    S.lj = P.has_lj;
    S.co = P.has_coul;
    S.vir = P.need_virial;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        S.step[d] = sizeof(T) == 4 ? (T)P.Lf_fix[d] : (T)P.Lfix64[d];
    S.c = row_const<T>(P, 0.0);
    return S;
}

// Energies and virials of a block: each lane rounds its share of a row to
// fixed point on its own, in two words (2^-32 eV, and the rest in 2^-63 eV),
// and adds them to its own columns of shared memory, so a system's sums
// depend neither on the order nor on which other systems share the launch;
// the columns go to the system once per block and system.  (A block sum per
// item cost two barriers and up to 80 shuffles per 64 atoms.)
// The columns are dynamic shared memory, `sums` of them (2, or all kPairSums
// if a system of the launch needs its virial): what they take is L1 the
// gathers do not have.
// No word can wrap: a share of 256 eV or more goes to the system straight
// away, what it has above 2^32 of the accumulator's units in the high word,
// and a block's sum of 2^18 eV or more is split the same way, so that of
// 2^12 blocks and 2^32 shares the accumulator receives less than 2^63.
struct EnergyCols {
    long long* v; // [sum][word][thread]
    int sums;
    ATVB_DEV long long& at(int k, int word) const {
        return v[(2 * k + word) * kPairBlock + threadIdx.x];
    }
};
constexpr double kShareFix = 0.5 * kEFix; // 1/2: every pair is visited from both of its atoms
constexpr int kShareWide = 0x40800000;    // high word of 512.0: a share of 256 eV
constexpr long long kBlockWide = 1125899906842624; // 2^50

// v into this lane's column of sum k: the first of a system stores.
ATVB_DEV void energy_add1(const EnergyCols& e, int k, double v, bool first) {
    const double t = v * kShareFix;
    const long long h = __double2ll_rn(t);
    const long long l = __double2ll_rn((t - (double)h) * kAccLoScale);
    e.at(k, 0) = first ? h : e.at(k, 0) + h;
    e.at(k, 1) = first ? l : e.at(k, 1) + l;
}

ATVB_DEV int share_size(double v) { return __double2hiint(v) & 0x7fffffff; }

// A share v of sum k that energy_add1 has added, if it is wide (256 eV or more
// in size, or not a number: atoms that nearly coincide): out of the column
// again and straight to the system.  Shares are cut off where the sum of as
// many as the system can have would leave the high word (2^37 eV in a million
// atoms); not a number counts as the largest.
ATVB_DEV void energy_wide(const EnergyCols& e, const SysParams& P, int k, double v) {
    if (share_size(v) < kShareWide)
        return;
    const double t = v * kShareFix;
    const long long h0 = __double2ll_rn(t);
    e.at(k, 0) -= h0;
    e.at(k, 1) -= __double2ll_rn((t - (double)h0) * kAccLoScale);
    // 2^57 over the next power of two of the atoms (32 shares each): no division
    const double most = __hiloint2double((1023 + 57 - (32 - __clz(P.n))) << 20, 0);
    double a = fmin(fabs(t) * (1.0 / kAccHiScale), most);
    a = t < 0.0 ? -a : a;
    const double hi = floor(a);
    const double r = (a - hi) * kAccHiScale; // exact
    const long long h = __double2ll_rn(r);
    const long long l = __double2ll_rn((r - (double)h) * kAccLoScale);
    red_add_u64(&P.st->acc[pair_acc(k)], (unsigned long long)h);
    red_add_u64(P.acc_ext + k, (unsigned long long)l);
    red_add_u64(P.acc_ext + kPairSums + k, (unsigned long long)(long long)hi);
}

// The row share of every lane of the block (zeros past the last atom).
// The LJ and Coulomb sums unconditionally: skipping one the system has not
// made the mixed kernel spill (347 -> 361 us at 262,144 ions).  One test for
// wide shares, after the columns, and no call behind it (a division is one,
// too): 1,000,188 LJ atoms with virial 408 us a launch without it, 406 so, 423
// with a test before each column and a call; 108,000 atoms of a mixture 92.0,
// 92.2 and 98; steps of 13,500 of them 45.3, 45.6 and, with one test and a
// call, 48.6 us; of 256 LJ atoms 16.7 and 16.9.
ATVB_DEV void energy_add(const EnergyCols& e, const SysParams& P, const PairAcc& a, bool vir,
                         bool first) {
    vir = vir && e.sums == kPairSums;
    int size = max(share_size(a.elj), share_size(a.ec));
    energy_add1(e, 0, a.elj, first);
    energy_add1(e, 1, a.ec, first);
    if (vir)
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            size = max(size, share_size(a.v[k]));
            energy_add1(e, 2 + k, a.v[k], first);
        }
    if (size >= kShareWide) {
        energy_wide(e, P, 0, a.elj);
        energy_wide(e, P, 1, a.ec);
        if (vir)
#pragma unroll
            for (int k = 0; k < 6; ++k)
                energy_wide(e, P, 2 + k, a.v[k]);
    }
}

// Block-uniform.  `again`: the block goes on to another system.
ATVB_DEV void energy_flush(const EnergyCols& e, const SysParams& P, bool again) {
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    static_assert(kPairBlock / 32 >= kPairSums, "a warp per sum");
    if (w < (P.need_virial ? e.sums : 2)) {
        long long h = 0, l = 0;
#pragma unroll
        for (int k = 0; k < kPairBlock / 32; ++k) {
            h += e.v[2 * w * kPairBlock + k * 32 + lane];
            l += e.v[(2 * w + 1) * kPairBlock + k * 32 + lane];
        }
        h = warp_sum(h);
        l = warp_sum(l);
        if (lane == 0) {
            if (h >= kBlockWide || h <= -kBlockWide) {
                red_add_u64(P.acc_ext + kPairSums + w, (unsigned long long)(h >> 32));
                h &= 0xffffffffll;
            }
            if (h)
                red_add_u64(&P.st->acc[pair_acc(w)], (unsigned long long)h);
            if (l)
                red_add_u64(P.acc_ext + w, (unsigned long long)l);
        }
    }
    if (again)
        __syncthreads();
}

// Mixed: at least 3 resident blocks (80 registers); FP64: 2.
} // namespace atvb
