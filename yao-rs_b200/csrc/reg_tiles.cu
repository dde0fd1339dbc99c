// reg_tiles.cu — register passes (see reg_tiles.h): the planner that cuts a
// program of 1- and 2-qubit gates into passes and segments, and the kernel.
//
// A pass reads each 2^tbits-amplitude tile once, applies its ops and writes
// it back.  Each thread owns 2^RB amplitudes that differ in the segment's RB
// tile positions and applies all ops of the segment in registers; between
// segments the tile changes hands through shared memory (one barrier).
//
// What bounds it: issue.  A rotation of 16 amplitudes is 192 cycles a warp on
// the FP64 pipe (complex64: packed FP32), with about as many instructions for
// its description, coefficients, signs and the segment's addresses around it,
// and three warps a scheduler to overlap their latencies: the FP64 pipe is
// busy 55% of the time.  So ops are few and large: a rotation carries the
// phase before it and the CZ signs around it (561 ops for the 1950 gates of
// the layered circuit, n = 28, 20 layers), four of them share one diagonal
// for phases and signs and one way through the op loop, and 16 amplitudes a
// thread share each op's fixed cost.  Against the block passes of sv_tiles.cu
// on that circuit, kernel time: complex128 FUSED 185 -> 94 ms (105 without the
// layers of four and the kept places), complex64 FUSED 222 -> 91 ms (111);
// TILED at n = 25, 8 layers (no multiplication of gates, no FMA) 62.7 -> 23 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "reg_tiles.h"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace yao {

// ================================================================== device

struct RHdr {
    int32_t tbits, nsegs, blob16, nbuf;  // blob16: 16-byte words of the description
    int32_t ops16, coef16;               // first 16-byte word of the ops and of the coefficients
    int32_t use_tma, pad;
    uint32_t ntiles, pad2;
    int8_t tb[16];
    TmaPlan tma;
};

// Arithmetic on one amplitude type.  complex128: EXACT is num_complex's
// operations without FMA, else FMA.  complex64: coefficients split into
// high and low FP32 parts, each stored twice so that one packed FP32x2 FMA
// handles both components; the small low products are summed first.
template <bool EXACT>
struct A128 {
    typedef double2 Amp;
    static constexpr int kCoef16 = 1;  // 16-byte words a complex coefficient
    struct Coef {
        double2 c;
    };
    static __device__ __forceinline__ Coef load(const uint4* p) { return Coef{*(const double2*)p}; }
    static __device__ __forceinline__ bool is_one(const Coef& k) { return k.c.x == 1.0 && k.c.y == 0.0; }
    static __device__ __forceinline__ Amp mul(const Coef& k, Amp x) {
        if (EXACT) return cmulassign_x(x, k.c);
        return make_double2(fma(k.c.x, x.x, -k.c.y * x.y), fma(k.c.x, x.y, k.c.y * x.x));
    }
    static __device__ __forceinline__ Amp mad(Amp acc, const Coef& k, Amp x) {
        if (EXACT) return cadd_x(acc, cmul_x(k.c, x));
        return make_double2(fma(k.c.x, x.x, fma(-k.c.y, x.y, acc.x)), fma(k.c.x, x.y, fma(k.c.y, x.x, acc.y)));
    }
    // a w + b x
    static __device__ __forceinline__ Amp two(const Coef& a, Amp w, const Coef& b, Amp x) {
        if (EXACT) return cadd_x(cmul_x(a.c, w), cmul_x(b.c, x));
        return mad(make_double2(fma(a.c.x, w.x, -a.c.y * w.y), fma(a.c.x, w.y, a.c.y * w.x)), b, x);
    }
    // real matrix [[a, b], [c, d]]: p = (a, b), q = (c, d)
    struct Real {
        double2 p, q;
    };
    static __device__ __forceinline__ Real load_real(const uint4* m) { return Real{*(const double2*)m, *(const double2*)(m + 1)}; }
    static __device__ __forceinline__ void real(const Real& k, Amp& w, Amp& x) {
        const Amp y = make_double2(k.q.y * x.x, k.q.y * x.y), z = make_double2(k.p.y * x.x, k.p.y * x.y);
        x = make_double2(fma(k.q.x, w.x, y.x), fma(k.q.x, w.y, y.y));
        w = make_double2(fma(k.p.x, w.x, z.x), fma(k.p.x, w.y, z.y));
    }
    // first column real: p = (a, c), then b, d
    static __device__ __forceinline__ void rcol(const double2& p, const Coef& b, const Coef& d, Amp& w, Amp& x) {
        const Amp u = mul(b, x), v = mul(d, x);
        x = make_double2(fma(p.y, w.x, v.x), fma(p.y, w.y, v.y));
        w = make_double2(fma(p.x, w.x, u.x), fma(p.x, w.y, u.y));
    }
    // first row real: p = (a, b), then c, d
    static __device__ __forceinline__ void rrow(const double2& p, const Coef& c, const Coef& d, Amp& w, Amp& x) {
        const Amp v = two(c, w, d, x);
        w = make_double2(fma(p.x, w.x, p.y * x.x), fma(p.x, w.y, p.y * x.y));
        x = v;
    }
    typedef double2 Two;  // two real coefficients
    static __device__ __forceinline__ Two load_two(const uint4* m) { return *(const double2*)m; }
    // the second column of a matrix (the second of two reals) times -1 when
    // the top bit of s is set
    static __device__ __forceinline__ double flip(double x, uint32_t s) {
        return __hiloint2double(__double2hiint(x) ^ (int)s, __double2loint(x));
    }
    static __device__ __forceinline__ Real sign_real(const Real& k, uint32_t s) {
        return Real{make_double2(k.p.x, flip(k.p.y, s)), make_double2(k.q.x, flip(k.q.y, s))};
    }
    static __device__ __forceinline__ Two sign_two(const Two& k, uint32_t s) { return make_double2(k.x, flip(k.y, s)); }
    static __device__ __forceinline__ Coef sign_coef(const Coef& k, uint32_t s) {
        return Coef{make_double2(flip(k.c.x, s), flip(k.c.y, s))};
    }
    // x times -1 when the top bit of s is set
    static __device__ __forceinline__ Amp sign(Amp x, uint32_t s) {
        return make_double2(__hiloint2double(__double2hiint(x.x) ^ (int)s, __double2loint(x.x)),
                            __hiloint2double(__double2hiint(x.y) ^ (int)s, __double2loint(x.y)));
    }
    static __device__ __forceinline__ Amp neg(Amp x) { return make_double2(-x.x, -x.y); }
    static __device__ __forceinline__ Amp zero() { return make_double2(0.0, 0.0); }
};

__device__ __forceinline__ uint64_t pk(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// i x = (-im, re)
__device__ __forceinline__ uint64_t iturn(uint64_t x) {
    float re, im;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(re), "=f"(im) : "l"(x));
    return pk(-im, re);
}

struct A64 {
    typedef uint64_t Amp;
    static constexpr int kCoef16 = 2;
    struct Coef {
        uint64_t hr, hi, lr, li;
    };
    static __device__ __forceinline__ Coef load(const uint4* p) {
        const ulonglong2 a = *(const ulonglong2*)p, b = *(const ulonglong2*)(p + 1);
        return Coef{a.x, a.y, b.x, b.y};
    }
    static __device__ __forceinline__ bool is_one(const Coef& k) {
        return k.hr == 0x3f8000003f800000ull && k.hi == 0 && k.lr == 0 && k.li == 0;
    }
    static __device__ __forceinline__ Amp mul(const Coef& k, Amp x) {
        const uint64_t t = iturn(x);
        return fma2(k.hr, x, fma2(k.hi, t, fma2(k.lr, x, mul2(k.li, t))));
    }
    static __device__ __forceinline__ Amp mad(Amp acc, const Coef& k, Amp x) {
        const uint64_t t = iturn(x);
        return fma2(k.hr, x, fma2(k.hi, t, fma2(k.lr, x, fma2(k.li, t, acc))));
    }
    static __device__ __forceinline__ Amp two(const Coef& a, Amp w, const Coef& b, Amp x) {
        const uint64_t u = iturn(w), t = iturn(x);
        const uint64_t lo = fma2(b.lr, x, fma2(b.li, t, fma2(a.lr, w, mul2(a.li, u))));
        return fma2(b.hr, x, fma2(b.hi, t, fma2(a.hr, w, fma2(a.hi, u, lo))));
    }
    struct Real {
        Coef p, q;  // hr, lr: first of the two reals; hi, li: the second
    };
    typedef Coef Two;
    static __device__ __forceinline__ Two load_two(const uint4* m) { return load(m); }
    static __device__ __forceinline__ Real load_real(const uint4* m) { return Real{load(m), load(m + 2)}; }
    static __device__ __forceinline__ void real(const Real& k, Amp& w, Amp& x) {
        const Amp y = fma2(k.q.lr, w, mul2(k.q.li, x)), z = fma2(k.p.lr, w, mul2(k.p.li, x));
        const Amp v = fma2(k.q.hr, w, fma2(k.q.hi, x, y));
        w = fma2(k.p.hr, w, fma2(k.p.hi, x, z));
        x = v;
    }
    static __device__ __forceinline__ void rcol(const Coef& p, const Coef& b, const Coef& d, Amp& w, Amp& x) {
        const uint64_t t = iturn(x);
        const Amp lu = fma2(p.lr, w, fma2(b.lr, x, mul2(b.li, t))), lv = fma2(p.li, w, fma2(d.lr, x, mul2(d.li, t)));
        const Amp v = fma2(p.hi, w, fma2(d.hr, x, fma2(d.hi, t, lv)));
        w = fma2(p.hr, w, fma2(b.hr, x, fma2(b.hi, t, lu)));
        x = v;
    }
    static __device__ __forceinline__ void rrow(const Coef& p, const Coef& c, const Coef& d, Amp& w, Amp& x) {
        const Amp v = two(c, w, d, x);
        w = fma2(p.hr, w, fma2(p.hi, x, fma2(p.lr, w, mul2(p.li, x))));
        x = v;
    }
    static __device__ __forceinline__ Amp sign(Amp x, uint32_t s) { return x ^ ((uint64_t)s << 32 | s); }
    static __device__ __forceinline__ Coef sign_coef(const Coef& k, uint32_t s) {
        return Coef{sign(k.hr, s), sign(k.hi, s), sign(k.lr, s), sign(k.li, s)};
    }
    static __device__ __forceinline__ Two sign_two(const Two& k, uint32_t s) { return Coef{k.hr, sign(k.hi, s), k.lr, sign(k.li, s)}; }
    static __device__ __forceinline__ Real sign_real(const Real& k, uint32_t s) { return Real{sign_two(k.p, s), sign_two(k.q, s)}; }
    static __device__ __forceinline__ Amp neg(Amp x) { return x ^ 0x8000000080000000ull; }
    static __device__ __forceinline__ Amp zero() { return 0; }
};

// Negates the second member of the pairs in sg (bit j: pair of amplitude j).
template <typename A, int RB, int P>
__device__ __forceinline__ void r_sign(typename A::Amp (&v)[1 << RB], uint32_t sg) {
    if (sg) {
#pragma unroll
        for (int j = 0; j < (1 << RB); j++)
            if (!(j & (1 << P))) {
                // (measured both ways: complex128 2% faster without the tests, complex64 6% with them)
                if constexpr (sizeof(typename A::Amp) == 16)
                    v[j | (1 << P)] = A::sign(v[j | (1 << P)], (sg << (31 - j)) & 0x80000000u);
                else if ((sg >> j) & 1u)
                    v[j | (1 << P)] = A::neg(v[j | (1 << P)]);
            }
    }
}

template <typename A, int RB, int P>
__device__ __forceinline__ void r_real1(typename A::Amp (&v)[1 << RB], const uint4* m, uint32_t sg, uint32_t cs) {
    const typename A::Real k = A::sign_real(A::load_real(m), cs);
    r_sign<A, RB, P>(v, sg);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++)
        if (!(j & (1 << P))) A::real(k, v[j], v[j | (1 << P)]);
}

template <typename A, int RB, int P>
__device__ __forceinline__ void r_rcol1(typename A::Amp (&v)[1 << RB], const uint4* m, uint32_t sg, uint32_t cs) {
    const typename A::Two p = A::load_two(m);
    const typename A::Coef b = A::sign_coef(A::load(m + A::kCoef16), cs), d = A::sign_coef(A::load(m + 2 * A::kCoef16), cs);
    r_sign<A, RB, P>(v, sg);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++)
        if (!(j & (1 << P))) A::rcol(p, b, d, v[j], v[j | (1 << P)]);
}

template <typename A, int RB, int P>
__device__ __forceinline__ void r_rrow1(typename A::Amp (&v)[1 << RB], const uint4* m, uint32_t sg, uint32_t cs) {
    const typename A::Two p = A::sign_two(A::load_two(m), cs);
    const typename A::Coef c = A::load(m + A::kCoef16), d = A::sign_coef(A::load(m + 2 * A::kCoef16), cs);
    r_sign<A, RB, P>(v, sg);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++)
        if (!(j & (1 << P))) A::rrow(p, c, d, v[j], v[j | (1 << P)]);
}

template <typename A, int RB, int P, bool ALL>
__device__ __forceinline__ void r_dense1(typename A::Amp (&v)[1 << RB], const uint4* m, uint32_t jm, uint32_t sg, uint32_t cs) {
    const typename A::Coef a = A::load(m), b = A::sign_coef(A::load(m + A::kCoef16), cs), c = A::load(m + 2 * A::kCoef16),
                           d = A::sign_coef(A::load(m + 3 * A::kCoef16), cs);
    r_sign<A, RB, P>(v, sg);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++) {
        if (j & (1 << P)) continue;
        if (!ALL && !((jm >> j) & 1)) continue;
        const typename A::Amp w = v[j], x = v[j | (1 << P)];
        v[j] = A::two(a, w, b, x);
        v[j | (1 << P)] = A::two(c, w, d, x);
    }
}

// (A permutation without the tests costs registers: the compiler then has
// every other op's results moved to match it.)
template <typename A, int RB, int P>
__device__ __forceinline__ void r_x(typename A::Amp (&v)[1 << RB], uint32_t jm) {
#pragma unroll
    for (int j = 0; j < (1 << RB); j++) {
        if (j & (1 << P)) continue;
        if (!((jm >> j) & 1)) continue;
        const typename A::Amp w = v[j];
        v[j] = v[j | (1 << P)];
        v[j | (1 << P)] = w;
    }
}

template <typename A, bool EXACT, int RB, int P>
__device__ __forceinline__ void r_phase1(typename A::Amp (&v)[1 << RB], const typename A::Coef& c) {
    if (EXACT && A::is_one(c)) return;
#pragma unroll
    for (int j = 0; j < (1 << RB); j++)
        if (j & (1 << P)) v[j] = A::mul(c, v[j]);
}

// Which entry of its table a thread's diagonal op takes.
__device__ __forceinline__ uint32_t r_entry(const uint4& w1, uint32_t t, uint32_t lb) {
    const int ns = (int)(w1.z >> 8);
    uint32_t e = 0;
    for (int q = 0; q < ns; q++) {
        const uint32_t p = (q < 5 ? w1.y >> (6 * q) : w1.z) & 63u;
        e |= (p < 16 ? (lb >> p) & 1u : (t >> (p - 16)) & 1u) << q;
    }
    return e;
}

template <typename A, bool EXACT, int RB, int PAIR>
__device__ __forceinline__ void r_dense2(typename A::Amp (&v)[1 << RB], const uint4* m, uint32_t jm) {
    constexpr int B0 = 1 << (2 * PAIR), B1 = 2 << (2 * PAIR);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++) {
        if (j & (B0 | B1)) continue;
        if (!((jm >> j) & 1)) continue;
        const typename A::Amp x0 = v[j], x1 = v[j | B0], x2 = v[j | B1], x3 = v[j | B0 | B1];
        typename A::Amp y[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint4* mr = m + 4 * r * A::kCoef16;
            // exact: from zero, as a gate alone does (the sign of a zero)
            const typename A::Amp s = EXACT ? A::mad(A::mad(A::zero(), A::load(mr), x0), A::load(mr + A::kCoef16), x1)
                                            : A::two(A::load(mr), x0, A::load(mr + A::kCoef16), x1);
            y[r] = A::mad(A::mad(s, A::load(mr + 2 * A::kCoef16), x2), A::load(mr + 3 * A::kCoef16), x3);
        }
        v[j] = y[0];
        v[j | B0] = y[1];
        v[j | B1] = y[2];
        v[j | B0 | B1] = y[3];
    }
}

template <typename A, int RB, int PAIR>
__device__ __forceinline__ void r_swap(typename A::Amp (&v)[1 << RB], uint32_t jm) {
    constexpr int B0 = 1 << (2 * PAIR), B1 = 2 << (2 * PAIR);
#pragma unroll
    for (int j = 0; j < (1 << RB); j++) {
        if (j & (B0 | B1)) continue;
        if (!((jm >> j) & 1)) continue;
        const typename A::Amp w = v[j | B0];
        v[j | B0] = v[j | B1];
        v[j | B1] = w;
    }
}

// Density matrices: the register index of entry (row a, column b) of the
// pairs' qubits is b0 + 2 a0 + 4 b1 + 8 a1.  The Kraus sum of a channel is
// formed operator by operator like in the passes of one channel (dm.cu):
// acc = 0; acc += c_b (r_a entry), each product and sum rounded, with real
// weights (a pair of imaginary ones is a real pair).
__device__ __forceinline__ double2 d_kraus(double2 acc, double r, double c, double2 x) {
    return make_double2(__dadd_rn(acc.x, __dmul_rn(c, __dmul_rn(r, x.x))), __dadd_rn(acc.y, __dmul_rn(c, __dmul_rn(r, x.y))));
}

// Operator types of RC_CHAN1: 0 diagonal, 1 exchange of 0 and 1, 2 |0><1|,
// 3 |1><0| (times weights).  G groups of entries go
// through the operators together: an operator's words are read once for them,
// and their sums are independent (one group at a time waited for each sum).
// Measured on 11 qubits (64 MiB), 66 rotations and 15 CZ with a channel after
// each and 33 dampings: a pass for every gate and channel 5.1 ms, register
// passes with one group at a time 3.8, with two 2.8; bound by the rounded
// products and sums (no fused multiply-adds, like the lone passes).
template <int RB, int PAIR, int G>
__device__ __forceinline__ void r_chan1(double2 (&v)[1 << RB], const uint4* m, int nk) {
    constexpr int B = 1 << (2 * PAIR), A = 2 << (2 * PAIR);  // column, row
    constexpr int OTHER = PAIR ? 1 : 4;                      // the groups' first entries: multiples of this below A | B left out
#pragma unroll
    for (int g0 = 0; g0 < (1 << RB) / 4; g0 += G) {
        double2 x[G][4], y[G][4];
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int j = (g0 + g) * OTHER;
            x[g][0] = v[j];
            x[g][1] = v[j | B];
            x[g][2] = v[j | A];
            x[g][3] = v[j | A | B];
#pragma unroll
            for (int e = 0; e < 4; e++) y[g][e] = make_double2(0.0, 0.0);
        }
        for (int q = 0; q < nk; q++) {
            const uint32_t type = m[3 * q].x;
            const double2 r = *(const double2*)&m[3 * q + 1], c = *(const double2*)&m[3 * q + 2];
            if (type <= 1) {
#pragma unroll
                for (int g = 0; g < G; g++) {
                    if (type == 0) {
                        y[g][0] = d_kraus(y[g][0], r.x, c.x, x[g][0]);
                        y[g][1] = d_kraus(y[g][1], r.x, c.y, x[g][1]);
                        y[g][2] = d_kraus(y[g][2], r.y, c.x, x[g][2]);
                        y[g][3] = d_kraus(y[g][3], r.y, c.y, x[g][3]);
                    } else {
                        y[g][0] = d_kraus(y[g][0], r.x, c.x, x[g][3]);
                        y[g][1] = d_kraus(y[g][1], r.x, c.y, x[g][2]);
                        y[g][2] = d_kraus(y[g][2], r.y, c.x, x[g][1]);
                        y[g][3] = d_kraus(y[g][3], r.y, c.y, x[g][0]);
                    }
                }
            } else if (type == 2) {
#pragma unroll
                for (int g = 0; g < G; g++) y[g][0] = d_kraus(y[g][0], r.x, c.x, x[g][3]);
            } else {
#pragma unroll
                for (int g = 0; g < G; g++) y[g][3] = d_kraus(y[g][3], r.y, c.y, x[g][0]);
            }
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int j = (g0 + g) * OTHER;
            v[j] = y[g][0];
            v[j | B] = y[g][1];
            v[j | A] = y[g][2];
            v[j | A | B] = y[g][3];
        }
    }
}

// register index of (row i, column i ^ d) of the two qubits
__device__ __host__ constexpr int d_orbit(int i, int d) {
    return ((i ^ d) & 1) | ((i & 1) << 1) | ((((i ^ d) >> 1) & 1) << 2) | ((i >> 1) << 3);
}

// A 2-qubit channel whose operators all exchange a with a ^ x: the entries
// (i, i ^ d) of one d stay among themselves, so a few accumulators at a time
// serve; two values of d go through the operators together.
__device__ __forceinline__ void r_chan2(double2 (&v)[16], const uint4* m, int nk) {
#pragma unroll
    for (int d0 = 0; d0 < 4; d0 += 2) {
        double2 s[2][4], y[2][4];
#pragma unroll
        for (int g = 0; g < 2; g++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                s[g][i] = v[d_orbit(i, d0 + g)];
                y[g][i] = make_double2(0.0, 0.0);
            }
        for (int q = 0; q < nk; q++) {
            const uint4* w = m + 5 * q;
            const double* r = (const double*)(w + 1);
            const double* c = (const double*)(w + 3);
            switch (w[0].x) {
#define D_CHAN2(X)                                                                              \
    case X:                                                                                     \
        _Pragma("unroll") for (int g = 0; g < 2; g++) {                                         \
            _Pragma("unroll") for (int i = 0; i < 4; i++)                                       \
                y[g][i] = d_kraus(y[g][i], r[i], c[i ^ (d0 + g)], s[g][i ^ X]);                 \
        }                                                                                       \
        break;
                D_CHAN2(0)
                D_CHAN2(1)
                D_CHAN2(2)
            default:
                D_CHAN2(3)
#undef D_CHAN2
            }
        }
#pragma unroll
        for (int g = 0; g < 2; g++)
#pragma unroll
            for (int i = 0; i < 4; i++) v[d_orbit(i, d0 + g)] = y[g][i];
    }
}

__device__ __forceinline__ void r_pauli2(double2 (&v)[16], const uint4* m) {
#pragma unroll
    for (int d = 0; d < 4; d++) {
        double2 s[4];
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = v[d_orbit(i, d)];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double2 p = *(const double2*)&m[8 * d + 2 * i], q = *(const double2*)&m[8 * d + 2 * i + 1];
            v[d_orbit(i, d)] = make_double2(fma(p.x, s[0].x, fma(p.y, s[1].x, fma(q.x, s[2].x, q.y * s[3].x))),
                                            fma(p.x, s[0].y, fma(p.y, s[1].y, fma(q.x, s[2].y, q.y * s[3].y))));
        }
    }
}

// y_r = f_r sum_c R[r][c] x_c, or y_r = sum_c R[r][c] (f_c x_c): what the
// rotations, dampings and depolarizations of one qubit between two gates
// multiply to.  The 16 reals stay in registers for the four groups.
template <int RB, int PAIR>
__device__ __forceinline__ void r_real2(double2 (&v)[1 << RB], const uint4* m, bool cols) {
    constexpr int B0 = 1 << (2 * PAIR), B1 = 2 << (2 * PAIR);
    double2 R[8];
#pragma unroll
    for (int i = 0; i < 8; i++) R[i] = *(const double2*)&m[i];
    const double2* f = (const double2*)&m[8];
#pragma unroll
    for (int j = 0; j < (1 << RB); j++) {
        if (j & (B0 | B1)) continue;
        double2 x[4] = {v[j], v[j | B0], v[j | B1], v[j | B0 | B1]}, y[4];
        if (cols)
#pragma unroll
            for (int c = 0; c < 4; c++) x[c] = A128<false>::mul(A128<false>::Coef{f[c]}, x[c]);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const double2 p = R[2 * r], q = R[2 * r + 1];
            y[r] = make_double2(fma(p.x, x[0].x, fma(p.y, x[1].x, fma(q.x, x[2].x, q.y * x[3].x))),
                                fma(p.x, x[0].y, fma(p.y, x[1].y, fma(q.x, x[2].y, q.y * x[3].y))));
        }
        if (!cols)
#pragma unroll
            for (int r = 0; r < 4; r++) y[r] = A128<false>::mul(A128<false>::Coef{f[r]}, y[r]);
        v[j] = y[0];
        v[j | B0] = y[1];
        v[j | B1] = y[2];
        v[j | B0 | B1] = y[3];
    }
}

// A REAL1 op without pair signs from its words, without the way over the switch.
template <typename A, int RB, int P>
__device__ __forceinline__ void r_next(typename A::Amp (&v)[1 << RB], const uint4*& op, const uint4* coef, uint32_t t,
                                       uint32_t lb) {
    const uint4 w0 = op[0], w1 = op[1];
    op += 2;
    const bool on = (t & w0.w) == w1.x && (lb & (w0.z & 0xffffu)) == (w0.z >> 16);
    r_real1<A, RB, P>(v, coef + (size_t)w0.y * A::kCoef16, 0u, on && (w1.w >> 16) ? 0x80000000u : 0u);
}

// The ops of one segment on one thread's amplitudes.  t: the tile's number;
// lb: the thread's tile position (register positions at 0).
// DMX: density-matrix steps among the ops (a kernel of its own: their
// registers would spill the others' amplitudes).
template <typename A, bool EXACT, int RB, bool DMX>
__device__ __forceinline__ void r_ops(typename A::Amp (&v)[1 << RB], const uint4* ops, const uint4* coef, int begin,
                                      int end, uint32_t t, uint32_t lb) {
    for (int oi = begin; oi < end; oi++) {
        const uint4 w0 = ops[2 * oi], w1 = ops[2 * oi + 1];
        const bool on = (t & w0.w) == w1.x && (lb & (w0.z & 0xffffu)) == (w0.z >> 16);
        const uint32_t jm = on ? w0.x >> 16 : 0u;
        const uint32_t sg = EXACT ? 0u : w1.w & 0xffffu;                       // pairs negated
        const uint32_t cs = !EXACT && on && (w1.w >> 16) ? 0x80000000u : 0u;   // the second column negated
        const uint4* m = coef + (size_t)w0.y * A::kCoef16;
        switch (w0.x & 0xffu) {
        case RC_DENSE1 + 0: r_dense1<A, RB, 0, !EXACT>(v, m, jm, sg, cs); break;
        case RC_DENSE1 + 1: r_dense1<A, RB, 1, !EXACT>(v, m, jm, sg, cs); break;
        case RC_DENSE1 + 2:
            if constexpr (RB > 2) r_dense1<A, RB, 2, !EXACT>(v, m, jm, sg, cs);
            break;
        case RC_DENSE1 + 3:
            if constexpr (RB > 3) r_dense1<A, RB, 3, !EXACT>(v, m, jm, sg, cs);
            break;
        case RC_REAL1 + 0:
            if constexpr (!EXACT) r_real1<A, RB, 0>(v, m, sg, cs);
            break;
        case RC_REAL1 + 1:
            if constexpr (!EXACT) r_real1<A, RB, 1>(v, m, sg, cs);
            break;
        case RC_REAL1 + 2:
            if constexpr (!EXACT && RB > 2) r_real1<A, RB, 2>(v, m, sg, cs);
            break;
        case RC_REAL1 + 3:
            if constexpr (!EXACT && RB > 3) r_real1<A, RB, 3>(v, m, sg, cs);
            break;
        case RC_RCOL1 + 0:
            if constexpr (!EXACT) r_rcol1<A, RB, 0>(v, m, sg, cs);
            break;
        case RC_RCOL1 + 1:
            if constexpr (!EXACT) r_rcol1<A, RB, 1>(v, m, sg, cs);
            break;
        case RC_RCOL1 + 2:
            if constexpr (!EXACT && RB > 2) r_rcol1<A, RB, 2>(v, m, sg, cs);
            break;
        case RC_RCOL1 + 3:
            if constexpr (!EXACT && RB > 3) r_rcol1<A, RB, 3>(v, m, sg, cs);
            break;
        case RC_RROW1 + 0:
            if constexpr (!EXACT) r_rrow1<A, RB, 0>(v, m, sg, cs);
            break;
        case RC_RROW1 + 1:
            if constexpr (!EXACT) r_rrow1<A, RB, 1>(v, m, sg, cs);
            break;
        case RC_RROW1 + 2:
            if constexpr (!EXACT && RB > 2) r_rrow1<A, RB, 2>(v, m, sg, cs);
            break;
        case RC_RROW1 + 3:
            if constexpr (!EXACT && RB > 3) r_rrow1<A, RB, 3>(v, m, sg, cs);
            break;
        case RC_MASKED1 + 0: r_dense1<A, RB, 0, false>(v, m, jm, 0u, 0u); break;
        case RC_MASKED1 + 1: r_dense1<A, RB, 1, false>(v, m, jm, 0u, 0u); break;
        case RC_MASKED1 + 2:
            if constexpr (RB > 2) r_dense1<A, RB, 2, false>(v, m, jm, 0u, 0u);
            break;
        case RC_MASKED1 + 3:
            if constexpr (RB > 3) r_dense1<A, RB, 3, false>(v, m, jm, 0u, 0u);
            break;
        case RC_X + 0: r_x<A, RB, 0>(v, jm); break;
        case RC_X + 1: r_x<A, RB, 1>(v, jm); break;
        case RC_X + 2:
            if constexpr (RB > 2) r_x<A, RB, 2>(v, jm);
            break;
        case RC_X + 3:
            if constexpr (RB > 3) r_x<A, RB, 3>(v, jm);
            break;
        case RC_PHASE1 + 0: r_phase1<A, EXACT, RB, 0>(v, A::load(m + r_entry(w1, t, lb) * A::kCoef16)); break;
        case RC_PHASE1 + 1: r_phase1<A, EXACT, RB, 1>(v, A::load(m + r_entry(w1, t, lb) * A::kCoef16)); break;
        case RC_PHASE1 + 2:
            if constexpr (RB > 2) r_phase1<A, EXACT, RB, 2>(v, A::load(m + r_entry(w1, t, lb) * A::kCoef16));
            break;
        case RC_PHASE1 + 3:
            if constexpr (RB > 3) r_phase1<A, EXACT, RB, 3>(v, A::load(m + r_entry(w1, t, lb) * A::kCoef16));
            break;
        case RC_DENSE2 + 0: r_dense2<A, EXACT, RB, 0>(v, m, jm); break;
        case RC_DENSE2 + 1:
            if constexpr (RB > 3) r_dense2<A, EXACT, RB, 1>(v, m, jm);
            break;
        case RC_SWAP + 0: r_swap<A, RB, 0>(v, jm); break;
        case RC_SWAP + 1:
            if constexpr (RB > 3) r_swap<A, RB, 1>(v, jm);
            break;
        case RC_CHAN1 + 0:
            if constexpr (DMX && EXACT) r_chan1<RB, 0, (RB > 3 ? 2 : 1)>(v, m, (int)w1.y);
            break;
        case RC_CHAN1 + 1:
            if constexpr (DMX && EXACT && RB > 3) r_chan1<RB, 1, 2>(v, m, (int)w1.y);
            break;
        case RC_CHAN2:
            if constexpr (DMX && EXACT && RB > 3) r_chan2(v, m, (int)w1.y);
            break;
        case RC_PAULI2:
            if constexpr (DMX && !EXACT && RB > 3) r_pauli2(v, m);
            break;
        case RC_REAL2 + 0:
            if constexpr (DMX && !EXACT) r_real2<RB, 0>(v, m, w1.y != 0);
            break;
        case RC_REAL2 + 1:
            if constexpr (DMX && !EXACT && RB > 3) r_real2<RB, 1>(v, m, w1.y != 0);
            break;
        case RC_LAYER:
            if constexpr (!EXACT && RB > 3 && !DMX) {
                if (w1.y != ~0u) {
                    const uint4* d = coef + (size_t)w1.y * A::kCoef16;
#pragma unroll
                    for (int j = 1; j < (1 << RB); j++) v[j] = A::mul(A::load(d + (j - 1) * A::kCoef16), v[j]);
                }
                const uint4* next = ops + 2 * oi;
                r_next<A, RB, 0>(v, next, coef, t, lb);
                r_next<A, RB, 1>(v, next, coef, t, lb);
                r_next<A, RB, 2>(v, next, coef, t, lb);
                r_next<A, RB, 3>(v, next, coef, t, lb);
                oi += 3;
            }
            break;
        case RC_NEG:
#pragma unroll
            for (int j = 0; j < (1 << RB); j++)
                if ((jm >> j) & 1) v[j] = A::neg(v[j]);
            break;
        case RC_DIAG: {
            if (EXACT) break;  // not planned
            const uint4* md = m + ((size_t)r_entry(w1, t, lb) << RB) * A::kCoef16;
            // the tests also keep the loads apart: all coefficients at once would not fit the registers
#pragma unroll
            for (int j = 0; j < (1 << RB); j++)
                if ((jm >> j) & 1) v[j] = A::mul(A::load(md + j * A::kCoef16), v[j]);
            break;
        }
        default: {  // RC_PHASE
            const typename A::Coef c = A::load(m + r_entry(w1, t, lb) * A::kCoef16);
            if (EXACT && A::is_one(c)) break;  // as a gate alone: an entry of exactly 1 leaves its amplitudes alone
#pragma unroll
            for (int j = 0; j < (1 << RB); j++)
                if ((jm >> j) & 1) v[j] = A::mul(c, v[j]);
            break;
        }
        }
    }
}

__device__ __forceinline__ uint64_t r_base(const RHdr& h, uint32_t t) { return insert_zeros(t, h.tb, h.tbits); }
__device__ __forceinline__ uint64_t r_deposit(const RHdr& h, uint32_t l) {
    uint64_t o = 0;
    for (int j = 0; j < h.tbits; j++) o |= (uint64_t)((l >> j) & 1u) << h.tb[j];
    return o;
}

// A thread's place in a segment: its tile position (register positions at
// 0) and the swizzled byte offsets of that and of each register position.
template <int RB>
struct RPlace {
    uint32_t sb, so[RB];
    static __device__ __forceinline__ uint32_t position(const uint4& sg) {
        uint32_t lb = threadIdx.x;
#pragma unroll
        for (int i = 0; i < RB; i++) {
            const uint32_t p = (sg.z >> (8 * i)) & 0xffu;
            lb = ((lb >> p) << (p + 1)) | (lb & ((1u << p) - 1));
        }
        return lb;
    }
    __device__ __forceinline__ RPlace(const uint4& sg, uint32_t lb, uint32_t amp) {
#pragma unroll
        for (int i = 0; i < RB; i++) so[i] = tma::swizzle128(amp << ((sg.w >> (8 * i)) & 0xffu));
        sb = tma::swizzle128(lb * amp);
    }
    __device__ __forceinline__ uint32_t at(int j) const {
        uint32_t o = sb;
#pragma unroll
        for (int i = 0; i < RB; i++)
            if (j & (1 << i)) o ^= so[i];
        return o;
    }
};

// Threads of a CTA and CTAs an SM that the registers are divided for.  At 16
// amplitudes a thread, complex128 takes 168 registers (at 128 the compiler
// spills, and the register passes of the layered circuit, n = 28, 20 layers,
// took 118 ms against 109 ms then) and 2^11 tiles; complex64 takes 128 and
// 2^12 tiles (one more moving bit a pass: 111 ms against 116 ms then).
template <typename A, int RB>
constexpr int kRegThreads = RB < 4 ? 512 : sizeof(typename A::Amp) == 16 ? 128 : 256;
template <typename A, int RB>
constexpr int reg_ctas() {
    return RB < 4 ? 1 : sizeof(typename A::Amp) == 16 ? 3 : 2;
}

// Persistent: CTA b takes tiles b, b + grid, ...  A tile arrives in a shared
// buffer (TMA; small tiles and shapes without a tensor map by plain loads),
// changes hands there between segments, and leaves from the last segment's
// registers by plain stores (that segment's register positions are not the
// lowest, so a warp writes whole 128-byte runs).  The buffer is free once
// the last segment has read it: thread 0 then issues the load of the tile
// nbuf tiles on, which arrives while this one computes.  Every wait is
// bounded: one that gives up sets *err and the pass's result is void.
template <typename A, bool EXACT, int RB, bool DMX, bool TMA>
__device__ __forceinline__ void r_pass(typename A::Amp* __restrict__ st, const RHdr& hdr, const uint4* __restrict__ gblob,
                                       int* __restrict__ err, const CUtensorMap* tmap, uint32_t t, uint32_t grid) {
    typedef typename A::Amp Amp;
    constexpr uint32_t AB = sizeof(Amp);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full_bar[4];
    __shared__ uint64_t tbase[4];  // base index of the tile in each buffer
    __shared__ uint32_t place[kRegThreads<A, RB>];
    unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t tile_bytes = AB << hdr.tbits;
    const uint32_t nbuf = (uint32_t)hdr.nbuf;
    uint4* blob = (uint4*)(smem + (size_t)nbuf * tile_bytes);
    for (int i = threadIdx.x; i < hdr.blob16; i += blockDim.x) blob[i] = gblob[i];
    const bool use_tma = TMA && hdr.use_tma != 0;
    uint32_t pending = 0;  // thread 0: buffers with a load in flight
    auto load = [&](uint32_t tt, uint32_t b) {
        const uint64_t base = r_base(hdr, tt);
        tbase[b] = base;
        if (!use_tma) return;
        tc::mbar_arrive_expect_tx(&full_bar[b], tile_bytes);
        tma::load_boxes(tmap, hdr.tma, base, tc::smem_u32(smem) + b * tile_bytes, tc::smem_u32(&full_bar[b]));
        pending |= 1u << b;
    };
    if (threadIdx.x == 0) {
        if (use_tma) {
            tma::prefetch_map(tmap);
            for (uint32_t q = 0; q < nbuf; q++) tc::mbar_init(&full_bar[q], 1);
        }
        for (uint32_t q = 0; q < nbuf; q++)
            if ((uint64_t)t + (uint64_t)q * grid < hdr.ntiles) load(t + q * grid, q);
    }
    __syncthreads();
    const uint4* ops = blob + hdr.ops16;
    const uint4* coef = blob + hdr.coef16;
    const bool mine = threadIdx.x < (1u << (hdr.tbits - RB));
    const int last = hdr.nsegs - 1;
    // where the thread's amplitudes of the last segment go in a tile (its
    // lowest three bits are those of the tile position; read by it alone)
    place[threadIdx.x] = (uint32_t)(r_deposit(hdr, RPlace<RB>::position(blob[last])) >> 3);
    bool dead = false;
    uint32_t b = 0, par = 0;
    for (; t < hdr.ntiles; t += grid) {
        unsigned char* s = smem + (size_t)b * tile_bytes;
        if (use_tma) {
            if (!dead) {
                const uint64_t t0 = tma::now_ns();
                while (!tc::mbar_try_wait(&full_bar[b], par)) {
                    if (tma::now_ns() - t0 > tma::kWaitNs) {
                        dead = true;
                        atomicExch(err, 1);
                        break;
                    }
                }
                if (!dead && threadIdx.x == 0) pending &= ~(1u << b);
            }
        } else {
            for (uint32_t l = threadIdx.x; l < (1u << hdr.tbits); l += blockDim.x)
                *(Amp*)(s + tma::swizzle128(l * AB)) = st[tbase[b] | r_deposit(hdr, l)];
            __syncthreads();
        }
        const uint64_t base = tbase[b];
        for (int si = 0; si <= last; si++) {
            const uint4 sg = blob[si];
            if (si) __syncthreads();
            const uint32_t lb = RPlace<RB>::position(sg);
            Amp v[1 << RB];
            {
                const RPlace<RB> pl(sg, lb, AB);
                if (mine) {
#pragma unroll
                    for (int j = 0; j < (1 << RB); j++) v[j] = *(const Amp*)(s + pl.at(j));
                }
            }
            if (si == last) {
                tc::fence_proxy_async();  // this thread's writes to the buffer come before the next tile's copy
                __syncthreads();
                if (threadIdx.x == 0 && (uint64_t)t + (uint64_t)nbuf * grid < hdr.ntiles) load(t + nbuf * grid, b);
            }
            if (!mine) continue;
            r_ops<A, EXACT, RB, DMX>(v, ops, coef, (int)sg.x, (int)sg.y, t, lb);
            // the place again from the segment's words: kept through the ops
            // it would take registers from the amplitudes
            asm volatile("" ::: "memory");
            const uint4 sg2 = blob[si];
            const RPlace<RB> pl(sg2, lb, AB);
            if (si < last) {
#pragma unroll
                for (int j = 0; j < (1 << RB); j++) *(Amp*)(s + pl.at(j)) = v[j];
            } else {
                Amp* dst = st + (base | ((uint64_t)place[threadIdx.x] << 3) | (lb & 7u));
                uint64_t goff[RB];
#pragma unroll
                for (int i = 0; i < RB; i++) goff[i] = 1ull << hdr.tb[(sg2.w >> (8 * i)) & 0xffu];
#pragma unroll
                for (int j = 0; j < (1 << RB); j++) {
                    uint64_t o = 0;
#pragma unroll
                    for (int i = 0; i < RB; i++)
                        if (j & (1 << i)) o |= goff[i];
                    dst[o] = v[j];
                }
            }
        }
        if (!use_tma) __syncthreads();  // the next tile's base is in place
        b = b + 1 == nbuf ? 0u : b + 1;
        if (b == 0) par ^= 1u;
    }
    if (threadIdx.x == 0) {
        const uint64_t t0 = tma::now_ns();
        for (uint32_t q = 0; q < nbuf; q++)
            if (pending & (1u << q))
                for (uint32_t ph = 0; ph < 2; ph++)
                    while (!tc::mbar_try_wait(&full_bar[q], ph) && tma::now_ns() - t0 < tma::kWaitNs) {
                    }
    }
}

template <typename A, bool EXACT, int RB, bool DMX>
__global__ void __launch_bounds__(kRegThreads<A, RB>, reg_ctas<A, RB>())
    k_reg_tiles(typename A::Amp* __restrict__ st, const RHdr phdr, const uint4* __restrict__ gblob,
                int* __restrict__ err, const __grid_constant__ CUtensorMap tmap) {
    __shared__ RHdr hdr;
    if (threadIdx.x == 0) hdr = phdr;
    __syncthreads();
    r_pass<A, EXACT, RB, DMX, true>(st, hdr, gblob, err, &tmap, blockIdx.x, gridDim.x);
}

// One pass of each of many registers: a CTA belongs to the pass owner[CTA].
struct RBatchPass {
    RHdr hdr;
    uint64_t state, blob;   // addresses
    uint32_t cta0, ctas;    // its CTAs
};
static_assert(sizeof(RBatchPass) % 8 == 0, "copied by words");

template <typename A, bool EXACT, int RB>
__global__ void __launch_bounds__(kRegThreads<A, RB>, reg_ctas<A, RB>())
    k_reg_batch(const RBatchPass* __restrict__ passes, const uint32_t* __restrict__ owner) {
    __shared__ RBatchPass pass;
    const uint32_t* src = (const uint32_t*)(passes + owner[blockIdx.x]);
    for (uint32_t i = threadIdx.x; i < sizeof(RBatchPass) / 4; i += blockDim.x) ((uint32_t*)&pass)[i] = src[i];
    __syncthreads();
    r_pass<A, EXACT, RB, false, false>((typename A::Amp*)(uintptr_t)pass.state, pass.hdr,
                                       (const uint4*)(uintptr_t)pass.blob, nullptr, nullptr,
                                       blockIdx.x - pass.cta0, pass.ctas);
}

// ================================================================= planner

static uint64_t target_mask(const LGate& g) {
    uint64_t m = 0;
    for (int i = 0; i < g.k; i++) m |= (uint64_t)1 << g.tb[i];
    return m;
}
static uint64_t qubit_mask(const LGate& g) {
    uint64_t m = target_mask(g);
    for (int i = 0; i < g.nc; i++) m |= (uint64_t)1 << g.cb[i];
    return m;
}
// Bits that must be in the tile, and in registers: the ones a gate moves
// amplitudes along and, where order is free, a 1-qubit diagonal's (it then
// costs half the amplitudes and joins its neighbours).
static uint64_t need_mask(const LGate& g, bool exact) {
    return g.cls == GC_DIAG && !(g.k == 1 && g.nc == 0 && !exact) ? 0 : target_mask(g);
}
static bool is_perm(const LGate& g) { return g.cls == GC_X || g.cls == GC_SWAP; }

static bool reg_width(uint32_t nbits) { return nbits >= 4 && nbits <= 33; }
// (Gates without a target, or with a qubit twice, are left to the passes of
// one gate, which refuse them or give them a meaning.)
static bool reg_gate(const LGate& g) {
    if (g.k < 1 || __builtin_popcountll(qubit_mask(g)) != g.k + g.nc) return false;
    return !((g.cls == GC_DENSE && g.k > 2) || (g.cls == GC_X && g.k != 1));
}
// steps on two qubits of a density matrix: all four register positions
static bool four_bits(const LGate& g) { return g.cls == GC_CHAN2 || g.cls == GC_PAULI2; }

bool reg_supported(const std::vector<LGate>& prog, uint32_t nbits) {
    if (!reg_width(nbits)) return false;
    for (const LGate& g : prog)
        if (!reg_gate(g)) return false;
    return true;
}

// What the scans below ask of a gate: its qubits, the bits it needs in the
// tile, whether it only moves amplitudes.
struct GateBits {
    uint64_t qubits, need;
    bool perm;
};

// Which gates of a list may be taken next, scanning it in order: a gate
// passes skipped ones only when it shares no qubit with them (and, for an
// exact result, it or all of them are permutations).  A scan ends where no
// gate can pass any more, or after kScanSkipped skipped ones: a qubit that no
// gate touches for long would keep every scan going to the end of the program
// (80000 gates on 14 qubits, one of them idle: planned in 1.5 s).
constexpr size_t kScanSkipped = 1024;

struct Scan {
    bool exact;
    uint64_t blocked = 0;
    size_t skipped = 0;
    bool arith = false;  // some skipped gate computes
    explicit Scan(bool e) : exact(e) {}
    bool free(const GateBits& g) const { return !(g.qubits & blocked) && (!exact || !arith || g.perm); }
    void skip(const GateBits& g) {
        blocked |= g.qubits;
        arith |= !g.perm;
        skipped++;
    }
    bool closed(uint64_t all) const { return (blocked & all) == all || skipped >= kScanSkipped; }
};

static Cx cmul(Cx a, Cx b) { return Cx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
static Cx conj(Cx a) { return Cx{a.re, -a.im}; }
static bool is(Cx c, double re) { return c.re == re && c.im == 0.0; }

// Extended precision (64 bits of mantissa) on the host: products of gates,
// moduli and phases are taken from it with one rounding, and squares of any
// double fit.
struct CxL {
    long double re, im;
    CxL() : re(0.0L), im(0.0L) {}
    CxL(long double r, long double i) : re(r), im(i) {}
    CxL(Cx a) : re(a.re), im(a.im) {}
    Cx round() const { return Cx{(double)re, (double)im}; }
};
static CxL operator+(CxL a, CxL b) { return CxL(a.re + b.re, a.im + b.im); }
static CxL operator*(CxL a, CxL b) { return CxL(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
static CxL operator*(long double x, CxL a) { return CxL(x * a.re, x * a.im); }
static CxL conj(CxL a) { return CxL(a.re, -a.im); }
static bool is(CxL c, long double re) { return c.re == re && c.im == 0.0L; }
static long double norm2(CxL a) { return a.re * a.re + a.im * a.im; }
// a / |a|
static CxL unit(CxL a) { return 1.0L / std::sqrt(norm2(a)) * a; }

namespace {

constexpr long double kRoot2 = 1.41421356237309504880168872420969808L;

// What waits to be applied on one qubit: nothing, a diagonal or a matrix
// (the product of `factors` matrices, a unitary one times the root of 2^twos
// where the gates are unitary).
struct Pend {
    bool on = false;
    int factors = 0, twos = 0;
    CxL m[4];
    bool diag() const { return is(m[1], 0.0L) && is(m[2], 0.0L); }
    void mul(const Cx* u) {  // m <- u m
        if (!on) {
            std::copy(u, u + 4, m);
            on = true;
            factors = 1;
            twos = 0;
            return;
        }
        const CxL x[4] = {m[0], m[1], m[2], m[3]};
        factors++;
        if (is(u[1], 0.0) && is(u[2], 0.0)) {
            for (int j = 0; j < 4; j++) m[j] = CxL(u[j & 2 ? 3 : 0]) * x[j];
            return;
        }
        if (u[0].im == 0.0 && u[1].im == 0.0 && u[2].im == 0.0 && u[3].im == 0.0) {
            for (int i = 0; i < 2; i++)
                for (int j = 0; j < 2; j++) m[2 * i + j] = (long double)u[2 * i].re * x[j] + (long double)u[2 * i + 1].re * x[2 + j];
            return;
        }
        for (int i = 0; i < 2; i++)
            for (int j = 0; j < 2; j++) m[2 * i + j] = CxL(u[2 * i]) * x[j] + CxL(u[2 * i + 1]) * x[2 + j];
    }
    // m <- by H m, where H is a Hadamard without its factor: with by = 1
    // before a CZ and a half after it the two make 1 exactly (the root of a
    // half rounded, squared and doubled is 1 + 2.2e-16)
    void hadamard(long double by) {
        if (!on) {
            m[0] = m[3] = CxL(1.0L, 0.0L);
            m[1] = m[2] = CxL(0.0L, 0.0L);
            factors = twos = 0;
            on = true;
        }
        for (int j = 0; j < 2; j++) {
            const CxL x = m[j], y = m[2 + j];
            m[j] = by * (x + y);
            m[2 + j] = by * (x + -1.0L * y);
        }
        factors++;
        twos += by == 1.0L ? 1 : -1;
    }
    // To the rounding of the factors (a number within 1e-13 of 1 may multiply it).
    bool unitary() const {
        const long double two = std::ldexp(1.0L, twos), eps = 1e-15L * (factors + 1) * two;
        const long double a = norm2(m[0]) + norm2(m[2]), b = norm2(m[1]) + norm2(m[3]);
        const CxL x = conj(m[0]) * m[1] + conj(m[2]) * m[3];
        return std::fabs(a - two) < 1e-13L * two && std::fabs(a - b) < eps && std::fabs(x.re) < eps && std::fabs(x.im) < eps;
    }
};

struct Splitter {
    std::vector<Pend> pend;
    std::vector<LGate>& out;
    CxL scale{1.0L, 0.0L};  // of the whole state
    Splitter(uint32_t n, std::vector<LGate>& o) : pend(n), out(o) {}

    void emit1(int b, int cls, std::vector<Cx> m) {
        out.emplace_back();
        LGate& g = out.back();
        g.cls = cls;
        g.k = 1;
        g.tb[0] = b;
        g.m = std::move(m);
    }
    // Applies what waits on bit b, except a diagonal when `keep_diag`
    // (what comes next commutes with it).  Matrices are rounded once, here;
    // the state's scale takes what the rounded ones are off in norm, so that
    // a long circuit's norm strays by the roundings of its amplitudes alone.
    void flush(int b, bool keep_diag) {
        Pend& p = pend[b];
        if (!p.on) return;
        const CxL *m = p.m, one(1.0L, 0.0L), zero(0.0L, 0.0L);
        if (!p.diag()) {
            if (is(m[0], 0.0L) && is(m[3], 0.0L) && is(m[1], 1.0L) && is(m[2], 1.0L)) {
                emit1(b, GC_X, {});
                p.on = false;
                return;
            }
            if (!p.unitary()) {
                emit1(b, GC_DENSE, {m[0].round(), m[1].round(), m[2].round(), m[3].round()});
                p.on = false;
                return;
            }
            // r e^{i alpha} diag(1, f) [[c, -s], [s, c]] diag(1, l): the larger
            // of a column's entries fixes its phase.  r and the columns' norms
            // are the root of 2^twos to 1e-13, so series give their roots.
            const long double root = p.twos == 0 ? 1.0L : p.twos > 0 ? kRoot2 : 0.5L * kRoot2, two = root * root;
            const long double n0 = norm2(m[0]), n2 = norm2(m[2]), off = (n0 + n2) / two - 1.0L;
            const long double i0 = n0 > 0.0L ? 1.0L / std::sqrt(n0) : 0.0L, i2 = n2 > 0.0L ? 1.0L / std::sqrt(n2) : 0.0L;
            const long double col = (1.0L - 0.5L * off) / root, c = n0 * i0 * col, s = n2 * i2 * col;
            CxL al = one, f = one, l = one;
            if (c >= s) {
                al = i0 * m[0];
                const CxL fl = i0 * (m[3] * conj(al));  // f l
                f = s > 0.0L ? i2 * (m[2] * conj(al)) : fl;
                l = fl * conj(f);
            } else {
                const CxL g = i2 * m[2];       // alpha f
                const CxL h = -i2 * m[1];      // alpha l
                al = c > 0.0L ? i0 * m[0] : g;
                f = g * conj(al);
                l = h * conj(al);
            }
            // what is left of the diagonal after it waits for the next
            // rotation of this bit, else it joins the matrix
            const CxL g = keep_diag ? one : f;
            const Cx e[4] = {CxL(c, 0.0L).round(), (-s * l).round(), (s * g).round(), (c * (g * l)).round()};
            const CxL left = keep_diag ? CxL(f.round()) : one;
            const long double have = (norm2(e[0]) + norm2(e[1]) + norm2(e[2]) + norm2(e[3])) * (1.0L + norm2(left));
            const long double want = (n0 + n2 + norm2(m[1]) + norm2(m[3])) * 2.0L / two;
            scale = scale * (root * (1.0L + 0.5L * (want / have - 1.0L)) * al);
            emit1(b, GC_DENSE, std::vector<Cx>(e, e + 4));
            p.m[0] = one;
            p.m[1] = p.m[2] = zero;
            p.m[3] = left;
            p.on = !is(left, 1.0L);
            p.factors = 1;
            p.twos = 0;
            return;
        }
        if (keep_diag || !p.on) return;
        Cx d[2] = {m[0].round(), m[3].round()};
        if (p.unitary()) {
            const CxL a = m[0];
            d[0] = Cx{1.0, 0.0};
            d[1] = ((1.0L / norm2(a)) * (conj(a) * m[3])).round();
            const long double ratio = (norm2(a) + norm2(m[3])) / ((1.0L + norm2(d[1])) * norm2(a));
            scale = scale * ((1.0L + 0.5L * (ratio - 1.0L)) * a);
        }
        if (!(is(d[0], 1.0) && is(d[1], 1.0))) emit1(b, GC_DIAG, {d[0], d[1]});
        p.on = false;
    }
};

}  // namespace

void split_single_qubit(const std::vector<LGate>& prog, uint32_t nbits, std::vector<LGate>& out) {
    out.clear();
    out.reserve(prog.size() + nbits);  // (grown step by step, the gates' 576 bytes each move twice)
    Splitter sp(nbits, out);
    auto single = [](const LGate& g) { return g.k == 1 && g.nc == 0; };
    // per gate: whether the next gate on its target that is no 1-qubit
    // diagonal is a 1-qubit rotation
    std::vector<char> rot_next(prog.size(), 0), next(nbits, 0);
    for (size_t i = prog.size(); i-- > 0;) {
        const LGate& g = prog[i];
        rot_next[i] = next[g.tb[0]];
        if (single(g)) {
            if (g.cls == GC_DENSE) next[g.tb[0]] = 1;
            continue;
        }
        for (int q = 0; q < g.k; q++) next[g.tb[q]] = 0;
        for (int q = 0; q < g.nc; q++) next[g.cb[q]] = 0;
    }
    for (size_t i = 0; i < prog.size(); i++) {
        const LGate& g = prog[i];
        if (single(g)) {
            Cx u[4] = {{0, 0}, {1, 0}, {1, 0}, {0, 0}};  // GC_X
            if (g.cls == GC_DENSE) {
                std::copy(g.m.begin(), g.m.begin() + 4, u);
            } else if (g.cls == GC_DIAG) {
                u[0] = g.m[0];
                u[1] = u[2] = Cx{0, 0};
                u[3] = g.m[1];
            }
            sp.pend[g.tb[0]].mul(u);
            continue;
        }
        const int t = g.tb[0];
        if (g.cls == GC_X && g.nc == 1 && rot_next[i] && sp.pend[t].on && !sp.pend[t].diag() && sp.pend[t].unitary()) {
            sp.pend[t].hadamard(1.0L);
            sp.flush(t, true);
            sp.flush(g.cb[0], true);
            out.emplace_back();
            LGate& z = out.back();
            z.cls = GC_DIAG;
            z.k = 2;
            z.tb[0] = std::min(t, (int)g.cb[0]);
            z.tb[1] = std::max(t, (int)g.cb[0]);
            z.m.assign(4, Cx{1.0, 0.0});
            z.m[g.cv[0] ? 3 : (t == z.tb[0] ? 1 : 2)] = Cx{-1.0, 0.0};
            sp.pend[t].hadamard(0.5L);
            continue;
        }
        for (int q = 0; q < g.k; q++) sp.flush(g.tb[q], g.cls == GC_DIAG);
        for (int q = 0; q < g.nc; q++) sp.flush(g.cb[q], true);
        out.push_back(g);
    }
    for (uint32_t b = 0; b < nbits; b++) sp.flush((int)b, false);
    // the state's scale joins the last phase gate, else the last matrix
    const Cx scale = sp.scale.round();
    if (is(scale, 1.0)) return;
    for (int cls : {(int)GC_DIAG, (int)GC_DENSE})
        for (size_t i = out.size(); i-- > 0;)
            if (out[i].cls == cls && out[i].nc == 0) {
                for (Cx& x : out[i].m) x = cmul(x, scale);
                return;
            }
    sp.emit1(0, GC_DIAG, {scale, scale});
}

// Description of a pass kept below this, so that three CTAs of 2^11
// complex128 amplitudes (two buffers each) share an SM; a longer run of
// gates becomes further passes.  Two CTAs of 2^12 complex64 amplitudes leave
// more room, and its coefficients take twice the bytes (at 8 KB the layered
// circuit took 27 passes instead of 21).
constexpr size_t kRegBlobCap = 8 * 1024, kRegBlobCap64 = 16 * 1024;

namespace {

// Gates of one segment and the register positions they need.
struct SegPlan {
    std::vector<const LGate*> gates;
    std::vector<int> bits;                    // tile positions in registers
    std::vector<std::pair<int, int>> pairs;   // (even, odd) register positions of 2-qubit dense gates and swaps
};

// -1 where two bits have their values; a bit is a tile position, or 16 + a
// bit of the tile's number.
struct Sign {
    int bit[2], val[2];
};

struct PassBuilder {
    int rb;
    bool exact;
    bool dm_form;         // a density matrix's FUSED program
    int8_t local[64];     // global bit -> tile position, -1 outside
    int8_t outside[64];   // global bit -> bit of the tile's number
    RegPass* p;
    std::vector<std::pair<uint32_t, size_t>> shared;  // coefficients of density-matrix steps

    bool fits(const SegPlan& s, const LGate& g) const {
        if (!need_mask(g, exact)) return true;
        int fresh = 0;
        for (int i = 0; i < g.k; i++)
            if (std::find(s.bits.begin(), s.bits.end(), (int)local[g.tb[i]]) == s.bits.end()) fresh++;
        if ((int)s.bits.size() + fresh > rb) return false;
        size_t more = 0;  // pairs that it would add
        for (int i = 0; i + 1 < g.k; i += 2) {
            const int a = local[g.tb[i]], b = local[g.tb[i + 1]];
            bool have = false;
            for (const auto& q : s.pairs) {
                have |= q.first == a && q.second == b;
                have |= g.cls == GC_SWAP && q.first == b && q.second == a;
                if (!have && (q.first == a || q.second == a || q.first == b || q.second == b)) return false;
            }
            more += !have;
        }
        return s.pairs.size() + more <= (size_t)rb / 2;
    }
    void add(SegPlan& s, const LGate& g) const {
        s.gates.push_back(&g);
        if (!need_mask(g, exact)) return;
        for (int i = 0; i < g.k; i++)
            if (std::find(s.bits.begin(), s.bits.end(), (int)local[g.tb[i]]) == s.bits.end())
                s.bits.push_back(local[g.tb[i]]);
        for (int i = 0; i + 1 < g.k; i += 2) {
            const int a = local[g.tb[i]], b = local[g.tb[i + 1]];
            bool have = false;
            for (const auto& q : s.pairs) have |= q.first == a || q.first == b;
            if (!have) s.pairs.push_back({a, b});
        }
    }
    void emit(const SegPlan& s) {
        RSeg sg;
        memset(&sg, 0, sizeof(sg));
        std::vector<int> order;
        for (const auto& q : s.pairs) {
            order.push_back(q.first);
            order.push_back(q.second);
        }
        for (int b : s.bits)
            if (std::find(order.begin(), order.end(), b) == order.end()) order.push_back(b);
        // unused register positions: the highest free tile bits, so that the
        // lanes of a warp step through the low ones
        for (int b = p->tbits - 1; (int)order.size() < rb && b >= 0; b--)
            if (std::find(order.begin(), order.end(), b) == order.end()) order.push_back(b);
        std::vector<int> sorted(order);
        std::sort(sorted.begin(), sorted.end());
        for (int i = 0; i < rb; i++) {
            sg.sorted[i] = (int8_t)sorted[i];
            sg.order[i] = (int8_t)order[i];
        }
        auto pos = [&](int l) -> int {
            const auto it = std::find(order.begin(), order.end(), l);
            return it == order.end() ? -1 : (int)(it - order.begin());
        };
        sg.op_begin = (int32_t)p->ops.size();
        const uint32_t na = 1u << rb;
        // A diagonal under way (not in exact passes): a table over the
        // register index and at most one bit outside the registers, dep the
        // register positions it depends on.  Diagonals commute with each
        // other, so it is applied when a gate moves one of those positions.
        struct {
            bool on = false;
            uint32_t dep = 0;
            int sel = -1;
            std::vector<Cx> tab;
        } acc;
        auto push = [&](uint32_t code, uint32_t jm, const ROp& base) {
            ROp op = base;
            if (code == RC_PHASE && !op.ctl && !op.gmask)
                for (int q = 0; q < rb; q++) {
                    uint32_t bit = 0;
                    for (uint32_t j = 0; j < na; j++) bit |= ((j >> q) & 1u) << j;
                    if (jm == bit) code = RC_PHASE1 + (uint32_t)q;
                }
            op.head = code | (jm << 16);
            p->ops.push_back(op);
        };
        auto flush = [&]() {
            if (!acc.on) return;
            acc.on = false;
            const uint32_t ne = acc.sel >= 0 ? 2 : 1;
            uint32_t jm = 0;
            for (uint32_t j = 0; j < na; j++)
                for (uint32_t e = 0; e < ne; e++)
                    if (!is(acc.tab[e * na + j], 1.0)) jm |= 1u << j;
            if (!jm) return;
            bool same = true;  // one coefficient for every amplitude it changes
            const uint32_t j0 = (uint32_t)__builtin_ctz(jm);
            for (uint32_t j = 0; j < na; j++)
                for (uint32_t e = 0; e < ne; e++)
                    if ((jm >> j) & 1)
                        same &= acc.tab[e * na + j].re == acc.tab[e * na + j0].re && acc.tab[e * na + j].im == acc.tab[e * na + j0].im;
            ROp op;
            memset(&op, 0, sizeof(op));
            op.coef = (uint32_t)p->coef.size();
            if (acc.sel >= 0) {
                op.sel0 = (uint32_t)acc.sel;
                op.sel1 = 1u << 8;
            }
            if (same)
                for (uint32_t e = 0; e < ne; e++) p->coef.push_back(acc.tab[e * na + j0]);
            else
                p->coef.insert(p->coef.end(), acc.tab.begin(), acc.tab.begin() + ne * na);
            push(same ? RC_PHASE : RC_DIAG, jm, op);
        };
        // Signs under way (not in exact passes): -1 where both tile positions
        // / outside bits have their values.  The next rotation of a register
        // position takes it along; otherwise it becomes an RC_NEG op.
        std::vector<Sign> signs;
        auto flush_sign = [&](const Sign& z) {
            ROp op;
            memset(&op, 0, sizeof(op));
            uint32_t jm = (1u << na) - 1;
            for (int q = 0; q < 2; q++) {
                if (z.bit[q] >= 16) {
                    op.gmask |= 1u << (z.bit[q] - 16);
                    op.gval |= (uint32_t)z.val[q] << (z.bit[q] - 16);
                } else if (pos(z.bit[q]) >= 0) {
                    for (uint32_t j = 0; j < na; j++)
                        if (((j >> pos(z.bit[q])) & 1u) != (uint32_t)z.val[q]) jm &= ~(1u << j);
                } else {
                    op.ctl |= (1u << z.bit[q]) | ((uint32_t)z.val[q] << (16 + z.bit[q]));
                }
            }
            push(RC_NEG, jm, op);
        };
        for (const LGate* g : s.gates) {
            ROp op;
            memset(&op, 0, sizeof(op));
            uint32_t rmask = 0, rval = 0, tmask = 0, tval = 0;
            for (int c = 0; c < g->nc; c++) {
                const int l = local[g->cb[c]];
                if (l < 0) {
                    op.gmask |= 1u << outside[g->cb[c]];
                    op.gval |= (uint32_t)(g->cv[c] ? 1 : 0) << outside[g->cb[c]];
                } else if (pos(l) >= 0) {
                    rmask |= 1u << pos(l);
                    rval |= (uint32_t)(g->cv[c] ? 1 : 0) << pos(l);
                } else {
                    tmask |= 1u << l;
                    tval |= (uint32_t)(g->cv[c] ? 1 : 0) << l;
                }
            }
            op.ctl = tmask | (tval << 16);
            op.coef = (uint32_t)p->coef.size();
            if (g->cls == GC_DIAG) {
                Sign z;
                if (!exact && two_bit_sign(*g, z))
                    signs.push_back(z);
                else
                    diagonal(*g, op, rmask, rval, na, pos, acc, flush, push);
                continue;
            }
            uint32_t bm = 0, jm = 0, pairs = 0;
            for (int i = 0; i < g->k; i++) bm |= 1u << pos(local[g->tb[i]]);
            for (uint32_t j = 0; j < na; j++)
                if (!(j & bm)) {
                    pairs |= 1u << j;
                    if ((j & rmask) == rval) jm |= 1u << j;
                }
            if (acc.on && (acc.dep & bm)) flush();
            const uint32_t p0 = (uint32_t)pos(local[g->tb[0]]);
            const bool matrix = g->cls == GC_DENSE && g->k == 1 && g->nc == 0 && !exact;
            bool cond = false;  // the op's controls are taken by a sign
            for (size_t q = 0; q < signs.size();) {
                const Sign z = signs[q];
                int hit = -1;  // the sign's half that this gate moves
                for (int i = 0; i < g->k; i++)
                    for (int w = 0; w < 2; w++)
                        if (z.bit[w] == (int)local[g->tb[i]]) hit = w;
                if (hit < 0) {
                    q++;
                    continue;
                }
                signs.erase(signs.begin() + q);
                const int o = z.bit[1 - hit], ov = z.val[1 - hit];
                if (!matrix || z.val[hit] != 1) {
                    flush_sign(z);
                } else if (o < 16 && pos(o) >= 0) {
                    for (uint32_t j = 0; j < na; j++)
                        if (((pairs >> j) & 1u) && ((j >> pos(o)) & 1u) == (uint32_t)ov) op.sign ^= 1u << j;
                } else if (!cond) {
                    cond = true;
                    if (o < 16) {
                        op.ctl = (1u << o) | ((uint32_t)ov << (16 + o));
                    } else {
                        op.gmask = 1u << (o - 16);
                        op.gval = (uint32_t)ov << (o - 16);
                    }
                    op.sign |= pairs << 16;
                } else {
                    flush_sign(z);
                }
            }
            if (dm_form && g->cls == GC_DENSE && g->k == 2 && g->nc == 0) {
                std::vector<Cx> m;
                bool cols = false;
                if (real_up_to_phases(g->m, m, &cols)) {
                    op.coef = (uint32_t)p->coef.size();
                    op.sel0 = cols;
                    p->coef.insert(p->coef.end(), m.begin(), m.end());
                    push(RC_REAL2 + p0 / 2, 0xffffu, op);
                    continue;
                }
            }
            if (g->cls >= GC_CHAN1) {
                op.coef = coefs_of(dm_coefs(*g, p0 != 0));
                if (g->cls == GC_PAULI2) {
                    push(RC_PAULI2, 0xffffu, op);
                } else {
                    const uint32_t per = g->cls == GC_CHAN1 ? 3 : 5;
                    op.sel0 = (uint32_t)g->m.size() / per;
                    push(g->cls == GC_CHAN1 ? RC_CHAN1 + p0 / 2 : (uint32_t)RC_CHAN2, 0xffffu, op);
                }
                continue;
            }
            op.coef = (uint32_t)p->coef.size();
            uint32_t code;
            auto is_real = [&](int i) { return g->m[i].im == 0.0; };
            auto two = [&](int i, int j) { p->coef.push_back(Cx{g->m[i].re, g->m[j].re}); };
            if (matrix && is_real(0) && is_real(1) && is_real(2) && is_real(3)) {
                code = RC_REAL1 + p0;
                two(0, 1);
                two(2, 3);
            } else if (matrix && is_real(0) && is_real(2)) {
                code = RC_RCOL1 + p0;
                two(0, 2);
                p->coef.push_back(g->m[1]);
                p->coef.push_back(g->m[3]);
            } else if (matrix && is_real(0) && is_real(1)) {
                code = RC_RROW1 + p0;
                two(0, 1);
                p->coef.push_back(g->m[2]);
                p->coef.push_back(g->m[3]);
            } else {
                if (g->k == 1)
                    code = (g->cls == GC_X ? RC_X : g->nc == 0 ? RC_DENSE1 : RC_MASKED1) + p0;
                else
                    code = (g->cls == GC_SWAP ? RC_SWAP : RC_DENSE2) + p0 / 2;
                for (const Cx& c : g->m) p->coef.push_back(c);
            }
            push(code, jm, op);
        }
        for (const Sign& z : signs) flush_sign(z);
        flush();
        if (!exact && !dm_form && rb == 4) group_layers((size_t)sg.op_begin);
        sg.op_end = (int32_t)p->ops.size();
        if (sg.op_end > sg.op_begin) p->segs.push_back(sg);
    }

    // Brings matrices on positions 0 to 3 that are real up to a phase of the
    // second column together (RC_LAYER) where the ops in between commute with
    // them: such matrices on other positions, unless one negates the pairs of
    // the other's position.  The phases, and the signs between two of the four
    // (a CZ before both), become one diagonal: 4 x 4 + 4 multiply-adds an
    // amplitude instead of 4 x 6, and the four go through the op loop at once.
    // Measured on the layered circuit, n = 28, 20 layers: complex128 105 -> 96
    // ms, complex64 111 -> 99.  (Three of four positions with a test for each:
    // 98 and 104, the code is no longer one straight line.)
    void group_layers(size_t begin) {
        auto code = [](const ROp& op) { return (op.head & 0xffu) & ~3u; };
        auto pos = [](const ROp& op) { return (int)(op.head & 3u); };
        // pairs of position a negated where position b is 1
        auto cz = [](int a, int b) {
            uint32_t m = 0;
            for (uint32_t j = 0; j < 16; j++) m |= (uint32_t)(!((j >> a) & 1u) && ((j >> b) & 1u)) << j;
            return m;
        };
        // the positions whose bits negate pairs of op's; false: not a product of CZs
        auto reads = [&](const ROp& op, uint32_t& r) {
            uint32_t left = op.sign & 0xffffu;
            r = 0;
            for (int q = 0; q < 4; q++)
                if (q != pos(op) && (left >> (1u << q)) & 1u) {
                    left ^= cz(pos(op), q);
                    r |= 1u << q;
                }
            return left == 0;
        };
        // the second column's phase (its entries are rounded, and no further
        // from the phase than that); false: it has none
        auto phase = [&](const ROp& op, CxL& u, Cx (&m)[2]) {
            const Cx* c = &p->coef[op.coef];
            m[0] = c[0];
            m[1] = c[1];
            u = CxL(1.0L, 0.0L);
            if (code(op) == RC_REAL1) return true;
            const CxL b = c[1], d = c[2];
            const long double nb = norm2(b), nd = norm2(d), eps = 4e-16L * std::sqrt(std::max(nb, nd));
            u = unit(nb > nd ? b : d);
            const CxL x = b * conj(u), y = d * conj(u);
            m[0] = Cx{c[0].re, (double)x.re};
            m[1] = Cx{c[0].im, (double)y.re};
            return std::fabs(x.im) <= eps && std::fabs(y.im) <= eps;
        };
        std::vector<ROp> list(p->ops.begin() + (long)begin, p->ops.end()), out;
        while (!list.empty()) {
            int at[4] = {-1, -1, -1, -1};
            uint32_t held = 0, read = 0, have = 0, r[4];  // positions of passed ops; those they read; the group's
            CxL u[4];
            Cx m[4][2];
            for (size_t k = 0; k < list.size() && k < 16 && have != 15u; k++) {
                const ROp& op = list[k];
                if (code(op) != RC_RCOL1 && code(op) != RC_REAL1) break;
                const int P = pos(op);
                uint32_t rd;
                if (!reads(op, rd)) break;
                // (a sign that reads a member before it stays after that member)
                if (!(((held | read | have) >> P) & 1u) && !(rd & (held | have)) && phase(op, u[P], m[P])) {
                    at[P] = (int)k;
                    r[P] = rd;
                    have |= 1u << P;
                } else {
                    held |= 1u << P;
                    read |= rd;
                }
            }
            if (have != 15u) {
                out.push_back(list[0]);
                list.erase(list.begin());
                continue;
            }
            Cx d[16];
            uint32_t minus = 0;
            for (uint32_t j = 0; j < 16; j++) {
                CxL x(1.0L, 0.0L);
                for (int P = 0; P < 4; P++) {
                    if (!((j >> P) & 1u)) continue;
                    x = x * u[P];
                    if (__builtin_popcount(r[P] & j) & 1) minus ^= 1u << j;
                }
                d[j] = ((minus >> j) & 1u ? -1.0L * x : x).round();
            }
            const bool phases = !(is(u[0], 1.0L) && is(u[1], 1.0L) && is(u[2], 1.0L) && is(u[3], 1.0L));
            if (!phases && minus) {
                ROp neg;
                memset(&neg, 0, sizeof(neg));
                neg.head = RC_NEG | (minus << 16);
                out.push_back(neg);
            }
            for (int P = 0; P < 4; P++) {
                ROp op = list[(size_t)at[P]];
                op.head = (op.head & ~0xffu) | (P == 0 ? (uint32_t)RC_LAYER : (uint32_t)RC_REAL1 + (uint32_t)P);
                op.sign &= 0xffff0000u;
                op.sel0 = ~0u;
                // (in the place of the op's own coefficients)
                p->coef[op.coef] = m[P][0];
                p->coef[op.coef + 1] = m[P][1];
                if (P == 0 && phases) {
                    op.sel0 = (uint32_t)p->coef.size();
                    p->coef.insert(p->coef.end(), d + 1, d + 16);
                }
                out.push_back(op);
            }
            std::sort(at, at + 4);
            for (int q = 3; q >= 0; q--) list.erase(list.begin() + at[q]);
        }
        p->ops.resize(begin);
        p->ops.insert(p->ops.end(), out.begin(), out.end());
    }

    // A 4 x 4 matrix as a real one with a phase for every row, or for every
    // column: the reals (8), then the phases (4).
    static bool real_up_to_phases(const std::vector<Cx>& m, std::vector<Cx>& out, bool* cols) {
        for (int side = 0; side < 2; side++) {
            double R[16];
            Cx f[4];
            bool ok = true;
            for (int r = 0; r < 4 && ok; r++) {
                auto at = [&](int c) { return side ? m[4 * c + r] : m[4 * r + c]; };
                int big = 0;
                for (int c = 1; c < 4; c++)
                    if (std::hypot(at(c).re, at(c).im) > std::hypot(at(big).re, at(big).im)) big = c;
                const double norm = std::hypot(at(big).re, at(big).im);
                f[r] = norm > 0.0 ? unit(at(big)).round() : Cx{1.0, 0.0};
                for (int c = 0; c < 4; c++) {
                    const Cx x = cmul(at(c), conj(f[r]));
                    ok &= std::fabs(x.im) <= 1e-15 * norm;  // rounding of the products
                    R[side ? 4 * c + r : 4 * r + c] = x.re;
                }
            }
            if (!ok) continue;
            out.clear();
            for (int i = 0; i < 16; i += 2) out.push_back(Cx{R[i], R[i + 1]});
            out.insert(out.end(), f, f + 4);
            *cols = side == 1;
            return true;
        }
        return false;
    }

    // The coefficients of a density-matrix step; swapped: its first qubit sits
    // at the second pair of positions.
    static std::vector<Cx> dm_coefs(const LGate& g, bool swapped) {
        if (!four_bits(g) || !swapped) return g.m;
        auto sw = [](int i) { return ((i & 1) << 1) | (i >> 1); };
        std::vector<Cx> out(g.m);
        const double* in = &g.m[0].re;
        double* o = &out[0].re;
        if (g.cls == GC_PAULI2) {
            for (int d = 0; d < 4; d++)
                for (int i = 0; i < 4; i++)
                    for (int k = 0; k < 4; k++) o[16 * d + 4 * i + k] = in[16 * sw(d) + 4 * sw(i) + sw(k)];
            return out;
        }
        for (size_t q = 0; q < g.m.size() / 5; q++) {
            uint32_t x;
            memcpy(&x, &in[10 * q], 4);
            x = (uint32_t)sw((int)x);
            memcpy(&o[10 * q], &x, 4);
            for (int i = 0; i < 4; i++) {
                o[10 * q + 2 + i] = in[10 * q + 2 + sw(i)];
                o[10 * q + 6 + i] = in[10 * q + 6 + sw(i)];
            }
        }
        return out;
    }
    // Where the pass holds these coefficients (a circuit's channels are often
    // the same on every qubit).
    uint32_t coefs_of(const std::vector<Cx>& m) {
        for (const auto& q : shared)
            if (q.second == m.size() && memcmp(&p->coef[q.first], m.data(), m.size() * sizeof(Cx)) == 0) return q.first;
        const uint32_t at = (uint32_t)p->coef.size();
        p->coef.insert(p->coef.end(), m.begin(), m.end());
        shared.push_back({at, m.size()});
        return at;
    }

    // A CZ (one control or two targets, one entry -1, the others 1).
    bool two_bit_sign(const LGate& g, Sign& z) const {
        if (g.k + g.nc != 2) return false;
        int minus = -1;
        for (size_t i = 0; i < g.m.size(); i++) {
            if (is(g.m[i], 1.0)) continue;
            if (!is(g.m[i], -1.0) || minus >= 0) return false;
            minus = (int)i;
        }
        if (minus < 0) return false;
        auto where = [&](int b) { return local[b] >= 0 ? (int)local[b] : 16 + (int)outside[b]; };
        for (int q = 0; q < g.k; q++) {
            z.bit[q] = where(g.tb[q]);
            z.val[q] = (minus >> q) & 1;
        }
        if (g.nc) {
            z.bit[1] = where(g.cb[0]);
            z.val[1] = g.cv[0] ? 1 : 0;
        }
        return true;
    }

    // A diagonal gate: signs become RC_NEG ops; otherwise it joins the
    // diagonal under way or, in exact passes and when it depends on more
    // than one bit outside the registers, becomes one RC_PHASE op per
    // combination of its register targets.
    template <typename Pos, typename Acc, typename Flush, typename Push>
    void diagonal(const LGate& g, const ROp& base, uint32_t rmask, uint32_t rval, uint32_t na, const Pos& pos, Acc& acc,
                  const Flush& flush, const Push& push) {
        uint32_t dmask = 0;  // entry bits held in registers
        std::vector<int> sel, selbit;
        for (int i = 0; i < g.k; i++) {
            const int l = local[g.tb[i]];
            if (l >= 0 && pos(l) >= 0) {
                dmask |= 1u << i;
            } else {
                sel.push_back(l >= 0 ? l : 16 + outside[g.tb[i]]);
                selbit.push_back(i);
            }
        }
        auto entry = [&](uint32_t reg, uint32_t e) {  // register part of the entry index, entry of the selected bits
            uint32_t x = reg;
            for (size_t q = 0; q < sel.size(); q++) x |= ((e >> q) & 1u) << selbit[q];
            return g.m[x];
        };
        auto reg_part = [&](uint32_t j) {
            uint32_t x = 0;
            for (int i = 0; i < g.k; i++)
                if (dmask & (1u << i)) x |= ((j >> pos(local[g.tb[i]])) & 1u) << i;
            return x;
        };
        bool signs = true;
        for (const Cx& c : g.m) signs &= c.im == 0.0 && (c.re == 1.0 || c.re == -1.0);
        const bool ctl_outside = base.ctl || base.gmask;
        uint32_t dep = rmask;
        for (int i = 0; i < g.k; i++)
            if (dmask & (1u << i)) dep |= 1u << pos(local[g.tb[i]]);
        // a control outside the registers is one more selected bit
        const int nsel = (int)sel.size() + __builtin_popcount(base.ctl & 0xffffu) + __builtin_popcount(base.gmask);
        int one = -1;
        if (nsel == 1) one = !sel.empty() ? sel[0] : (base.ctl & 0xffffu) ? __builtin_ctz(base.ctl & 0xffffu) : 16 + __builtin_ctz(base.gmask);
        if (!exact && !(signs && nsel > 0) && nsel <= 1) {
            if (acc.on && one >= 0 && acc.sel >= 0 && acc.sel != one) flush();
            if (!acc.on) {
                acc.on = true;
                acc.dep = 0;
                acc.sel = -1;
                acc.tab.assign(2 * na, Cx{1.0, 0.0});
            }
            if (one >= 0) acc.sel = one;
            acc.dep |= dep;
            const uint32_t cval = ctl_outside ? ((base.ctl >> 16) || base.gval ? 1u : 0u) : 0u;
            for (uint32_t e = 0; e < 2; e++)
                for (uint32_t j = 0; j < na; j++) {
                    if ((j & rmask) != rval || (ctl_outside && e != cval)) continue;
                    Cx& x = acc.tab[e * na + j];
                    x = cmul(x, entry(reg_part(j), sel.empty() ? 0u : e));
                }
            return;
        }
        for (uint32_t s2 = 0; s2 < (1u << g.k); s2++) {
            if (s2 & ~dmask) continue;
            uint32_t jm = 0;
            for (uint32_t j = 0; j < na; j++)
                if ((j & rmask) == rval && reg_part(j) == s2) jm |= 1u << j;
            if (!jm) continue;
            const uint32_t ne = 1u << sel.size();
            if (signs && !exact) {  // (exact: multiplied, as a gate alone does)
                for (uint32_t e = 0; e < ne; e++) {
                    if (entry(s2, e).re == 1.0) continue;
                    ROp op = base;
                    for (size_t q = 0; q < sel.size(); q++) {
                        const uint32_t bit = (e >> q) & 1u;
                        if (sel[q] < 16)
                            op.ctl |= (1u << sel[q]) | (bit << (16 + sel[q]));
                        else {
                            op.gmask |= 1u << (sel[q] - 16);
                            op.gval |= bit << (sel[q] - 16);
                        }
                    }
                    push(RC_NEG, jm, op);
                }
                continue;
            }
            ROp op = base;
            op.coef = (uint32_t)p->coef.size();
            bool any = false;
            for (uint32_t e = 0; e < ne; e++) {
                any |= !is(entry(s2, e), 1.0);
                p->coef.push_back(entry(s2, e));
            }
            if (!any) {
                p->coef.resize(op.coef);
                continue;
            }
            for (size_t q = 0; q < sel.size(); q++) {
                if (q < 5)
                    op.sel0 |= (uint32_t)sel[q] << (6 * q);
                else
                    op.sel1 |= (uint32_t)sel[q];
            }
            op.sel1 |= (uint32_t)sel.size() << 8;
            push(RC_PHASE, jm, op);
        }
    }
};

size_t pass_bytes(const RegPass& p, size_t coef_bytes) {
    return p.segs.size() * sizeof(RSeg) + p.ops.size() * sizeof(ROp) + p.coef.size() * coef_bytes;
}

}  // namespace

// The plan of prog[0 .. ngates).
static void reg_plan_range(const LGate* prog, size_t ngates, uint32_t nbits, int32_t precision, int tbits_max,
                           bool exact, RegPlan& out, bool dm = false, uint64_t batch_tiles = 0) {
    out.passes.clear();
    out.blob.clear();
    const size_t amp = precision == YAO_C128 ? 16 : 8, coef_bytes = precision == YAO_C128 ? 16 : 32;
    const int low = precision == YAO_C128 ? 3 : 4;  // 128-byte runs: the tile's lowest bits
    const int tbits = std::min((int)nbits, tbits_max);
    const bool whole = (int)nbits <= tbits;
    const uint64_t lowmask = whole ? 0 : ((1ull << low) - 1);
    const int cap = whole ? (int)nbits : tbits - low;
    const size_t blob_cap = precision == YAO_C128 ? kRegBlobCap : kRegBlobCap64;
    std::vector<GateBits> bits(ngates);
    uint64_t all = 0;  // the bits that gates touch
    for (size_t i = 0; i < ngates; i++) {
        bits[i] = GateBits{qubit_mask(prog[i]), need_mask(prog[i], exact), is_perm(prog[i])};
        all |= bits[i].qubits;
    }
    // Amplitudes a thread: 16 once the tiles fill the GPU twice over, else 4
    // (8 in a 2^12 tile: at most 512 threads), which shortens an op's chain
    // where the time of one CTA is the time of the pass.
    const uint64_t ntiles = 1ull << (nbits - tbits);
    // (A batch counts the tiles of all its registers, in 2^tbits_max tiles.)
    int rb = std::max(ntiles, batch_tiles) >= kManyTiles ? 4 : ((batch_tiles ? tbits_max : tbits) > 11 ? 3 : 2);
    bool four = false;
    for (size_t i = 0; i < ngates; i++) four |= four_bits(prog[i]);
    if (four) rb = 4;
    std::vector<char> used(ngates, 0);
    size_t i0 = 0, left = ngates;
    while (left) {
        // the gates of this pass (at most twice what its description holds)
        std::vector<size_t> run;
        uint64_t hi = 0;
        {
            Scan sc(exact);
            for (size_t j = i0; j < ngates && !sc.closed(all) && run.size() < 2 * blob_cap / sizeof(ROp); j++) {
                if (used[j]) continue;
                const uint64_t nh = hi | (bits[j].need & ~lowmask);
                if (!sc.free(bits[j]) || __builtin_popcountll(nh) > cap) {
                    sc.skip(bits[j]);
                    continue;
                }
                hi = nh;
                run.push_back(j);
            }
        }
        uint64_t tile = hi | lowmask;
        for (uint32_t b = 0; __builtin_popcountll(tile) < tbits; b++) tile |= 1ull << b;
        RegPass p;
        p.tbits = tbits;
        p.rb = rb;
        p.ntiles = ntiles;
        PassBuilder pb;
        pb.rb = rb;
        pb.exact = exact;
        pb.dm_form = !exact && dm;
        int nt = 0, no = 0;
        for (uint32_t b = 0; b < 64; b++) {
            pb.local[b] = pb.outside[b] = -1;
            if (b >= nbits) continue;
            if ((tile >> b) & 1) {
                p.tb[nt] = (int8_t)b;
                pb.local[b] = (int8_t)nt++;
            } else {
                pb.outside[b] = (int8_t)no++;
            }
        }
        pb.p = &p;
        // its segments, until the description is full
        std::vector<char> done(run.size(), 0);
        size_t ndone = 0, first = 0;
        while (ndone < run.size()) {
            SegPlan s;
            Scan sc(exact);
            std::vector<size_t> took;
            size_t bytes = pass_bytes(p, coef_bytes) + sizeof(RSeg);
            bool full = false;
            for (size_t j = first; j < run.size() && !full && !sc.closed(all); j++) {
                if (done[j]) continue;
                const LGate& g = prog[run[j]];
                if (!sc.free(bits[run[j]]) || !pb.fits(s, g)) {
                    sc.skip(bits[run[j]]);
                    continue;
                }
                // a diagonal may become one op per combination of its register targets;
                // a channel's coefficients are there already, mostly
                // (a layer of four matrices: their reals and a diagonal)
                const size_t more = !exact && rb == 4 && g.cls == GC_DENSE && g.k == 1 ? 3 * coef_bytes : 0;
                const size_t nb = (g.cls == GC_DIAG ? std::min<size_t>(1u << g.k, 16) : 1) * sizeof(ROp) + more +
                                  (g.cls >= GC_CHAN1 ? std::min<size_t>(g.m.size(), 4) : g.m.size()) * coef_bytes;
                if (bytes + nb > blob_cap && !(p.ops.empty() && s.gates.empty())) {
                    full = true;
                    break;
                }
                bytes += nb;
                pb.add(s, g);
                took.push_back(j);
            }
            if (took.empty()) break;  // the description is full
            // The count above is a guess: a diagonal may bring a table, a
            // channel more coefficients.  Without its last gates the segment
            // fits (a gate alone always does).
            const size_t segs0 = p.segs.size(), ops0 = p.ops.size(), coef0 = p.coef.size(), shared0 = pb.shared.size();
            pb.emit(s);
            while (pass_bytes(p, coef_bytes) > blob_cap && (took.size() > 1 || ops0 > 0)) {
                p.segs.resize(segs0);
                p.ops.resize(ops0);
                p.coef.resize(coef0);
                pb.shared.resize(shared0);
                full = true;
                took.resize(took.size() * 3 / 4);
                if (took.empty()) break;
                s = SegPlan();
                for (size_t j : took) pb.add(s, prog[run[j]]);
                pb.emit(s);
            }
            for (size_t j : took) done[j] = 1;
            ndone += took.size();
            while (first < run.size() && done[first]) first++;
            if (full) break;
        }
        for (size_t j = 0; j < run.size(); j++)
            if (done[j]) {
                used[run[j]] = 1;
                left--;
            }
        while (i0 < ngates && used[i0]) i0++;
        if (p.ops.empty()) continue;
        // the tile leaves from the last segment's registers: whole 128-byte
        // runs a warp need the low positions on the lanes
        if (tbits - rb >= low) {
            bool lowest = false;
            for (int q = 0; q < rb; q++) lowest |= p.segs.back().sorted[q] < low;
            if (lowest) {
                RSeg sg;
                memset(&sg, 0, sizeof(sg));
                sg.op_begin = sg.op_end = (int32_t)p.ops.size();
                for (int q = 0; q < rb; q++) sg.sorted[q] = sg.order[q] = (int8_t)(tbits - rb + q);
                p.segs.push_back(sg);
            }
        }
        out.passes.push_back(std::move(p));
    }
    // one packed description for the whole plan
    size_t total = 0;
    for (RegPass& p : out.passes) {
        p.blob_off = total;
        p.blob_bytes = pass_bytes(p, coef_bytes);
        total += (p.blob_bytes + 255) / 256 * 256;
    }
    out.blob.assign(total, 0);
    for (RegPass& p : out.passes) {
        unsigned char* d = out.blob.data() + p.blob_off;
        memcpy(d, p.segs.data(), p.segs.size() * sizeof(RSeg));
        d += p.segs.size() * sizeof(RSeg);
        memcpy(d, p.ops.data(), p.ops.size() * sizeof(ROp));
        d += p.ops.size() * sizeof(ROp);
        for (const Cx& c : p.coef) {
            if (amp == 16) {
                memcpy(d, &c, 16);
            } else {
                const float hr = (float)c.re, hi = (float)c.im;
                const float f[8] = {hr, hr, hi, hi, (float)(c.re - (double)hr), (float)(c.re - (double)hr),
                                    (float)(c.im - (double)hi), (float)(c.im - (double)hi)};
                memcpy(d, f, 32);
            }
            d += coef_bytes;
        }
    }
}

void reg_plan(const std::vector<LGate>& prog, uint32_t nbits, int32_t precision, int tbits, bool exact, RegPlan& out,
              uint64_t batch_tiles) {
    reg_plan_range(prog.data(), prog.size(), nbits, precision, tbits, exact, out, false, batch_tiles);
}

// ================================================================== launch

int kernel_fit(Ctx* ctx, const void* kernel, KernelFit* out, bool all) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, KernelFit> known;
    std::lock_guard<std::mutex> g(mu);
    KernelFit& f = known[{ctx->device, kernel}];
    if (!f.limit) {
        int v = 0;
        cudaFuncAttributes fa;
        YAO_CUDA(cudaDeviceGetAttribute(&f.total, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device));
        YAO_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
        YAO_CUDA(cudaFuncGetAttributes(&fa, kernel));
        f.fixed = (int)fa.sharedSizeBytes;
        YAO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v - f.fixed));
        if (all)
            YAO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        f.limit = v - f.fixed;
    }
    *out = f;
    return YAO_OK;
}

template <typename A, bool EXACT, int RB, bool DMX>
static int launch_k(Ctx* ctx, void* st, RHdr& hdr, const uint4* blob, size_t blob_bytes, const CUtensorMap& tmap) {
    auto kern = k_reg_tiles<A, EXACT, RB, DMX>;
    KernelFit fit;
    int sf = kernel_fit(ctx, (const void*)kern, &fit, true);
    if (sf) return sf;
    const size_t tile = sizeof(typename A::Amp) << hdr.tbits;
    const unsigned threads = std::max(32u, 1u << (hdr.tbits - RB));
    // as many CTAs as the registers allow, then as many tile buffers as fit
    auto ctas = [&](int nbuf) {
        const size_t per = (size_t)nbuf * tile + blob_bytes + 1024 + fit.fixed + 1024;
        const size_t limit = (size_t)reg_ctas<A, RB>() * kRegThreads<A, RB> / threads;
        return std::min<size_t>((size_t)fit.total / per, std::max<size_t>(1, limit));
    };
    hdr.nbuf = 1;
    while (hdr.use_tma && hdr.nbuf < 4 && ctas(hdr.nbuf + 1) == ctas(hdr.nbuf)) hdr.nbuf++;
    const size_t smem = (size_t)hdr.nbuf * tile + blob_bytes + 1024;
    if (smem > (size_t)fit.limit) return fail(YAO_ERR_UNSUPPORTED, "register pass does not fit an SM");
    int per_sm = 0;
    YAO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)threads, smem));
    if (per_sm < 1) return fail(YAO_ERR_UNSUPPORTED, "register pass does not fit an SM");
    const unsigned grid = (unsigned)std::min<uint64_t>(hdr.ntiles, (uint64_t)per_sm * (uint64_t)ctx->num_sms);
    kern<<<grid, threads, smem, ctx->stream>>>((typename A::Amp*)st, hdr, blob, ctx->d_err, tmap);
    return YAO_OK;
}

template <typename A, bool EXACT, bool DMX>
static int launch_rb(Ctx* ctx, void* st, int rb, RHdr& hdr, const uint4* blob, size_t bytes, const CUtensorMap& tmap) {
    if (rb == 4) return launch_k<A, EXACT, 4, DMX>(ctx, st, hdr, blob, bytes, tmap);
    if (rb == 3) return launch_k<A, EXACT, 3, DMX>(ctx, st, hdr, blob, bytes, tmap);
    return launch_k<A, EXACT, 2, DMX>(ctx, st, hdr, blob, bytes, tmap);
}

static void pass_header(const RegPass& p, RHdr& h) {
    memset(&h, 0, sizeof(h));
    h.tbits = p.tbits;
    h.nsegs = (int32_t)p.segs.size();
    h.blob16 = (int32_t)(p.blob_bytes / 16);
    h.ops16 = (int32_t)(p.segs.size() * sizeof(RSeg) / 16);
    h.coef16 = h.ops16 + (int32_t)(p.ops.size() * sizeof(ROp) / 16);
    h.ntiles = (uint32_t)p.ntiles;
    h.nbuf = 1;
    memcpy(h.tb, p.tb, sizeof(h.tb));
}

int reg_launch(Ctx* ctx, void* st, uint32_t nbits, int32_t precision, bool exact, const RegPlan& plan, size_t first,
               size_t step, bool* queued) {
    if (queued) *queued = false;
    if (plan.passes.empty()) return YAO_OK;
    unsigned char* dblob = nullptr;
    YAO_CUDA(alloc_async(ctx, (void**)&dblob, plan.blob.size()));
    YAO_CUDA(cudaMemcpyAsync(dblob, plan.blob.data(), plan.blob.size(), cudaMemcpyHostToDevice, ctx->stream));
    if (queued) *queued = true;
    const size_t amp = precision == YAO_C128 ? 16 : 8;
    int s = YAO_OK;
    for (size_t i = first; i < plan.passes.size() && !s; i += step) {
        const RegPass& p = plan.passes[i];
        RHdr h;
        pass_header(p, h);
        CUtensorMap tmap;
        memset(&tmap, 0, sizeof(tmap));
        // (one tile: nothing to overlap, and no wait that could give up)
        h.use_tma = p.ntiles > 1 && tma_enabled() && tma_make_plan(p.tb, p.tbits, nbits, amp, st, h.tma, &tmap) ? 1 : 0;
        if (h.use_tma) ctx->err_unread.store(true);
        const uint4* blob = (const uint4*)(dblob + p.blob_off);
        bool dmx = false;
        for (const ROp& op : p.ops) dmx |= (op.head & 0xffu) >= RC_CHAN1;
        {
            ProfScope prof(ctx, exact ? "reg_pass_exact" : "reg_pass_fused",
                           (double)p.ntiles * (double)((uint64_t)1 << p.tbits) * 2.0 * (double)amp);
            if (precision == YAO_C128)
                s = exact ? (dmx ? launch_rb<A128<true>, true, true>(ctx, st, p.rb, h, blob, p.blob_bytes, tmap)
                                 : launch_rb<A128<true>, true, false>(ctx, st, p.rb, h, blob, p.blob_bytes, tmap))
                          : (dmx ? launch_rb<A128<false>, false, true>(ctx, st, p.rb, h, blob, p.blob_bytes, tmap)
                                 : launch_rb<A128<false>, false, false>(ctx, st, p.rb, h, blob, p.blob_bytes, tmap));
            else
                s = launch_rb<A64, false, false>(ctx, st, p.rb, h, blob, p.blob_bytes, tmap);
        }
        ctx->launches++;
        if (!s && cudaPeekAtLastError() != cudaSuccess) s = cuda_fail(cudaGetLastError(), "register pass launch");
    }
    cudaFreeAsync(dblob, ctx->stream);
    return s;
}

template <typename A, bool EXACT, int RB>
static int launch_batch_level(Ctx* ctx, const RBatchPass* passes, const uint32_t* owner, unsigned ctas, int tbits,
                              size_t blob_bytes) {
    auto kern = k_reg_batch<A, EXACT, RB>;
    const size_t smem = (sizeof(typename A::Amp) << tbits) + blob_bytes + 1024;
    KernelFit fit;
    int s = kernel_fit(ctx, (const void*)kern, &fit);
    if (s) return s;
    if (smem > (size_t)fit.limit) return fail(YAO_ERR_UNSUPPORTED, "register pass does not fit an SM");
    kern<<<ctas, std::max(32u, 1u << (tbits - RB)), smem, ctx->stream>>>(passes, owner);
    ctx->launches++;
    YAO_CUDA(cudaGetLastError());
    return YAO_OK;
}

// Level after level: one launch runs the next pass of every register that has
// one left, a CTA a tile (plain loads: the registers sit in L2).  The launch
// order is the only wait between a register's passes.  Measured on 60 layered
// circuits, 10 to 18 qubits and 10 to 40 layers, FUSED: 19 launches, 1.6 ms
// on the device against 2.9 of the block passes; planning, which the rest of
// the call mostly is, 1.6 ms on 16 host threads.
int reg_batch(Ctx* ctx, const std::vector<RegPlan>& plans, const std::vector<Reg*>& regs, bool exact) {
    const int32_t precision = regs[0]->precision;
    const size_t amp = precision == YAO_C128 ? 16 : 8;
    constexpr uint32_t kMaxCtas = 2048;  // a register's CTAs in a launch
    size_t levels = 0, npasses = 0, nowner = 0, nblob = 0;
    std::vector<size_t> blob_at(plans.size());
    for (size_t c = 0; c < plans.size(); c++) {
        levels = std::max(levels, plans[c].passes.size());
        npasses += plans[c].passes.size();
        for (const RegPass& p : plans[c].passes) nowner += (size_t)std::min<uint64_t>(p.ntiles, kMaxCtas);
        blob_at[c] = nblob;
        nblob += (plans[c].blob.size() + 255) / 256 * 256;
    }
    if (npasses == 0) return YAO_OK;
    const size_t b_pass = (npasses * sizeof(RBatchPass) + 255) / 256 * 256, b_owner = (nowner * 4 + 255) / 256 * 256;
    const size_t total = nblob + b_pass + b_owner;
    int st;
    if ((st = grow_host(&ctx->batch_host, &ctx->batch_host_bytes, total))) return st;
    if ((st = grow_dev(ctx, &ctx->batch_dev, &ctx->batch_dev_bytes, total))) return st;
    char* h = (char*)ctx->batch_host;
    char* d = (char*)ctx->batch_dev;
    for (size_t c = 0; c < plans.size(); c++) memcpy(h + blob_at[c], plans[c].blob.data(), plans[c].blob.size());
    RBatchPass* hp = (RBatchPass*)(h + nblob);
    uint32_t* ho = (uint32_t*)(h + nblob + b_pass);
    struct Level {
        size_t owner;
        uint32_t ctas;
        int tbits, rb;
        size_t blob;
        double bytes;
    };
    std::vector<Level> todo;
    size_t at = 0, own = 0;
    for (size_t l = 0; l < levels; l++) {
        Level lv{own, 0, 0, 0, 0, 0.0};
        for (size_t c = 0; c < plans.size(); c++) {
            if (l >= plans[c].passes.size()) continue;
            const RegPass& p = plans[c].passes[l];
            RBatchPass& b = hp[at];
            memset(&b, 0, sizeof(b));
            pass_header(p, b.hdr);
            b.state = (uint64_t)(uintptr_t)regs[c]->d;
            b.blob = (uint64_t)(uintptr_t)(d + blob_at[c] + p.blob_off);
            b.cta0 = lv.ctas;
            b.ctas = (uint32_t)std::min<uint64_t>(p.ntiles, kMaxCtas);
            for (uint32_t q = 0; q < b.ctas; q++) ho[own++] = (uint32_t)at;
            lv.ctas += b.ctas;
            lv.tbits = std::max(lv.tbits, p.tbits);
            lv.rb = p.rb;
            lv.blob = std::max(lv.blob, p.blob_bytes);
            lv.bytes += (double)p.ntiles * (double)(1ull << p.tbits) * 2.0 * (double)amp;
            at++;
        }
        todo.push_back(lv);
    }
    YAO_CUDA(cudaMemcpyAsync(d, h, total, cudaMemcpyHostToDevice, ctx->stream));
    const RBatchPass* dp = (const RBatchPass*)(d + nblob);
    const uint32_t* dow = (const uint32_t*)(d + nblob + b_pass);
    for (const Level& lv : todo) {
        ProfScope prof(ctx, exact ? "reg_batch_exact" : "reg_batch_fused", lv.bytes);
        const uint32_t* o = dow + lv.owner;
        if (precision != YAO_C128)
            st = lv.rb == 4 ? launch_batch_level<A64, false, 4>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob)
                            : launch_batch_level<A64, false, 2>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob);
        else if (exact)
            st = lv.rb == 4 ? launch_batch_level<A128<true>, true, 4>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob)
                            : launch_batch_level<A128<true>, true, 2>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob);
        else
            st = lv.rb == 4 ? launch_batch_level<A128<false>, false, 4>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob)
                            : launch_batch_level<A128<false>, false, 2>(ctx, dp, o, lv.ctas, lv.tbits, lv.blob);
        if (st) break;
    }
    // (the tables are free for the next call)
    const cudaError_t ce = cudaStreamSynchronize(ctx->stream);
    if (!st && ce != cudaSuccess) return cuda_fail(ce, "batched register passes");
    return st;
}

// ==================================================== gate-by-gate programs

// Seconds (estimate) of a gate's own launch: 3 us and its amplitudes, read
// and written, at 6.2 TB/s.
static double gate_seconds(const LGate& g, double state_bytes) {
    double part = 1.0;
    if (g.cls == GC_SWAP) part = 0.5;
    if (g.cls == GC_DIAG) {
        size_t n = 0;
        for (const Cx& c : g.m) n += !is(c, 1.0);
        part = (double)n / (double)g.m.size();
    }
    return 3e-6 + 2.0 * state_bytes * part / (double)(1ull << g.nc) / 6.2e12;
}
// FP64 operations of an exact op on every amplitude
static double gate_flops(const LGate& g) {
    return (g.cls == GC_DIAG ? 3.0 : g.cls == GC_DENSE ? (g.k == 1 ? 14.0 : 30.0) : 0.0) / (double)(1ull << g.nc);
}

int plain_run(Ctx* ctx, Reg* r, const std::vector<LGate>& prog) {
    const uint32_t n = r->nbits;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    YAO_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    const bool passes = r->precision == YAO_C128 && reg_width(n) && cs == cudaStreamCaptureStatusNone;
    const double bytes = (double)r->bytes(), amps = (double)(1ull << n);
    for (size_t i = 0; i < prog.size();) {
        size_t end = i;  // the gates from i on that a register pass can run
        while (passes && end < prog.size() && reg_gate(prog[end])) end++;
        if (end - i >= 2) {
            // Passes where they are estimated to be faster: 8 us and the state
            // read and written at 5.2 TB/s each, and the gates' arithmetic at
            // 1e13 operations a second (measured: 22 passes of 696 gates,
            // n = 25, 23 ms).  A few gates that touch a fraction of a large
            // state, and gates that share no pass, stay launches of their own.
            RegPlan plan;
            reg_plan_range(&prog[i], end - i, n, YAO_C128, 11, true, plan);
            double alone = 0.0, joint = (double)plan.passes.size() * (8e-6 + 2.0 * bytes / 5.2e12);
            for (size_t q = i; q < end; q++) {
                alone += gate_seconds(prog[q], bytes);
                joint += gate_flops(prog[q]) * amps / 1e13;
            }
            if (joint < alone) {
                bool queued;
                int s = reg_launch(ctx, r->d, n, YAO_C128, true, plan, 0, 1, &queued);
                if (s && (queued || s != YAO_ERR_OUT_OF_MEMORY)) return s;
                if (!s) {
                    i = end;
                    continue;
                }
                clear_error();  // no memory for the description: the launches need none
            }
        }
        for (end = std::max(i + 1, end); i < end; i++) {
            int s = launch_gate(ctx, r->d, r->precision, n, prog[i]);
            if (s) return s;
        }
    }
    return YAO_OK;
}

// ==================================================== density matrices

// entry (r, c) of a lowered Kraus operator
static Cx entry_of(const LGate& g, int r, int c) {
    const int nl = 1 << g.k;
    if (g.cls == GC_DIAG) return r == c ? g.m[r] : Cx{0.0, 0.0};
    return g.m[(size_t)r * nl + c];
}

static LGate dm_gate_on(const DMStep& s, int cls, int k) {
    LGate g;
    g.cls = cls;
    g.k = 2 * k;
    for (int i = 0; i < k; i++) {
        g.tb[2 * i] = s.cols[0].tb[i];
        g.tb[2 * i + 1] = s.rows[0].tb[i];
    }
    return g;
}

// The Kraus sum of a channel as GC_CHAN1 / GC_CHAN2: every operator has one
// non-zero entry at most in a row, the same ones in K and conj(K), all real or
// all imaginary (two imaginary weights multiply like real ones of opposite
// sign).  False for other channels.
static bool kraus_step(const std::vector<DMStep>& steps, size_t at, std::vector<LGate>& cache, LGate& g) {
    const DMStep& s = steps[at];
    if (s.like >= 0) {  // the same channel elsewhere: its coefficients, or none
        if (cache[s.like].m.empty()) return false;
        g = dm_gate_on(s, cache[s.like].cls, s.rows[0].k);
        g.m = cache[s.like].m;
        return true;
    }
    if (s.rows.empty()) return false;
    const int k = s.rows[0].k, nl = 1 << k;
    if (k < 1 || k > 2 || s.rows.size() > (size_t)kMaxKraus) return false;
    g = dm_gate_on(s, k == 1 ? GC_CHAN1 : GC_CHAN2, k);
    for (size_t q = 0; q < s.rows.size(); q++) {
        int src[4];
        double r[4] = {0, 0, 0, 0}, c[4] = {0, 0, 0, 0};
        const bool diag = s.rows[q].cls == GC_DIAG;
        bool real = true, imag = true;
        for (int a = 0; a < nl; a++) {
            src[a] = -1;
            for (int b = 0; b < nl; b++) {
                const Cx x = entry_of(s.rows[q], a, b), y = entry_of(s.cols[q], a, b);
                if (is(x, 0.0) != is(y, 0.0)) return false;
                // a diagonal's zeros multiply too (an infinity becomes NaN)
                if (diag ? a != b : is(x, 0.0)) continue;
                if (src[a] >= 0) return false;
                src[a] = b;
                real &= x.im == 0.0 && y.im == 0.0;
                imag &= x.re == 0.0 && y.re == 0.0;
            }
        }
        if (!real && (diag || !imag)) return false;
        for (int a = 0; a < nl; a++) {
            if (src[a] < 0) continue;
            const Cx x = entry_of(s.rows[q], a, src[a]), y = entry_of(s.cols[q], a, src[a]);
            r[a] = real ? x.re : -x.im;
            c[a] = real ? y.re : y.im;
        }
        uint32_t type = 0;
        if (k == 1) {
            if (src[0] == 0 && src[1] == 1) type = 0;
            else if (src[0] == 1 && src[1] == 0) type = 1;
            else if (src[0] == 1 && src[1] < 0) type = 2;
            else if (src[0] < 0 && src[1] == 0) type = 3;
            else return false;
        } else {
            type = (uint32_t)src[0];
            for (int a = 0; a < nl; a++)
                if (src[a] < 0 || src[a] != (a ^ src[0])) return false;
        }
        Cx head{0.0, 0.0};
        memcpy(&head.re, &type, 4);
        g.m.push_back(head);
        for (int a = 0; a < nl; a += 2) g.m.push_back(Cx{r[a], r[a + 1]});
        for (int a = 0; a < nl; a += 2) g.m.push_back(Cx{c[a], c[a + 1]});
    }
    cache[at] = g;
    return !g.m.empty();
}

// PLAIN steps on a density matrix.  Runs of gates and channels that the exact
// register passes hold (the same products and sums in the same order as the
// lone passes) share passes where the passes cost less; others run alone.
int dm_plain_run(Ctx* ctx, DM* d, const std::vector<DMStep>& steps) {
    const uint32_t nb = 2 * d->nbits;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    YAO_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    const bool passes = reg_width(nb) && cs == cudaStreamCaptureStatusNone;
    const double bytes = (double)d->bytes(), entries = (double)(1ull << nb);
    auto alone_step = [&](const DMStep& s) -> int {
        if (s.channel && s.like >= 0) {
            std::vector<LGate> rows = steps[s.like].rows, cols = steps[s.like].cols;
            for (LGate& g : rows) std::copy(s.rows[0].tb, s.rows[0].tb + kMaxTargets, g.tb);
            for (LGate& g : cols) std::copy(s.cols[0].tb, s.cols[0].tb + kMaxTargets, g.tb);
            return launch_dm_channel(ctx, d, rows, cols, {}, {});
        }
        if (s.channel) return launch_dm_channel(ctx, d, s.rows, s.cols, {}, {});
        for (size_t i = 0; i < s.rows.size(); i++) {
            int st = launch_dm_gate(ctx, d, s.rows[i], s.cols[i]);
            if (st) return st;
        }
        return YAO_OK;
    };
    std::vector<LGate> cache(steps.size());
    for (size_t i = 0; i < steps.size();) {
        // the steps from i on that a register pass can run
        std::vector<LGate> prog;
        size_t end = i;
        double alone = 0.0, flops = 0.0;
        for (; passes && end < steps.size(); end++) {
            const DMStep& s = steps[end];
            if (s.channel) {
                LGate g;
                if (!kraus_step(steps, end, cache, g)) break;
                // measured: 1-qubit channels at 5.3 TB/s, 2-qubit ones at 1.8
                alone += 3e-6 + 2.0 * bytes / (g.cls == GC_CHAN1 ? 5.3e12 : 1.8e12);
                flops += 6.0 * (double)(s.like >= 0 ? steps[s.like] : s).rows.size();
                prog.push_back(std::move(g));
                continue;
            }
            bool ok = true;
            for (const LGate& g : s.rows) ok &= reg_gate(g);
            if (!ok) break;
            for (size_t q = 0; q < s.rows.size(); q++) {
                alone += 3e-6 + 2.0 * bytes / 6.2e12;
                flops += 2.0 * gate_flops(s.rows[q]);
                prog.push_back(s.rows[q]);
                prog.push_back(s.cols[q]);
            }
        }
        if (end - i >= 2) {
            // the rule of plain_run
            RegPlan plan;
            reg_plan_range(prog.data(), prog.size(), nb, YAO_C128, 11, true, plan);
            if ((double)plan.passes.size() * (8e-6 + 2.0 * bytes / 5.2e12) + flops * entries / 1e13 < alone) {
                bool queued;
                int s = reg_launch(ctx, d->d, nb, YAO_C128, true, plan, 0, 1, &queued);
                if (s && (queued || s != YAO_ERR_OUT_OF_MEMORY)) return s;
                if (!s) {
                    i = end;
                    continue;
                }
                clear_error();  // as in plain_run
            }
        }
        for (end = std::max(i + 1, end); i < end; i++) {
            int s = alone_step(steps[i]);
            if (s) return s;
        }
    }
    return YAO_OK;
}

// FUSED steps on a density matrix; *done = false where a step has no form here
// (three or more targets, other 2-qubit channels): the block passes take it.
// Measured on 12 qubits (256 MiB), eight layers of rotations, CZ (a channel
// after each) and dampings: block passes 13.5 ms, these 5.3 (4.4 on the
// device, bound by double-precision multiply-adds: a complex 4 x 4 step takes
// 16 an entry, a real one with phases 12).
int dm_fused_run(Ctx* ctx, DM* d, const std::vector<DMStep>& steps, bool* done) {
    *done = false;
    const uint32_t nb = 2 * d->nbits;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    YAO_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    if (!reg_width(nb) || cs != cudaStreamCaptureStatusNone) return YAO_OK;
    // Everything on one qubit is a 4 x 4 superoperator on its column and row
    // bit (they multiply together), a 2-qubit Pauli-type channel four real
    // 4 x 4 matrices; other gates act on row and column bits apart.
    std::vector<LGate> prog;
    std::vector<std::vector<Cx>> cache(steps.size());
    for (size_t si = 0; si < steps.size(); si++) {
        const DMStep& s = steps[si];
        const int k = s.rows[0].k, nl = 1 << k;
        if (s.like >= 0) {
            LGate g = dm_gate_on(s, k == 1 ? GC_DENSE : GC_PAULI2, k);
            g.m = cache[s.like];
            prog.push_back(std::move(g));
            continue;
        }
        if (!s.channel && (k > 1 || s.rows[0].nc || s.rows.size() > 1)) {
            for (size_t i = 0; i < s.rows.size(); i++) {
                if (!reg_gate(s.rows[i])) return YAO_OK;
                prog.push_back(s.rows[i]);
                prog.push_back(s.cols[i]);
            }
            continue;
        }
        auto at = [&](const LGate& g, int r, int c) {
            return g.cls == GC_X ? Cx{r != c ? 1.0 : 0.0, 0.0} : entry_of(g, r, c);
        };
        if (k < 1 || k > 2) return YAO_OK;
        // S[(a, b), (c, e)] = sum_q K_q[a][c] conj(K_q)[b][e], (a, b) at b + nl a
        std::vector<Cx> S((size_t)nl * nl * nl * nl, Cx{0.0, 0.0});
        for (size_t q = 0; q < s.rows.size(); q++)
            for (int a = 0; a < nl; a++)
                for (int b = 0; b < nl; b++)
                    for (int c = 0; c < nl; c++)
                        for (int e = 0; e < nl; e++) {
                            const Cx t = cmul(at(s.rows[q], a, c), at(s.cols[q], b, e));
                            Cx& x = S[(size_t)(b + nl * a) * nl * nl + (e + nl * c)];
                            x.re += t.re;
                            x.im += t.im;
                        }
        if (k == 1) {
            LGate g = dm_gate_on(s, GC_DENSE, 1);
            cache[si] = S;
            g.m = std::move(S);
            prog.push_back(std::move(g));
            continue;
        }
        LGate g = dm_gate_on(s, GC_PAULI2, 2);
        g.m.assign(32, Cx{0.0, 0.0});
        double* m = &g.m[0].re;
        for (int a = 0; a < 4; a++)
            for (int b = 0; b < 4; b++)
                for (int c = 0; c < 4; c++)
                    for (int e = 0; e < 4; e++) {
                        const Cx x = S[(size_t)(b + 4 * a) * 16 + (e + 4 * c)];
                        if (is(x, 0.0)) continue;
                        if ((a ^ c) != (b ^ e) || x.im != 0.0) return YAO_OK;
                        m[16 * (a ^ b) + 4 * a + c] = x.re;
                    }
        cache[si] = g.m;
        prog.push_back(std::move(g));
    }
    std::vector<LGate> work;
    fuse_two_qubit(prog, nb, work);
    if (!reg_supported(work, nb)) return YAO_OK;
    RegPlan plan;
    reg_plan_range(work.data(), work.size(), nb, YAO_C128, 11, false, plan, true);
    int s = reg_launch(ctx, d->d, nb, YAO_C128, false, plan, 0, 1);
    if (s) return s;
    *done = true;
    return ctx->err_unread.load() ? read_device_err(ctx, "density-matrix apply") : YAO_OK;
}

}  // namespace yao
