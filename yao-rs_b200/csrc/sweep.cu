// sweep.cu — energies and adjoint gradients (src/ad.rs:75-156) of one or many
// parameter vectors of one circuit, over register-held tiles.
//
// The 1-qubit gates between the gates that touch their qubit form a run.  For
// a generator G of one of its gates, with W the product of the run's later
// gates, the dot taken after that gate is Re <lambda | W G W^dagger psi> on
// the states after the whole run; W G W^dagger is an anti-Hermitian 2 x 2
// matrix, so every dot of the run is a combination of four sums over the
// run's amplitude pairs,
//     Im conj(l0) x0, Im conj(l1) x1, Re, Im of conj(l0) x1 -+ conj(l1) x0,
// which do not depend on the parameters.  The sweep over the states measures
// these sums and applies one matrix a run; products of gates, and gradients
// from the sums, are computed per set and run by two small kernels.  The
// states of all sets lie back to back and share one op list; only a run's
// matrix is the set's own.
//
// A pass takes 2^11-amplitude tiles of psi and lambda.  Each thread holds 8
// amplitudes of both that differ in three tile positions and applies a
// segment's ops in registers; tiles change hands between segments in shared
// memory, and enter and leave through registers.  What bounds it: per run 36
// (44 without a real first column) FP64 instructions a pair beside an op's
// own latency, at 16 warps an SM.  Large batches go through in groups whose
// states stay in the L2 cache.  Against one launch a gate over all sets (13
// qubits, 208 parameters, 192 sets): 24.6 -> 1.7 ms a call, of which the
// sweep is 0.76 ms and the forward passes 0.47.  Against the tiled sweep of
// ad_tiles.cu (22 qubits, 352 parameters): 4.14 -> 2.86 ms.
#include "sweep.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>

#include "device_common.cuh"
#include "tma_sm100.cuh"

namespace yao {

constexpr int kSB = 3;                 // register bits: 8 amplitudes of psi and of lambda a thread
constexpr int kSTile = 11;             // tile bits
constexpr int kSThreads = 1 << (kSTile - kSB);
constexpr int kSLow = 3;               // 128-byte runs
constexpr int kSMaxRuns = 40;          // runs of a pass (their sums and matrices in shared memory)
constexpr int kSMaxOps = 160;          // ops of a pass
constexpr int kSMaxSkipped = 1024;     // steps a pass's scan skips: an idle qubit does not take it to the circuit's end

enum SCode : uint32_t {
    SC_RUN = 0,    // + position: the run's matrix (and sums); pairs in the mask swap first where the controls match
    SC_RUNC = 4,   // + position: the same, first column real
    SC_X = 8,      // + position: swaps the masked pairs
    SC_SWAP = 12,  // positions 0 and 1
    SC_NEG = 13    // the masked amplitudes times -1
};

// head: code, mask in bits 16..23; run: the run's place in the pass; ctl: mask
// and value on the thread's tile positions; gmask / gval: on the tile's number
struct SOp {
    uint32_t head, run, ctl, gmask, gval, pad[3];
};
struct SSeg {
    int32_t op_begin, op_end;
    int8_t sorted[4], order[4];
};
static_assert(sizeof(SOp) == 32 && sizeof(SSeg) == 16, "staged as 16-byte words");

struct SHdr {
    int32_t n, tbits, nsegs, nops, nruns, nruns_all;
    uint32_t ntiles;            // per set
    uint32_t per_set, nunits;   // CTAs' work units: per_set of them a set
    int32_t run[kSMaxRuns];     // the pass's runs
    int8_t tb[16];
};

__device__ __forceinline__ double2 s_mul(double2 a, double2 x) {
    return make_double2(fma(a.x, x.x, -a.y * x.y), fma(a.x, x.y, a.y * x.x));
}
__device__ __forceinline__ double2 s_mad(double2 c, double2 a, double2 x) {
    return make_double2(fma(a.x, x.x, fma(-a.y, x.y, c.x)), fma(a.x, x.y, fma(a.y, x.x, c.y)));
}

template <int P, bool RC>
__device__ __forceinline__ void s_apply(const double2* m, double2 (&v)[1 << kSB]) {
    const double2 a = m[0], b = m[1], c = m[2], d = m[3];
#pragma unroll
    for (int j = 0; j < (1 << kSB); j++) {
        if (j & (1 << P)) continue;
        const double2 w = v[j], x = v[j | (1 << P)];
        if (RC) {
            const double2 u = s_mul(b, x), y = s_mul(d, x);
            v[j] = make_double2(fma(a.x, w.x, u.x), fma(a.x, w.y, u.y));
            v[j | (1 << P)] = make_double2(fma(c.x, w.x, y.x), fma(c.x, w.y, y.y));
        } else {
            v[j] = s_mad(s_mul(a, w), b, x);
            v[j | (1 << P)] = s_mad(s_mul(c, w), d, x);
        }
    }
}

template <int P>
__device__ __forceinline__ void s_x(double2 (&v)[1 << kSB], uint32_t jm) {
#pragma unroll
    for (int j = 0; j < (1 << kSB); j++) {
        if (j & (1 << P)) continue;
        if (!((jm >> j) & 1)) continue;
        const double2 w = v[j];
        v[j] = v[j | (1 << P)];
        v[j | (1 << P)] = w;
    }
}

// The four sums of a run over the thread's pairs, summed over the warp down
// to two lanes a value, added to the warp's accumulators acc[0..7] (value v
// in 2 v and 2 v + 1).
template <int P>
__device__ __forceinline__ void s_sums(const double2 (&x)[1 << kSB], const double2 (&l)[1 << kSB], bool mine, double* acc) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int j = 0; j < (1 << kSB); j++) {
        if (j & (1 << P)) continue;
        const double2 x0 = x[j], x1 = x[j | (1 << P)], l0 = l[j], l1 = l[j | (1 << P)];
        s0 = fma(l0.x, x0.y, fma(-l0.y, x0.x, s0));
        s1 = fma(l1.x, x1.y, fma(-l1.y, x1.x, s1));
        s2 = fma(l0.x, x1.x, fma(l0.y, x1.y, fma(-l1.x, x0.x, fma(-l1.y, x0.y, s2))));
        s3 = fma(l0.x, x1.y, fma(-l0.y, x1.x, fma(-l1.y, x0.x, fma(l1.x, x0.y, s3))));
    }
    if (!mine) s0 = s1 = s2 = s3 = 0.0;
    const uint32_t lane = threadIdx.x & 31;
    const bool h = lane & 16, g = lane & 8;
    double a = h ? s2 : s0, b = h ? s3 : s1;
    a += __shfl_xor_sync(0xffffffffu, h ? s0 : s2, 16);
    b += __shfl_xor_sync(0xffffffffu, h ? s1 : s3, 16);
    double v = g ? b : a;
    v += __shfl_xor_sync(0xffffffffu, g ? a : b, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if ((lane & 6) == 0) acc[(lane >> 3) * 2 + (lane & 1)] += v;
}

// One pass.  BACK: psi and lambda with the runs' sums; else psi alone.
template <bool BACK>
__global__ void __launch_bounds__(kSThreads, 2)
    k_sweep(double2* __restrict__ psi, double2* __restrict__ lam, const __grid_constant__ SHdr hdr,
            const uint4* __restrict__ gblob, const double2* __restrict__ coef, double* __restrict__ partial) {
    constexpr int NA = 1 << kSB;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int8_t tb[16];
    const uint32_t T = 1u << hdr.tbits, nw = blockDim.x >> 5;
    double2* sp = (double2*)smem;                                  // exchange buffers
    double2* sl = sp + T;
    double2* cf = sp + (BACK ? 2 : 1) * (size_t)T;                 // the set's matrices, four entries a run
    uint4* blob = (uint4*)(cf + 4 * hdr.nruns);
    double* acc = (double*)(blob + hdr.nsegs + 2 * hdr.nops);      // [run][warp][8]
    for (int i = threadIdx.x; i < hdr.nsegs + 2 * hdr.nops; i += blockDim.x) blob[i] = gblob[i];
    if (threadIdx.x < 16) tb[threadIdx.x] = hdr.tb[threadIdx.x];
    __syncthreads();
    const uint4* ops = blob + hdr.nsegs;
    const bool mine = threadIdx.x < (T >> kSB);
    const int last = hdr.nsegs - 1;
    for (uint32_t unit = blockIdx.x; unit < hdr.nunits; unit += gridDim.x) {
        const uint32_t set = unit / hdr.per_set, chunk = unit % hdr.per_set;
        for (int i = threadIdx.x; i < 4 * hdr.nruns; i += blockDim.x)
            cf[i] = coef[((size_t)set * hdr.nruns_all + hdr.run[i >> 2]) * 4 + (i & 3)];
        if (BACK)
            for (int i = threadIdx.x; i < hdr.nruns * (int)nw * 8; i += blockDim.x) acc[i] = 0.0;
        __syncthreads();
        for (uint32_t t = chunk; t < hdr.ntiles; t += hdr.per_set) {
            const uint64_t base = ((uint64_t)set << hdr.n) | insert_zeros(t, tb, hdr.tbits);
            for (int si = 0; si <= last; si++) {
                const uint4 sg = blob[si];
                uint32_t lb = threadIdx.x, so[kSB];
                uint64_t go[kSB];
#pragma unroll
                for (int i = 0; i < kSB; i++) {
                    const uint32_t p = (sg.z >> (8 * i)) & 0xffu, q = (sg.w >> (8 * i)) & 0xffu;
                    lb = ((lb >> p) << (p + 1)) | (lb & ((1u << p) - 1));
                    so[i] = tma::swizzle128(16u << q);
                    go[i] = 1ull << tb[q];
                }
                const uint32_t sb = tma::swizzle128(lb * 16u);
                uint64_t gb = base;
                if (si == 0 || si == last)
                    for (int j = 0; j < hdr.tbits; j++) gb |= (uint64_t)((lb >> j) & 1u) << tb[j];
                auto at = [&](int j) {
                    uint32_t o = sb;
#pragma unroll
                    for (int i = 0; i < kSB; i++)
                        if (j & (1 << i)) o ^= so[i];
                    return o;
                };
                auto gat = [&](int j) {
                    uint64_t o = gb;
#pragma unroll
                    for (int i = 0; i < kSB; i++)
                        if (j & (1 << i)) o |= go[i];
                    return o;
                };
                double2 x[NA], l[NA];
                if (si > 0) __syncthreads();
#pragma unroll
                for (int j = 0; j < NA; j++) x[j] = l[j] = make_double2(0.0, 0.0);
                if (mine) {
                    if (si == 0) {
#pragma unroll
                        for (int j = 0; j < NA; j++) {
                            x[j] = psi[gat(j)];
                            if (BACK) l[j] = lam[gat(j)];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < NA; j++) {
                            x[j] = *(const double2*)((const unsigned char*)sp + at(j));
                            if (BACK) l[j] = *(const double2*)((const unsigned char*)sl + at(j));
                        }
                    }
                }
                for (int oi = (int)sg.x; oi < (int)sg.y; oi++) {
                    const uint4 w0 = ops[2 * oi];
                    const uint32_t gval = ops[2 * oi + 1].x;
                    const bool on = (t & w0.w) == gval && (lb & (w0.z & 0xffffu)) == (w0.z >> 16);
                    const uint32_t jm = on ? w0.x >> 16 : 0u;
                    const double2* m = cf + 4 * w0.y;
                    double* a = acc + ((size_t)w0.y * nw + (threadIdx.x >> 5)) * 8;
                    switch (w0.x & 0xffu) {
#define S_RUN(P, RC)                                                            \
    if (w0.x >> 16) {                                                           \
        s_x<P>(x, jm);                                                          \
        if (BACK) s_x<P>(l, jm);                                                \
    }                                                                           \
    if (BACK) s_sums<P>(x, l, mine, a);                                         \
    s_apply<P, RC>(m, x);                                                       \
    if (BACK) s_apply<P, RC>(m, l);                                             \
    break
                    case SC_RUN + 0: S_RUN(0, false);
                    case SC_RUN + 1: S_RUN(1, false);
                    case SC_RUN + 2: S_RUN(2, false);
                    case SC_RUNC + 0: S_RUN(0, true);
                    case SC_RUNC + 1: S_RUN(1, true);
                    case SC_RUNC + 2: S_RUN(2, true);
#undef S_RUN
#define S_X(P)                     \
    s_x<P>(x, jm);                 \
    if (BACK) s_x<P>(l, jm);       \
    break
                    case SC_X + 0: S_X(0);
                    case SC_X + 1: S_X(1);
                    case SC_X + 2: S_X(2);
#undef S_X
                    case SC_SWAP:
#pragma unroll
                        for (int j = 0; j < NA; j += 4)
                            if ((jm >> j) & 1) {
                                double2 w = x[j + 1];
                                x[j + 1] = x[j + 2];
                                x[j + 2] = w;
                                w = l[j + 1];
                                l[j + 1] = l[j + 2];
                                l[j + 2] = w;
                            }
                        break;
                    default:  // SC_NEG
#pragma unroll
                        for (int j = 0; j < NA; j++)
                            if ((jm >> j) & 1) {
                                x[j] = make_double2(-x[j].x, -x[j].y);
                                l[j] = make_double2(-l[j].x, -l[j].y);
                            }
                        break;
                    }
                }
                if (mine) {
                    if (si == last) {
#pragma unroll
                        for (int j = 0; j < NA; j++) {
                            psi[gat(j)] = x[j];
                            if (BACK) lam[gat(j)] = l[j];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < NA; j++) {
                            *(double2*)((unsigned char*)sp + at(j)) = x[j];
                            if (BACK) *(double2*)((unsigned char*)sl + at(j)) = l[j];
                        }
                    }
                }
            }
            if (last > 0) __syncthreads();  // the buffers have been read
        }
        if (BACK) {
            __syncthreads();
            for (int i = threadIdx.x; i < 4 * hdr.nruns; i += blockDim.x) {
                double s = 0.0;
                for (uint32_t w = 0; w < nw; w++) {
                    const double* a = acc + ((size_t)(i >> 2) * nw + w) * 8 + 2 * (i & 3);
                    s += a[0] + a[1];
                }
                partial[((size_t)unit * hdr.nruns) * 4 + i] = s;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------- gate products and gradients

// One gate of a run, first to last: a parametric gate (its parameter) or a
// constant matrix.
struct SFactor {
    int32_t type, slot;  // slot < 0: constant
    double2 m[4];
};
struct SRunDev {
    int32_t begin, end;  // factors
    int32_t real_col;    // the matrix's dagger has a real first column up to a phase
    int32_t pad;
};

struct M2d {
    double2 e[4];
};
__device__ __forceinline__ M2d d_mul(const M2d& a, const M2d& b) {
    M2d r;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) r.e[2 * i + j] = s_mad(s_mul(a.e[2 * i], b.e[j]), a.e[2 * i + 1], b.e[2 + j]);
    return r;
}
__device__ __forceinline__ M2d d_adj(const M2d& a) {
    return M2d{{make_double2(a.e[0].x, -a.e[0].y), make_double2(a.e[2].x, -a.e[2].y), make_double2(a.e[1].x, -a.e[1].y),
                make_double2(a.e[3].x, -a.e[3].y)}};
}
__device__ M2d d_factor(const SFactor& f, const double* p) {
    M2d m;
    if (f.slot < 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) m.e[i] = f.m[i];
        return m;
    }
    double s, c;
    const double2 z = make_double2(0.0, 0.0);
    if (f.type == YAO_GATE_PHASE) {
        sincos(p[f.slot], &s, &c);
        return M2d{{make_double2(1.0, 0.0), z, z, make_double2(c, s)}};
    }
    sincos(0.5 * p[f.slot], &s, &c);
    if (f.type == YAO_GATE_RX)
        return M2d{{make_double2(c, 0.0), make_double2(0.0, -s), make_double2(0.0, -s), make_double2(c, 0.0)}};
    if (f.type == YAO_GATE_RY)
        return M2d{{make_double2(c, 0.0), make_double2(-s, 0.0), make_double2(s, 0.0), make_double2(c, 0.0)}};
    return M2d{{make_double2(c, -s), z, z, make_double2(c, s)}};
}

// fwd / back[set][run]: the run's matrix and its dagger (its first column
// made real by a phase, which psi and lambda share, where real_col says so)
__global__ void k_sweep_coefs(const SFactor* __restrict__ fac, const SRunDev* __restrict__ runs, int nruns, int np,
                              const double* __restrict__ params, uint32_t nsets, double2* __restrict__ fwd,
                              double2* __restrict__ back) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nsets * (uint32_t)nruns; i += gridDim.x * blockDim.x) {
        const uint32_t set = i / nruns;
        const SRunDev r = runs[i % nruns];
        M2d m = d_factor(fac[r.begin], params + (size_t)set * np);
        for (int f = r.begin + 1; f < r.end; f++) m = d_mul(d_factor(fac[f], params + (size_t)set * np), m);
        M2d b = d_adj(m);
        if (r.real_col) {
            const double2 big = fabs(b.e[0].x) + fabs(b.e[0].y) >= fabs(b.e[2].x) + fabs(b.e[2].y) ? b.e[0] : b.e[2];
            const double h = 1.0 / hypot(big.x, big.y);
            const double2 ph = make_double2(big.x * h, -big.y * h);
#pragma unroll
            for (int q = 0; q < 4; q++) b.e[q] = s_mul(ph, b.e[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (fwd) fwd[(size_t)i * 4 + q] = m.e[q];
            back[(size_t)i * 4 + q] = b.e[q];
        }
    }
}

struct SPlace {
    uint64_t off;        // the run's pass's partial sums
    int32_t nruns, at;   // runs of that pass, this run's place
};

// grads[set][slot] from the runs' sums
__global__ void k_sweep_grads(const SFactor* __restrict__ fac, const SRunDev* __restrict__ runs,
                              const SPlace* __restrict__ place, int nruns, int np, uint32_t per_set,
                              const double* __restrict__ params, uint32_t nsets, const double* __restrict__ partial,
                              double* __restrict__ grads) {
    // a warp a (set, run): the lanes add up the units' sums
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < nsets * (uint32_t)nruns; i += warps) {
        const uint32_t set = i / nruns;
        const SRunDev r = runs[i % nruns];
        const SPlace pl = place[i % nruns];
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        for (uint32_t u = lane; u < per_set; u += 32) {
            const double* q = partial + pl.off + (((size_t)set * per_set + u) * pl.nruns + pl.at) * 4;
#pragma unroll
            for (int v = 0; v < 4; v++) s[v] += q[v];
        }
#pragma unroll
        for (int v = 0; v < 4; v++) s[v] = warp_sum(s[v]);
        if (lane) continue;
        const double* p = params + (size_t)set * np;
        const double2 z = make_double2(0.0, 0.0);
        M2d w{{make_double2(1.0, 0.0), z, z, make_double2(1.0, 0.0)}};
        for (int f = r.end - 1; f >= r.begin; f--) {
            if (fac[f].slot >= 0) {
                M2d g{{z, z, z, z}};
                switch (fac[f].type) {
                case YAO_GATE_RX: g.e[1] = g.e[2] = make_double2(0.0, -0.5); break;
                case YAO_GATE_RY: g.e[1] = make_double2(-0.5, 0.0); g.e[2] = make_double2(0.5, 0.0); break;
                case YAO_GATE_RZ: g.e[0] = make_double2(0.0, -0.5); g.e[3] = make_double2(0.0, 0.5); break;
                default: g.e[3] = make_double2(0.0, 1.0); break;
                }
                g = d_mul(w, d_mul(g, d_adj(w)));
                const double dot = fma(-g.e[0].y, s[0], fma(-g.e[3].y, s[1], fma(g.e[1].x, s[2], -g.e[1].y * s[3])));
                grads[(size_t)set * np + fac[f].slot] = 2.0 * dot;
            }
            w = d_mul(w, d_factor(fac[f], p));
        }
    }
}

// Re <psi_s|lambda_s>, `per` blocks a set: the sum of block b is set b / per's
__global__ void __launch_bounds__(256) k_sweep_energy(const double2* __restrict__ psi, const double2* __restrict__ lam,
                                                      uint64_t n, uint32_t per, double* __restrict__ sums) {
    __shared__ double sm[8];
    const uint64_t set = blockIdx.x / per, part = blockIdx.x % per;
    const double2 *p = psi + set * n, *l = lam + set * n;
    double e = 0.0;
    for (uint64_t i = part * blockDim.x + threadIdx.x; i < n; i += (uint64_t)per * blockDim.x)
        e = fma(p[i].x, l[i].x, fma(p[i].y, l[i].y, e));
    block_sum_write(&e, 1, sm, sums + blockIdx.x);
}
// values[set] from its blocks' sums, a warp a set
__global__ void __launch_bounds__(128) k_sweep_energy_final(const double* __restrict__ sums, uint32_t per, uint32_t nsets,
                                                            double* __restrict__ values) {
    const uint32_t set = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (set >= nsets) return;
    double e = 0.0;
    for (uint32_t i = threadIdx.x & 31; i < per; i += 32) e += sums[(size_t)set * per + i];
    e = warp_sum(e);
    if ((threadIdx.x & 31) == 0) values[set] = e;
}

__global__ void k_sweep_broadcast(const double2* __restrict__ src, double2* __restrict__ dst, uint64_t mask, uint64_t total) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = src[i & mask];
}

// ================================================================== planner

namespace {

enum ItemKind { IT_RUN, IT_X, IT_SWAP, IT_NEG };

// One step of the circuit: a run, or a gate of its own.
struct Item {
    ItemKind kind = IT_RUN;
    int run = -1;
    int tb[2] = {-1, -1};
    int k = 1;
    std::vector<std::pair<int, int>> ctl;  // (bit, value); IT_NEG: all its bits
    uint64_t need = 0, qubits = 0;
};

struct SPass {
    SHdr hdr;
    std::vector<SSeg> segs;
    std::vector<SOp> ops;
    std::vector<int> runs;
};

}  // namespace

struct SweepPlan {
    uint32_t n = 0;
    int np = 0;
    std::vector<SFactor> factors;
    std::vector<SRunDev> runs;
    std::vector<Item> items;  // in circuit order
    std::vector<SPass> fwd, back;
};

static bool unit_diag(const SFactor& f) {
    if (f.slot >= 0) return f.type == YAO_GATE_RZ || f.type == YAO_GATE_PHASE;
    auto one = [](double2 z) { return std::fabs(z.x * z.x + z.y * z.y - 1.0) < 1e-13; };
    return f.m[1].x == 0 && f.m[1].y == 0 && f.m[2].x == 0 && f.m[2].y == 0 && one(f.m[0]) && one(f.m[3]);
}
static bool real_matrix(const SFactor& f) {
    if (f.slot >= 0) return f.type == YAO_GATE_RY;
    return f.m[0].y == 0 && f.m[1].y == 0 && f.m[2].y == 0 && f.m[3].y == 0;
}

static uint64_t target_bits(const LGate& l) {
    uint64_t m = 0;
    for (int q = 0; q < l.k; q++) m |= 1ull << l.tb[q];
    return m;
}

// U^dagger U = 1 to the rounding of the entries.  The steps of a sweep change
// places on disjoint qubits: a dot of lambda and psi stays the same under a
// matrix on another qubit when that matrix is unitary, else it does not.
static bool unitary(const SFactor& f) {
    const double2 *m = f.m;
    auto sq = [](double2 z) { return z.x * z.x + z.y * z.y; };
    const double re = m[0].x * m[1].x + m[0].y * m[1].y + m[2].x * m[3].x + m[2].y * m[3].y,
                 im = m[0].x * m[1].y - m[0].y * m[1].x + m[2].x * m[3].y - m[2].y * m[3].x;
    const double eps = 1e-14;
    return std::fabs(sq(m[0]) + sq(m[2]) - 1.0) < eps && std::fabs(sq(m[1]) + sq(m[3]) - 1.0) < eps &&
           std::fabs(re) < eps && std::fabs(im) < eps;
}

// The passes of `items` in the given order.  A step is taken past skipped
// ones that share no qubit with it: the sums and states change by rounding
// only.  back: an X joins the run on its target that follows it.
static void plan_items(const std::vector<const Item*>& items, uint32_t n, bool back, std::vector<SPass>& out) {
    const int tbits = std::min<int>((int)n, kSTile);
    const bool whole = (int)n <= tbits;
    const uint64_t lowmask = whole ? 0 : (1ull << kSLow) - 1;
    uint64_t all = 0;  // the bits that steps touch
    for (const Item* it : items) all |= it->qubits;
    const int cap = whole ? (int)n : tbits - kSLow;
    std::vector<char> used(items.size(), 0);
    size_t first = 0, left = items.size();
    while (left) {
        uint64_t hi = 0, blocked = 0;
        std::vector<size_t> take;
        int nruns = 0, skipped = 0;
        for (size_t j = first; j < items.size() && (blocked & all) != all && (int)take.size() < kSMaxOps && skipped < kSMaxSkipped;
             j++) {
            if (used[j]) continue;
            const Item& it = *items[j];
            const uint64_t nh = hi | (it.need & ~lowmask);
            if ((it.qubits & blocked) || __builtin_popcountll(nh) > cap || (it.kind == IT_RUN && nruns >= kSMaxRuns)) {
                blocked |= it.qubits;
                skipped++;
                continue;
            }
            hi = nh;
            nruns += it.kind == IT_RUN;
            take.push_back(j);
            used[j] = 1;
            left--;
        }
        while (first < items.size() && used[first]) first++;
        uint64_t tile = hi | lowmask;
        for (uint32_t b = 0; __builtin_popcountll(tile) < tbits; b++) tile |= 1ull << b;
        SPass p;
        memset(&p.hdr, 0, sizeof(p.hdr));
        p.hdr.n = (int32_t)n;
        p.hdr.tbits = tbits;
        p.hdr.ntiles = 1u << (n - tbits);
        int local[64], outside[64], nt = 0, no = 0;
        for (uint32_t b = 0; b < n; b++) {
            local[b] = outside[b] = -1;
            if ((tile >> b) & 1) {
                p.hdr.tb[nt] = (int8_t)b;
                local[b] = nt++;
            } else {
                outside[b] = no++;
            }
        }
        std::vector<char> done(take.size(), 0);
        size_t ndone = 0;
        while (ndone < take.size()) {
            // the steps of a segment: at most three positions move
            std::vector<int> bits;
            int pair[2] = {-1, -1};
            std::vector<const Item*> seq;
            uint64_t blk = 0;
            for (size_t q = 0; q < take.size() && (blk & all) != all; q++) {
                if (done[q]) continue;
                const Item& it = *items[take[q]];
                int fresh = 0;
                if (it.need)
                    for (int i = 0; i < it.k; i++)
                        fresh += std::find(bits.begin(), bits.end(), local[it.tb[i]]) == bits.end();
                bool ok = !(it.qubits & blk) && (int)bits.size() + fresh <= kSB;
                if (ok && it.kind == IT_SWAP) {
                    const int a = local[it.tb[0]], b = local[it.tb[1]];
                    ok = pair[0] < 0 || (pair[0] == std::min(a, b) && pair[1] == std::max(a, b));
                    if (ok) {
                        pair[0] = std::min(a, b);
                        pair[1] = std::max(a, b);
                    }
                }
                if (!ok) {
                    blk |= it.qubits;
                    continue;
                }
                if (it.need)
                    for (int i = 0; i < it.k; i++)
                        if (std::find(bits.begin(), bits.end(), local[it.tb[i]]) == bits.end())
                            bits.push_back(local[it.tb[i]]);
                seq.push_back(&it);
                done[q] = 1;
                ndone++;
            }
            std::vector<int> order;
            if (pair[0] >= 0) order = {pair[0], pair[1]};
            for (int b : bits)
                if (std::find(order.begin(), order.end(), b) == order.end()) order.push_back(b);
            for (int b = tbits - 1; (int)order.size() < kSB && b >= 0; b--)
                if (std::find(order.begin(), order.end(), b) == order.end()) order.push_back(b);
            std::vector<int> sorted(order);
            std::sort(sorted.begin(), sorted.end());
            SSeg sg;
            memset(&sg, 0, sizeof(sg));
            for (int i = 0; i < kSB; i++) {
                sg.sorted[i] = (int8_t)sorted[i];
                sg.order[i] = (int8_t)order[i];
            }
            sg.op_begin = (int32_t)p.ops.size();
            auto pos = [&](int b) -> int {  // register position of a global bit, -1
                if (local[b] < 0) return -1;
                const auto f = std::find(order.begin(), order.end(), local[b]);
                return f == order.end() ? -1 : (int)(f - order.begin());
            };
            // controls of `it` on op, and the mask of register indices they allow
            auto controls = [&](const Item& it, SOp& op) {
                uint32_t jm = 0xffu;
                for (const auto& c : it.ctl) {
                    const int r = pos(c.first);
                    if (r >= 0) {
                        for (uint32_t j = 0; j < (1u << kSB); j++)
                            if (((j >> r) & 1u) != (uint32_t)c.second) jm &= ~(1u << j);
                    } else if (local[c.first] >= 0) {
                        op.ctl |= (1u << local[c.first]) | ((uint32_t)c.second << (16 + local[c.first]));
                    } else {
                        op.gmask |= 1u << outside[c.first];
                        op.gval |= (uint32_t)c.second << outside[c.first];
                    }
                }
                return jm;
            };
            auto first_of = [](uint32_t jm, int r) {  // the masked pairs' first members
                for (uint32_t j = 0; j < (1u << kSB); j++)
                    if ((j >> r) & 1u) jm &= ~(1u << j);
                return jm;
            };
            std::vector<char> gone(seq.size(), 0);
            for (size_t q = 0; q < seq.size(); q++) {
                if (gone[q]) continue;
                const Item* it = seq[q];
                SOp op;
                memset(&op, 0, sizeof(op));
                if (it->kind == IT_X) {
                    const int r = pos(it->tb[0]);
                    const uint32_t jm = first_of(controls(*it, op), r);
                    // the next step on the target, when it is a run and
                    // nothing before it touches the target: it moves up here
                    size_t f = q + 1;
                    while (back && f < seq.size() && (gone[f] || !(seq[f]->qubits & (1ull << it->tb[0])))) f++;
                    if (back && f < seq.size() && seq[f]->kind == IT_RUN) {
                        gone[f] = 1;
                        it = seq[f];
                        op.run = (uint32_t)p.runs.size();
                        p.runs.push_back(it->run);
                        op.head = SC_RUN + (uint32_t)r + (jm << 16);
                        p.ops.push_back(op);
                        continue;
                    }
                    op.head = SC_X + (uint32_t)r + (jm << 16);
                } else if (it->kind == IT_RUN) {
                    op.run = (uint32_t)p.runs.size();
                    p.runs.push_back(it->run);
                    op.head = SC_RUN + (uint32_t)pos(it->tb[0]);
                } else if (it->kind == IT_SWAP) {
                    uint32_t jm = controls(*it, op);
                    for (uint32_t j = 0; j < (1u << kSB); j++)
                        if (j & 3u) jm &= ~(1u << j);
                    op.head = SC_SWAP + (jm << 16);
                } else {
                    op.head = SC_NEG + (controls(*it, op) << 16);
                }
                p.ops.push_back(op);
            }
            sg.op_end = (int32_t)p.ops.size();
            p.segs.push_back(sg);
        }
        // tiles enter and leave through registers: the low positions on the
        // lanes make whole 128-byte runs
        auto plain = [&](int at) {
            SSeg sg;
            memset(&sg, 0, sizeof(sg));
            sg.op_begin = sg.op_end = at;
            for (int i = 0; i < kSB; i++) sg.sorted[i] = sg.order[i] = (int8_t)(tbits - kSB + i);
            return sg;
        };
        if (tbits >= kSLow + kSB) {
            if (p.segs.front().sorted[0] < kSLow) p.segs.insert(p.segs.begin(), plain(0));
            if (p.segs.back().sorted[0] < kSLow) p.segs.push_back(plain((int)p.ops.size()));
        }
        out.push_back(std::move(p));
    }
}

SweepPlan* sweep_plan_new(const Circuit* c, uint32_t n) {
    if (n < 3 || n > 30) return nullptr;
    std::unique_ptr<SweepPlan> pl(new SweepPlan());
    pl->n = n;
    std::vector<std::vector<SFactor>> pend(n);
    auto flush = [&](int b) {
        if (pend[b].empty()) return;
        SRunDev r;
        memset(&r, 0, sizeof(r));
        r.begin = (int32_t)pl->factors.size();
        // matrix = diagonals after real gates: its dagger is real . diagonal
        size_t q = 0;
        while (q < pend[b].size() && real_matrix(pend[b][q])) q++;
        bool rc = true;
        for (; q < pend[b].size(); q++) rc &= unit_diag(pend[b][q]);
        r.real_col = rc;
        pl->factors.insert(pl->factors.end(), pend[b].begin(), pend[b].end());
        r.end = (int32_t)pl->factors.size();
        pend[b].clear();
        Item it;
        it.kind = IT_RUN;
        it.run = (int)pl->runs.size();
        it.tb[0] = b;
        it.need = it.qubits = 1ull << b;
        pl->runs.push_back(r);
        pl->items.push_back(it);
    };
    for (const Element& el : c->elems) {
        if (el.kind == YAO_ELEM_CHANNEL) return nullptr;
        if (el.kind != YAO_ELEM_GATE) continue;
        const GateElem& g = el.g;
        std::vector<LGate> lg;
        lower_gate(g, n, 0, false, lg);
        const int np = gate_num_params(g.type);
        if (np) {
            if (np != 1 || !g.ctrls.empty() || lg.size() != 1 || lg[0].k != 1) return nullptr;
            SFactor f;
            memset(&f, 0, sizeof(f));
            f.type = g.type;
            f.slot = pl->np++;
            pend[lg[0].tb[0]].push_back(f);
            continue;
        }
        for (const LGate& l : lg) {
            if (l.k == 1 && l.nc == 0) {
                SFactor f;
                memset(&f, 0, sizeof(f));
                f.type = g.type;
                f.slot = -1;
                if (l.cls == GC_X) {
                    f.m[1] = f.m[2] = make_double2(1.0, 0.0);
                } else if (l.cls == GC_DIAG) {
                    f.m[0] = make_double2(l.m[0].re, l.m[0].im);
                    f.m[3] = make_double2(l.m[1].re, l.m[1].im);
                } else {
                    for (int q = 0; q < 4; q++) f.m[q] = make_double2(l.m[q].re, l.m[q].im);
                }
                if (!unitary(f)) return nullptr;
                pend[l.tb[0]].push_back(f);
                continue;
            }
            if (__builtin_popcountll(l.cmask() | target_bits(l)) != l.k + l.nc) return nullptr;  // a qubit twice
            Item it;
            it.k = l.k;
            for (int q = 0; q < l.k && q < 2; q++) it.tb[q] = l.tb[q];
            for (int q = 0; q < l.nc; q++) it.ctl.push_back({l.cb[q], l.cv[q] ? 1 : 0});
            if (l.cls == GC_X && l.k == 1) {
                it.kind = IT_X;
                it.need = 1ull << l.tb[0];
            } else if (l.cls == GC_SWAP) {
                it.kind = IT_SWAP;
                it.need = (1ull << l.tb[0]) | (1ull << l.tb[1]);
            } else if (l.cls == GC_DIAG) {
                // one entry -1, the others 1
                int minus = -1;
                for (size_t q = 0; q < l.m.size(); q++) {
                    if (l.m[q].im != 0.0 || std::fabs(l.m[q].re) != 1.0) return nullptr;
                    if (l.m[q].re == 1.0) continue;
                    if (minus >= 0) return nullptr;
                    minus = (int)q;
                }
                if (minus < 0) continue;
                it.kind = IT_NEG;
                for (int q = 0; q < l.k; q++) it.ctl.push_back({l.tb[q], (minus >> q) & 1});
            } else {
                return nullptr;
            }
            it.qubits = it.need;
            for (const auto& q : it.ctl) it.qubits |= 1ull << q.first;
            for (uint32_t b = 0; b < n; b++)
                if ((it.qubits >> b) & 1) flush((int)b);
            pl->items.push_back(it);
        }
    }
    for (uint32_t b = 0; b < n; b++) flush((int)b);
    if (pl->np == 0) return nullptr;
    std::vector<const Item*> seq;
    for (const Item& it : pl->items) seq.push_back(&it);
    plan_items(seq, n, false, pl->fwd);
    std::reverse(seq.begin(), seq.end());
    plan_items(seq, n, true, pl->back);
    // runs whose dagger has a real first column: the cheaper product
    for (SPass& p : pl->back)
        for (SOp& op : p.ops)
            if ((op.head & 0xffu) < SC_RUNC && pl->runs[p.runs[op.run]].real_col) op.head += SC_RUNC;
    for (auto* ps : {&pl->fwd, &pl->back})
        for (SPass& p : *ps) {
            p.hdr.nsegs = (int32_t)p.segs.size();
            p.hdr.nops = (int32_t)p.ops.size();
            p.hdr.nruns = (int32_t)p.runs.size();
            p.hdr.nruns_all = (int32_t)pl->runs.size();
            for (size_t i = 0; i < p.runs.size(); i++) p.hdr.run[i] = p.runs[i];
        }
    return pl.release();
}

void sweep_plan_free(SweepPlan* p) { delete p; }

// ================================================================ execution

namespace {

// Device copies of a plan and the buffers of a sweep over `group` sets, in one
// stream-ordered allocation.
struct SweepRun {
    Ctx* ctx;
    const SweepPlan* p;
    uint32_t group;
    uint32_t per_set = 1;
    char* buf = nullptr;
    uint4* blob = nullptr;
    SFactor* fac = nullptr;
    SRunDev* runs = nullptr;
    SPlace* place = nullptr;
    double* params = nullptr;
    double2 *cf = nullptr, *cb = nullptr;
    double *partial = nullptr, *grads = nullptr;
    std::vector<size_t> off_f, off_b;   // passes' descriptions
    std::vector<uint64_t> part;         // passes' partial sums

    ~SweepRun() {
        if (buf) cudaFreeAsync(buf, ctx->stream);
    }

    static size_t smem_bytes(const SPass& s, bool back) {
        const size_t T = (size_t)1 << s.hdr.tbits;
        const size_t warps = std::max<size_t>(32, T >> kSB) / 32;
        return (back ? 2 : 1) * T * 16 + s.hdr.nruns * 64 + s.segs.size() * sizeof(SSeg) + s.ops.size() * sizeof(SOp) +
               (back ? s.hdr.nruns * warps * 64 : 0);
    }

    int init(const double* host_params, size_t nsets) {
        // per_set units share a set's tiles: about three units for every CTA
        // the GPU holds, so that the last round is a small part
        const uint32_t ntiles = p->back.empty() ? 1 : p->back[0].hdr.ntiles, units = 6u * (uint32_t)ctx->num_sms;
        per_set = std::max(1u, std::min(ntiles, (units + group - 1) / group));
        std::vector<uint4> h;
        auto add = [&](const std::vector<SPass>& ps, std::vector<size_t>& off) {
            for (const SPass& s : ps) {
                off.push_back(h.size());
                h.resize(h.size() + s.segs.size() + 2 * s.ops.size());
                memcpy(&h[off.back()], s.segs.data(), s.segs.size() * sizeof(SSeg));
                memcpy(&h[off.back() + s.segs.size()], s.ops.data(), s.ops.size() * sizeof(SOp));
            }
        };
        add(p->fwd, off_f);
        add(p->back, off_b);
        std::vector<SPlace> pl(p->runs.size());
        uint64_t np = 0;
        for (const SPass& s : p->back) {
            part.push_back(np);
            for (size_t i = 0; i < s.runs.size(); i++) pl[s.runs[i]] = SPlace{np, s.hdr.nruns, (int32_t)i};
            np += (uint64_t)group * per_set * s.runs.size() * 4;
        }
        auto al = [](size_t x) { return (x + 255) / 256 * 256; };
        const size_t b_blob = al(h.size() * 16), b_fac = al(p->factors.size() * sizeof(SFactor)),
                     b_runs = al(p->runs.size() * sizeof(SRunDev)), b_place = al(pl.size() * sizeof(SPlace)),
                     b_par = al(nsets * p->np * 8), b_cf = al((size_t)group * p->runs.size() * 64),
                     b_part = al(np * 8), b_grad = al(nsets * p->np * 8);
        if (alloc_async(ctx, (void**)&buf, b_blob + b_fac + b_runs + b_place + b_par + 2 * b_cf + b_part + b_grad) !=
            cudaSuccess) {
            cudaGetLastError();
            buf = nullptr;
            return fail(YAO_ERR_OUT_OF_MEMORY, "cannot allocate the gradient's buffers");
        }
        char* q = buf;
        auto take = [&](size_t b) {
            char* r = q;
            q += b;
            return r;
        };
        blob = (uint4*)take(b_blob);
        fac = (SFactor*)take(b_fac);
        runs = (SRunDev*)take(b_runs);
        place = (SPlace*)take(b_place);
        params = (double*)take(b_par);
        cf = (double2*)take(b_cf);
        cb = (double2*)take(b_cf);
        partial = (double*)take(b_part);
        grads = (double*)take(b_grad);
        cudaStream_t s = ctx->stream;
        YAO_CUDA(cudaMemcpyAsync(blob, h.data(), h.size() * 16, cudaMemcpyHostToDevice, s));
        YAO_CUDA(cudaMemcpyAsync(fac, p->factors.data(), p->factors.size() * sizeof(SFactor), cudaMemcpyHostToDevice, s));
        YAO_CUDA(cudaMemcpyAsync(runs, p->runs.data(), p->runs.size() * sizeof(SRunDev), cudaMemcpyHostToDevice, s));
        YAO_CUDA(cudaMemcpyAsync(place, pl.data(), pl.size() * sizeof(SPlace), cudaMemcpyHostToDevice, s));
        YAO_CUDA(cudaMemcpyAsync(params, host_params, nsets * p->np * 8, cudaMemcpyHostToDevice, s));
        KernelFit fit;
        int sf = kernel_fit(ctx, (const void*)k_sweep<true>, &fit);
        if (!sf) sf = kernel_fit(ctx, (const void*)k_sweep<false>, &fit);
        if (sf) return sf;
        return YAO_OK;
    }

    int coefs(size_t first_set, uint32_t nsets, bool forward) {
        const uint32_t total = nsets * (uint32_t)p->runs.size();
        k_sweep_coefs<<<grid_for(total, 128, ctx->num_sms), 128, 0, ctx->stream>>>(
            fac, runs, (int)p->runs.size(), p->np, params + first_set * p->np, nsets, forward ? cf : nullptr, cb);
        ctx->launches++;
        YAO_CUDA(cudaGetLastError());
        return YAO_OK;
    }

    int passes(bool back, double2* psi, double2* lam, uint32_t nsets) {
        const std::vector<SPass>& ps = back ? p->back : p->fwd;
        for (size_t i = 0; i < ps.size(); i++) {
            SHdr h = ps[i].hdr;
            h.per_set = per_set;
            h.nunits = nsets * per_set;
            const unsigned threads = std::max(32u, (1u << h.tbits) >> kSB);
            const size_t smem = smem_bytes(ps[i], back);
            int per_sm = 0;
            YAO_CUDA(back ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep<true>, (int)threads, smem)
                          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep<false>, (int)threads, smem));
            const unsigned grid = (unsigned)std::min<uint64_t>(h.nunits, (uint64_t)std::max(1, per_sm) * ctx->num_sms);
            ProfScope prof(ctx, back ? "sweep_reverse" : "sweep_forward",
                           (double)nsets * (double)(1ull << h.n) * (back ? 64.0 : 32.0));
            if (back)
                k_sweep<true><<<grid, threads, smem, ctx->stream>>>(psi, lam, h, blob + off_b[i], cb, partial + part[i]);
            else
                k_sweep<false><<<grid, threads, smem, ctx->stream>>>(psi, nullptr, h, blob + off_f[i], cf, nullptr);
            ctx->launches++;
            YAO_CUDA(cudaGetLastError());
        }
        return YAO_OK;
    }

    int gradients(size_t first_set, uint32_t nsets) {
        const uint32_t total = nsets * (uint32_t)p->runs.size();
        k_sweep_grads<<<grid_for(total, 4, ctx->num_sms, 16), 128, 0, ctx->stream>>>(
            fac, runs, place, (int)p->runs.size(), p->np, per_set, params + first_set * p->np, nsets, partial,
            grads + first_set * p->np);
        ctx->launches++;
        YAO_CUDA(cudaGetLastError());
        return YAO_OK;
    }
};

}  // namespace

int sweep_reverse(Ctx* ctx, const SweepPlan* p, void* psi, void* lam, const double* params, double* grad) {
    SweepRun r{ctx, p, 1};
    int s = r.init(params, 1);
    if (!s) s = r.coefs(0, 1, false);
    if (!s) s = r.passes(true, (double2*)psi, (double2*)lam, 1);
    if (!s) s = r.gradients(0, 1);
    if (s) return s;
    YAO_CUDA(cudaMemcpyAsync(grad, r.grads, (size_t)p->np * 8, cudaMemcpyDeviceToHost, ctx->stream));
    return read_device_err(ctx, "expect_grad");
}

int sweep_batch(Ctx* ctx, const SweepPlan* p, const std::vector<MonoTerm>& terms, const double* params, size_t nsets,
                const Reg* psi0, double* values, double* grads) {
    const uint64_t N = 1ull << p->n;
    // sets at a time, at least one: psi and lambda within 64 MB, so that a pass
    // finds in the L2 cache what the last one left there; matrices (two a run)
    // and sums, each read once, within 256 MB (the smaller groups of 64 MB in
    // all: 44.6 against 40.9 ms on 6 qubits, 720 parameters, 16384 sets)
    const size_t states = ((size_t)64 << 20) / (N * 32), runs = ((size_t)256 << 20) / (p->runs.size() * (2 * 64 + 32));
    const size_t group = std::max<size_t>(1, std::min({nsets, states, runs}));
    SweepRun r{ctx, p, (uint32_t)group};
    int s = r.init(params, nsets);
    if (s) return s;
    char* st = nullptr;
    // few sets of large states: several blocks for the energy of one, 16
    // amplitudes a thread at least (one block read both states of a set by
    // itself: at 22 qubits 7.8 ms a set, now 0.03)
    const uint32_t per = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>(N / 4096, (4ull * (uint64_t)ctx->num_sms + group - 1) / group));
    const size_t b_state = group * N * 16, b_val = (nsets * 8 + 255) / 256 * 256, b_sum = group * per * 8;
    if (alloc_async(ctx, (void**)&st, 2 * b_state + b_val + b_sum) != cudaSuccess) {
        cudaGetLastError();
        return fail(YAO_ERR_OUT_OF_MEMORY, "cannot allocate the batched gradient buffers");
    }
    double2 *psi = (double2*)st, *lam = (double2*)(st + b_state);
    double *vals = (double*)(st + 2 * b_state), *sums = (double*)(st + 2 * b_state + b_val);
    for (size_t f = 0; f < nsets && !s; f += group) {
        const uint32_t m = (uint32_t)std::min(group, nsets - f);
        k_sweep_broadcast<<<grid_for(m * N, 256, ctx->num_sms), 256, 0, ctx->stream>>>((const double2*)psi0->d, psi, N - 1, m * N);
        ctx->launches++;
        if ((s = r.coefs(f, m, true)) || (s = r.passes(false, psi, nullptr, m)) ||
            (s = build_lambda_sets(ctx, psi, lam, p->n, m, terms)))
            break;
        {
            ProfScope prof(ctx, "sweep_energy", (double)m * (double)N * 32.0);
            k_sweep_energy<<<m * per, 256, 0, ctx->stream>>>(psi, lam, N, per, per > 1 ? sums : vals + f);
        }
        ctx->launches++;
        if (per > 1) {
            k_sweep_energy_final<<<(m + 3) / 4, 128, 0, ctx->stream>>>(sums, per, m, vals + f);
            ctx->launches++;
        }
        if (!(s = r.passes(true, psi, lam, m))) s = r.gradients(f, m);
    }
    cudaError_t ce = cudaGetLastError();
    if (!s && ce == cudaSuccess) ce = cudaMemcpyAsync(values, vals, nsets * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (!s && ce == cudaSuccess) ce = cudaMemcpyAsync(grads, r.grads, nsets * p->np * 8, cudaMemcpyDeviceToHost, ctx->stream);
    cudaFreeAsync(st, ctx->stream);
    const int ws = wait_results(ctx, "expect_grad_batch");
    if (!s && ce != cudaSuccess) return cuda_fail(ce, "expect_grad_batch");
    return s ? s : ws;
}

}  // namespace yao
