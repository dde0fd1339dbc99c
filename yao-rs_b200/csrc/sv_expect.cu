// sv_expect.cu — expectation value of a sum of Pauli strings over tiles of
// the state (src/expect.rs:7-36).
//
// One launch per X mask read the whole state for each mask (27 launches for
// the 48 terms of a 24-qubit transverse-field Ising chain).  Here a pass reads
// it once for every string whose X mask lies in the pass's tile bits (2^11
// complex128 or 2^12 complex64 amplitudes by TMA: three passes for that
// chain), and diagonal strings ride along with the first.  A thread holds 8
// amplitudes that differ in three tile positions; the strings that flip only
// those are pairs in its registers, others read their partners from shared
// memory.  What bounds it: the reads of the state (three of 268 MB: 0.12 ms at
// the copy rate) and about as much FP64 and sign arithmetic.  24 qubits, 48
// terms: 2.17 -> 0.35 ms of kernels.
//
// A Pauli string P with phase i^(base + 2 popc(i & d2)) at index i is
// Hermitian or i times a Hermitian string; for a Hermitian one the index pair
// (i, i ^ x) contributes 2 Re(conj(psi_i) phase(i) psi_{i ^ x}).  All sums are
// FP64, in an order fixed by the launch shape.
#include <algorithm>
#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "tc_sm100.cuh"
#include "tma_sm100.cuh"

namespace yao {

constexpr int kEB = 3;  // register bits: 8 amplitudes a thread

// A string of a segment, 32 bytes.  flags: register flips in bits 0..2, bit 3:
// the imaginary part of the pair product, bits 8..15: sign of register index
// j, bits 16..: the register bits that sign depends on; xt: flips outside the registers (tile positions); dlo, dhi: sign bits on
// the thread's tile position and on the tile's number.
struct ETerm {
    uint32_t flags, xt, dlo, dhi;
    double cre, cim;
};
// diagonal strings [diag, term), sorted by their register bits, others [term, end); the register positions
// ascending
struct ESeg {
    int32_t diag, term, end;
    int8_t pos[4];
};
static_assert(sizeof(ETerm) == 32 && sizeof(ESeg) == 16, "staged as 16-byte words");

struct EHdr {
    int32_t tbits, nsegs, nterms, nbuf;
    int32_t use_tma, pad;
    uint32_t ntiles, pad2;
    int8_t tb[16];
    TmaPlan tma;
};

__device__ __forceinline__ double2 e_load(const double2* p) { return *p; }
__device__ __forceinline__ double2 e_load(const float2* p) {
    const float2 v = *p;
    return make_double2((double)v.x, (double)v.y);
}

__device__ __forceinline__ double flip(double v, uint32_t top) {
    return __hiloint2double(__double2hiint(v) ^ (int)(top & 0x80000000u), __double2loint(v));
}
// Re (or Im) of conj(a) b
__device__ __forceinline__ double e_pair(double2 a, double2 b, bool im) {
    return im ? fma(a.x, b.y, -a.y * b.x) : fma(a.x, b.x, a.y * b.y);
}

template <int XR>
__device__ __forceinline__ double e_flip(const double2 (&v)[1 << kEB], uint32_t jp, bool im) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < (1 << kEB); j++)
        if ((j ^ XR) > j) s += flip(e_pair(v[j], v[j ^ XR], im), jp << (31 - j));
    return s;
}

template <typename V, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 3 : 1)
    k_expect_tiles(const V* __restrict__ st, const EHdr phdr, const uint4* __restrict__ gblob,
                   double* __restrict__ partial, int* __restrict__ err, const __grid_constant__ CUtensorMap tmap) {
    constexpr uint32_t AB = sizeof(V);
    constexpr int NA = 1 << kEB;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ EHdr hdr;
    __shared__ uint64_t full_bar[4];
    __shared__ double red[2 * THREADS / 32];
    if (threadIdx.x == 0) hdr = phdr;
    __syncthreads();
    unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t tile_bytes = AB << hdr.tbits, nbuf = (uint32_t)hdr.nbuf, grid = gridDim.x;
    uint4* blob = (uint4*)(smem + (size_t)nbuf * tile_bytes);
    for (int i = threadIdx.x; i < hdr.nsegs + 2 * hdr.nterms; i += blockDim.x) blob[i] = gblob[i];
    const ESeg* segs = (const ESeg*)blob;
    const uint4* terms = blob + hdr.nsegs;
    const bool use_tma = hdr.use_tma != 0;
    uint32_t t = blockIdx.x, pending = 0;
    auto load = [&](uint32_t tt, uint32_t b) {
        tc::mbar_arrive_expect_tx(&full_bar[b], tile_bytes);
        tma::load_boxes(&tmap, hdr.tma, insert_zeros(tt, hdr.tb, hdr.tbits), tc::smem_u32(smem) + b * tile_bytes,
                        tc::smem_u32(&full_bar[b]));
        pending |= 1u << b;
    };
    if (use_tma && threadIdx.x == 0) {
        tma::prefetch_map(&tmap);
        for (uint32_t q = 0; q < nbuf; q++) tc::mbar_init(&full_bar[q], 1);
        for (uint32_t q = 0; q < nbuf; q++)
            if ((uint64_t)t + (uint64_t)q * grid < hdr.ntiles) load(t + q * grid, q);
    }
    __syncthreads();
    const bool mine = threadIdx.x < ((1u << hdr.tbits) >> kEB);
    bool dead = false;
    uint32_t b = 0, par = 0;
    double acc[2] = {0.0, 0.0};
    for (; t < hdr.ntiles; t += grid) {
        const unsigned char* s = smem + (size_t)b * tile_bytes;
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
            const uint64_t base = insert_zeros(t, hdr.tb, hdr.tbits);
            for (uint32_t l = threadIdx.x; l < (1u << hdr.tbits); l += blockDim.x) {
                uint64_t o = base;
                for (int j = 0; j < hdr.tbits; j++) o |= (uint64_t)((l >> j) & 1u) << hdr.tb[j];
                *(V*)(smem + tma::swizzle128(l * AB)) = st[o];  // the one buffer
            }
            __syncthreads();
        }
        if (mine)
            for (int si = 0; si < hdr.nsegs; si++) {
                const ESeg sg = segs[si];
                uint32_t lb = threadIdx.x, so[kEB];
#pragma unroll
                for (int i = 0; i < kEB; i++) {
                    const uint32_t p = (uint32_t)sg.pos[i];
                    lb = ((lb >> p) << (p + 1)) | (lb & ((1u << p) - 1));
                    so[i] = tma::swizzle128(AB << p);
                }
                const uint32_t sb = tma::swizzle128(lb * AB);
                auto at = [&](int j) {
                    uint32_t o = sb;
#pragma unroll
                    for (int i = 0; i < kEB; i++)
                        if (j & (1 << i)) o ^= so[i];
                    return o;
                };
                double2 v[NA];
#pragma unroll
                for (int j = 0; j < NA; j++) v[j] = e_load((const V*)(s + at(j)));
                if (sg.diag < sg.term) {
                    double p[NA];
#pragma unroll
                    for (int j = 0; j < NA; j++) p[j] = fma(v[j].x, v[j].x, v[j].y * v[j].y);
                    // their signed sums over the register index (Walsh):
                    // p[q] <- sum over j of (-1)^popc(j & q) p[j]
#pragma unroll
                    for (int h = 1; h < NA; h *= 2)
#pragma unroll
                        for (int j = 0; j < NA; j++)
                            if (!(j & h)) {
                                const double x = p[j], y = p[j | h];
                                p[j] = x + y;
                                p[j | h] = x - y;
                            }
                    int ti = sg.diag;
#pragma unroll
                    for (int q = 0; q < NA; q++)  // the strings are sorted by q
                        for (; ti < sg.term; ti++) {
                            const uint4 w = terms[2 * ti];
                            if ((w.x >> 16) != (uint32_t)q) break;
                            const double2 c = *(const double2*)&terms[2 * ti + 1];
                            const double x = flip(p[q], (uint32_t)(__popc(lb & w.z) + __popc(t & w.w)) << 31);
                            acc[0] = fma(c.x, x, acc[0]);
                            acc[1] = fma(c.y, x, acc[1]);
                        }
                }
                for (int ti = sg.term; ti < sg.end; ti++) {
                    const uint4 w = terms[2 * ti];
                    const double2 c = *(const double2*)&terms[2 * ti + 1];
                    const uint32_t jp = (w.x >> 8) & 0xffu;
                    const bool im = (w.x & 8u) != 0;
                    double x = 0.0;
                    if (w.y == 0) {
                        switch (w.x & 7u) {
                        case 1: x = e_flip<1>(v, jp, im); break;
                        case 2: x = e_flip<2>(v, jp, im); break;
                        case 3: x = e_flip<3>(v, jp, im); break;
                        case 4: x = e_flip<4>(v, jp, im); break;
                        case 5: x = e_flip<5>(v, jp, im); break;
                        case 6: x = e_flip<6>(v, jp, im); break;
                        default: x = e_flip<7>(v, jp, im); break;
                        }
                    } else {
                        // partners elsewhere in the tile: every index of the
                        // pair adds its half
                        uint32_t o = tma::swizzle128(w.y * AB);
#pragma unroll
                        for (int i = 0; i < kEB; i++)
                            if ((w.x >> i) & 1u) o ^= so[i];
#pragma unroll
                        for (int j = 0; j < NA; j++)
                            x += flip(e_pair(v[j], e_load((const V*)(s + (at(j) ^ o))), im), jp << (31 - j));
                    }
                    x = flip(x, (uint32_t)(__popc(lb & w.z) + __popc(t & w.w)) << 31);
                    acc[0] = fma(c.x, x, acc[0]);
                    acc[1] = fma(c.y, x, acc[1]);
                }
            }
        __syncthreads();  // the tile has been read
        if (use_tma && threadIdx.x == 0 && (uint64_t)t + (uint64_t)nbuf * grid < hdr.ntiles) load(t + nbuf * grid, b);
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
    block_sum_write(acc, 2, red, partial + 2 * (size_t)blockIdx.x);
}

// ------------------------------------------------------------------ host

namespace {

struct EPass {
    uint64_t tile = 0;  // tile bits
    std::vector<const MonoTerm*> diag, flips;
};

}  // namespace

template <typename V, int TBITS>
static int expect_tiles(Ctx* ctx, const Reg* r, const std::vector<EPass>& passes, Cx* out) {
    constexpr int THREADS = (1 << TBITS) >> kEB;
    auto kern = k_expect_tiles<V, THREADS>;
    const uint32_t n = r->nbits;
    const int tbits = std::min<int>((int)n, TBITS);
    const uint32_t ntiles = 1u << (n - tbits);
    // descriptions of all passes, one upload
    std::vector<uint4> blob;
    struct Launch {
        EHdr hdr;
        size_t off;
    };
    std::vector<Launch> ls;
    size_t most = 0;
    for (const EPass& p : passes) {
        Launch l;
        memset(&l.hdr, 0, sizeof(l.hdr));
        l.hdr.tbits = tbits;
        l.hdr.ntiles = ntiles;
        int local[64], outside[64], nt = 0, no = 0;
        for (uint32_t b = 0; b < n; b++) {
            local[b] = outside[b] = -1;
            if ((p.tile >> b) & 1) {
                l.hdr.tb[nt] = (int8_t)b;
                local[b] = nt++;
            } else {
                outside[b] = no++;
            }
        }
        auto positions = [&](uint64_t m) {
            std::vector<int> v;
            for (uint32_t b = 0; b < n; b++)
                if ((m >> b) & 1) v.push_back(local[b]);
            return v;
        };
        // segments: strings that flip the same three positions share one
        struct S {
            std::vector<int> bits;
            std::vector<const MonoTerm*> terms;
        };
        std::vector<S> segs;
        for (const MonoTerm* m : p.flips) {
            const std::vector<int> x = positions(m->xmask);
            S* to = nullptr;
            for (S& s : segs) {
                std::vector<int> u(s.bits);
                for (int b : x)
                    if (std::find(u.begin(), u.end(), b) == u.end()) u.push_back(b);
                if (u.size() <= (size_t)kEB) {
                    s.bits = u;
                    to = &s;
                    break;
                }
            }
            if (!to) {
                segs.push_back(S{std::vector<int>(x.end() - std::min<size_t>(x.size(), kEB), x.end()), {}});
                to = &segs.back();
            }
            to->terms.push_back(m);
        }
        if (segs.empty()) segs.push_back(S{});
        std::vector<ESeg> es;
        std::vector<ETerm> et;
        for (size_t q = 0; q < segs.size(); q++) {
            S& s = segs[q];
            for (int b = tbits - 1; (int)s.bits.size() < kEB && b >= 0; b--)
                if (std::find(s.bits.begin(), s.bits.end(), b) == s.bits.end()) s.bits.push_back(b);
            std::sort(s.bits.begin(), s.bits.end());
            ESeg e;
            memset(&e, 0, sizeof(e));
            for (int i = 0; i < kEB; i++) e.pos[i] = (int8_t)s.bits[i];
            auto add = [&](const MonoTerm* m) {
                ETerm w;
                memset(&w, 0, sizeof(w));
                // i^base: the anti-Hermitian strings are i times a Hermitian one
                int base = m->base & 3;
                double cre = m->coeff.re, cim = m->coeff.im;
                const bool odd = __builtin_popcountll(m->xmask & m->d2mask) & 1;
                if (((base & 1) != 0) != odd) {
                    base = (base + 3) & 3;
                    const double x = cre;
                    cre = -cim;
                    cim = x;
                }
                if (base & 1) w.flags |= 8u;
                double f = base == 1 || base == 2 ? -1.0 : 1.0;  // Re(i z) = -Im z
                uint32_t reg = 0;
                for (uint32_t b = 0; b < n; b++) {
                    const int at = local[b] < 0 ? -1 : (int)(std::find(s.bits.begin(), s.bits.end(), local[b]) - s.bits.begin());
                    const bool in_reg = at >= 0 && at < kEB;
                    if ((m->xmask >> b) & 1) {
                        if (in_reg)
                            w.flags |= 1u << at;
                        else
                            w.xt |= 1u << local[b];
                    }
                    if ((m->d2mask >> b) & 1) {
                        if (in_reg)
                            reg |= 1u << at;
                        else if (local[b] >= 0)
                            w.dlo |= 1u << local[b];
                        else
                            w.dhi |= 1u << outside[b];
                    }
                }
                for (uint32_t j = 0; j < (1u << kEB); j++)
                    if (__builtin_popcount(j & reg) & 1) w.flags |= 1u << (8 + j);
                w.flags |= reg << 16;
                if (m->xmask && !w.xt) f *= 2.0;
                w.cre = f * cre;
                w.cim = f * cim;
                et.push_back(w);
            };
            e.diag = (int32_t)et.size();
            if (q == 0)
                for (const MonoTerm* m : p.diag) add(m);
            std::stable_sort(et.begin() + e.diag, et.end(),
                             [](const ETerm& x, const ETerm& y) { return x.flags >> 16 < y.flags >> 16; });
            e.term = (int32_t)et.size();
            for (const MonoTerm* m : s.terms) add(m);
            e.end = (int32_t)et.size();
            es.push_back(e);
        }
        l.hdr.nsegs = (int32_t)es.size();
        l.hdr.nterms = (int32_t)et.size();
        l.off = blob.size();
        blob.resize(blob.size() + es.size() + 2 * et.size());
        memcpy(&blob[l.off], es.data(), es.size() * sizeof(ESeg));
        memcpy(&blob[l.off + es.size()], et.data(), et.size() * sizeof(ETerm));
        most = std::max(most, es.size() + 2 * et.size());
        ls.push_back(l);
    }
    const size_t tile = sizeof(V) << tbits;
    KernelFit fit;
    int sf = kernel_fit(ctx, (const void*)kern, &fit);
    if (sf) return sf;
    // two tile buffers a CTA (the next tile arrives while this one is summed)
    int nbuf = ntiles > 1 ? 2 : 1;
    size_t smem = (size_t)nbuf * tile + most * 16 + 1024;
    int per_sm = 0;
    YAO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, smem));
    if (per_sm < 1) return fail(YAO_ERR_UNSUPPORTED, "expectation pass does not fit an SM");
    const int grid = (int)std::min<uint64_t>(ntiles, (uint64_t)per_sm * (uint64_t)ctx->num_sms);
    const size_t npart = 2 * (size_t)grid * ls.size();
    if (ctx->ensure_scratch(sizeof(double) * (npart + 2)) || ctx->ensure_host_pinned(3 * sizeof(double)))
        return YAO_ERR_OUT_OF_MEMORY;
    double* part = (double*)ctx->scratch;
    uint4* dblob = nullptr;
    YAO_CUDA(alloc_async(ctx, (void**)&dblob, blob.size() * sizeof(uint4)));
    YAO_CUDA(cudaMemcpyAsync(dblob, blob.data(), blob.size() * sizeof(uint4), cudaMemcpyHostToDevice, ctx->stream));
    for (size_t q = 0; q < ls.size(); q++) {
        EHdr& h = ls[q].hdr;
        CUtensorMap tmap;
        memset(&tmap, 0, sizeof(tmap));
        h.use_tma = ntiles > 1 && tma_enabled() && tma_make_plan(h.tb, tbits, n, sizeof(V), r->d, h.tma, &tmap) ? 1 : 0;
        h.nbuf = h.use_tma ? nbuf : 1;  // plain loads take turns in the first buffer: nothing arrives ahead
        ProfScope prof(ctx, "expect_tiles", (double)r->bytes());
        kern<<<grid, THREADS, smem, ctx->stream>>>((const V*)r->d, h, dblob + ls[q].off, part + 2 * (size_t)grid * q,
                                                   ctx->d_err, tmap);
        ctx->launches++;
    }
    YAO_CUDA(cudaGetLastError());
    YAO_CUDA(cudaFreeAsync(dblob, ctx->stream));
    int s = launch_final_sum(ctx, part, grid * (int)ls.size(), 2, part + npart);
    if (s) return s;
    double* hp = (double*)ctx->host_pinned;
    YAO_CUDA(cudaMemcpyAsync(hp, part + npart, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    YAO_CUDA(cudaMemcpyAsync(hp + 2, ctx->d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    ctx->err_unread.store(false);
    YAO_CUDA(cudaStreamSynchronize(ctx->stream));
    int herr;
    memcpy(&herr, hp + 2, sizeof(int));
    if (herr) {
        YAO_CUDA(cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));
        return fail(YAO_ERR_TIMEOUT, "expect: a bounded wait of a kernel (tile copy) gave up");
    }
    out->re += hp[0];
    out->im += hp[1];
    return YAO_OK;
}

int expect_sum(Ctx* ctx, const Reg* r, const std::vector<MonoTerm>& terms, Cx* out) {
    *out = Cx{0.0, 0.0};
    const uint32_t n = r->nbits;
    const bool c64 = r->precision != YAO_C128;
    const int low = c64 ? 4 : 3, tbits = std::min<int>((int)n, c64 ? 12 : 11);
    const bool whole = (int)n <= tbits;
    const uint64_t lowmask = whole ? 0 : ((1ull << low) - 1);
    const int cap = whole ? (int)n : tbits - low;
    // passes: a string joins the first whose tile takes its X mask.  Strings
    // with projectors, and masks wider than a tile, go one mask a launch; so
    // does everything on registers of less than 8 amplitudes.
    constexpr size_t kMaxPassTerms = 512;  // 16 KiB of descriptions
    std::vector<EPass> passes;
    std::vector<uint64_t> hi;
    std::vector<MonoTerm> rest;
    for (const MonoTerm& m : terms) {
        const bool pauli = m.d1mask == 0 && m.need0 == 0 && m.need1 == 0 && m.zero == 0;
        if (!pauli || n < (uint32_t)kEB || n > 33 || __builtin_popcountll(m.xmask & ~lowmask) > cap) {
            rest.push_back(m);
            continue;
        }
        size_t q = 0;
        for (; q < passes.size(); q++)
            if (__builtin_popcountll(hi[q] | (m.xmask & ~lowmask)) <= cap &&
                passes[q].diag.size() + passes[q].flips.size() < kMaxPassTerms)
                break;
        if (q == passes.size()) {
            passes.emplace_back();
            hi.push_back(0);
        }
        hi[q] |= m.xmask & ~lowmask;
        (m.xmask ? passes[q].flips : passes[q].diag).push_back(&m);
    }
    for (size_t q = 0; q < passes.size(); q++) {
        uint64_t t = hi[q] | lowmask;
        for (uint32_t b = 0; __builtin_popcountll(t) < tbits; b++) t |= 1ull << b;
        passes[q].tile = t;
    }
    if (!passes.empty()) {
        int s = c64 ? expect_tiles<float2, 12>(ctx, r, passes, out) : expect_tiles<double2, 11>(ctx, r, passes, out);
        if (s && s != YAO_ERR_OUT_OF_MEMORY) return s;
        if (s) {  // no memory for the descriptions: one mask a launch
            clear_error();
            rest = terms;
        }
    }
    if (rest.empty()) return YAO_OK;
    std::vector<Cx> vals;
    int s = expect_terms(ctx, r, rest, vals);
    if (s) return s;
    for (size_t t = 0; t < rest.size(); t++) {
        const Cx c = rest[t].coeff, v = vals[t];
        out->re += c.re * v.re - c.im * v.im;
        out->im += c.re * v.im + c.im * v.re;
    }
    return YAO_OK;
}

}  // namespace yao
