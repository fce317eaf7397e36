// Pauli sums over a complex128 statevector by shared-memory tiles: expectation
// values of many terms, and out = sum_t c_t P_t v, many X masks per read.
//
// Replaces the reference's one-contraction-per-term pauli_expectation_sv
// (tensorQ/statevector_sim.py:217-234) for Hamiltonians of many terms.
// pauli_group_kernel (reduce.cu) reads the state once per X mask: a 27-qubit
// Ising energy (27 X masks and the diagonal) is 28 passes. Here a pass stages
// tiles of 2^m amplitudes (32 KB: the low L bits, runs of 128 bytes, times up
// to 8 chosen high bits) and evaluates every term whose X mask lies in the
// tile's bits; a chain Hamiltonian of 27 qubits is 3 passes.
//
// Inside a tile, X masks are grouped into runs of at most 4 linearly
// independent masks (over GF(2)). A thread holds the 16 amplitudes base ^
// span(run basis) in registers, base enumerating the cosets, so that any mask
// of the span -- one bit, a pair, or a long string -- pairs registers known at
// compile time. A term's sign (-1)^popcount(x & z) splits into the register's
// part (a 16-bit table per term), the thread's part (one bit per term, fixed
// over the tiles) and the tile's part (one ballot per tile). The two members of
// a pair contribute equally, so a term costs two multiply-adds per pair; the
// diagonal terms share one 16-point Walsh transform of |v|^2 and cost one add
// each per 16 amplitudes.
//
// Measured (Ising terms, one state): 25 qubits 9.82 -> 7.12 ms, 17 qubits 230 ->
// 129 us, 8 qubits 50 -> 35 us against one pass per X mask. Where the general
// kernels (reduce.cu) are the faster ones, see expect_pays and apply_pays.
//
// What bounds it: the FP64 pipe (two multiply-adds per pair and term, four adds
// per amplitude for the diagonal). All sums run in a fixed order, so results are
// bitwise reproducible.
#include <algorithm>
#include <exception>
#include <vector>

#include "pauli_tiles.cuh"

namespace qgb {

constexpr int kPtMaxTerms = 44;   // terms per pass: 1 KB of per-thread sums each, so that two CTAs fit an SM
constexpr int kPtMaxRuns = 16;
constexpr int kPtMaxHigh = 8;
constexpr int kPtM = 11;        // tile bits: 32 KB
constexpr int kPtThreads = 128;  // 16 amplitudes each
constexpr int kPtWarps = kPtThreads / 32;
constexpr int kPtLow = 3;       // 128-byte runs

struct PtTerm {
    uint64_t z;      // whole Z mask, for the tile's part of the sign
    double coeff;
    int slot;
    uint16_t zt;     // Z mask on the tile's bits
    uint16_t wtab;   // bit c: parity of (combination c of the run basis) & z
    uint8_t x;       // X mask as a combination of the run basis (0: diagonal)
    uint8_t zr;      // bit j: parity of basis vector j & z
    uint8_t im;      // odd number of Y factors: the pair's imaginary part
    uint8_t neg;     // constant sign
};

struct PtRun {
    uint16_t basis[4];   // tile masks, reduced: basis[j] has the only set bit at piv[j]
    uint8_t piv[4];      // pivot tile bits, ascending
    int begin, end;      // its terms, diagonal ones first, by zr
    uint8_t dstart[17];  // diagonal terms of zr = r: begin + dstart[r] .. begin + dstart[r + 1]
};

struct PtArgs {
    int n, m, L, nruns, nterms, n_outer, accumulate;
    uint64_t tiles, stride;
    uint64_t high_off[4];                 // global offset of tile index bit log2(kPtThreads) + j
    int high_bits[kPtMaxHigh];            // global bit of tile bit L + h
    uint8_t outer_bits[2 * QGB_MAX_QUBITS];
    PtRun run[kPtMaxRuns];
    PtTerm term[kPtMaxTerms];
};
static_assert(sizeof(PtArgs) <= 4000, "kernel parameter space");

// Tile index of an amplitude in shared memory: its low three bits XORed with a
// fold of the higher ones, so that the lanes of a warp reach distinct banks
// whichever bits a run holds in registers. Linear over XOR.
__device__ __forceinline__ uint32_t pt_swz(uint32_t e) { return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u); }

__device__ __forceinline__ double flip(double v, uint32_t sign) {
    return __hiloint2double(__double2hiint(v) ^ int(sign), __double2loint(v));
}

__device__ __forceinline__ uint32_t pt_base(uint32_t g, const PtRun& r) {
#pragma unroll
    for (int j = 0; j < 4; ++j) g = ((g >> r.piv[j]) << (r.piv[j] + 1)) | (g & ((1u << r.piv[j]) - 1u));
    return g;
}

// Global offset of tile `t`'s first amplitude: its bits at the outer positions,
// gathered by the warp (every lane of the warp calls it with the same t).
__device__ __forceinline__ uint64_t pt_outer(uint64_t t, const PtArgs& a) {
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {  // two rounds: up to 64 outer bits
        const int j = lane + 32 * r;
        if (j < a.n_outer && ((t >> j) & 1ull)) {
            const int b = a.outer_bits[j];
            if (b < 32) lo |= 1u << b;
            else hi |= 1u << (b - 32);
        }
    }
    lo = __reduce_or_sync(0xffffffffu, lo);
    hi = __reduce_or_sync(0xffffffffu, hi);
    return (uint64_t(hi) << 32) | lo;
}

// This thread's amplitudes of a tile are e = tid + j * kPtThreads, 16 of a full
// one: the part of their global offset that comes from tid.
__device__ __forceinline__ uint64_t pt_gran_off(const PtArgs& a) {
    const uint32_t e = threadIdx.x;
    uint64_t off = e & ((1u << a.L) - 1u);
    const uint32_t h = e >> a.L;
    for (int j = 0; j < a.m - a.L; ++j) off |= uint64_t((h >> j) & 1u) << a.high_bits[j];
    return off;
}

__device__ __forceinline__ void pt_load(double2* tile, const double2* s, uint64_t off, uint64_t outer, const PtArgs& a) {
#pragma unroll
    for (int j = 0; j < (1 << kPtM) / kPtThreads; ++j) {
        const uint32_t g = threadIdx.x + uint32_t(j) * kPtThreads;
        if (g >= (1u << a.m)) break;
        const uint64_t go = off | (j & 1 ? a.high_off[0] : 0) | (j & 2 ? a.high_off[1] : 0) | (j & 4 ? a.high_off[2] : 0) |
                            (j & 8 ? a.high_off[3] : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         uint32_t(__cvta_generic_to_shared(tile + pt_swz(g)))),
                     "l"(s + (outer | go))
                     : "memory");
    }
}

// 16 amplitudes of a coset, register c = combination c of the run basis.
__device__ __forceinline__ void pt_offsets(uint32_t (&so)[16], const PtRun& r) {
    so[0] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t v = pt_swz(r.basis[j]);
#pragma unroll
        for (int c = 0; c < (1 << j); ++c) so[(1 << j) + c] = so[c] ^ v;
    }
}

// Sum over the 8 pairs {c, c ^ X} of the real (IM: imaginary) part of
// conj(v[c ^ X]) v[c], signed by the register's part of the term's sign
// (SIGNED = false: all plus).
template <int X, bool IM, bool SIGNED>
__device__ __forceinline__ double pt_pairs(const double2 (&v)[16], uint32_t wtab) {
    constexpr int top = X >= 8 ? 8 : X >= 4 ? 4 : X >= 2 ? 2 : 1;
    asm volatile("" : "+r"(wtab));  // its shifts stay inside this case (hoisted over the switch they spill)
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c)
        if (!(c & top)) {
            const double2 y = v[c ^ X], x = v[c];
            double& s = (c & (top == 1 ? 2 : 1)) ? s1 : s0;
            const uint32_t sg = SIGNED ? (wtab << (31 - c)) & 0x80000000u : 0u;
            if constexpr (IM) {
                s = fma(y.x, SIGNED ? flip(x.y, sg) : x.y, s);
                s = fma(-y.y, SIGNED ? flip(x.x, sg) : x.x, s);
            } else {
                s = fma(y.x, SIGNED ? flip(x.x, sg) : x.x, s);
                s = fma(y.y, SIGNED ? flip(x.y, sg) : x.y, s);
            }
        }
    return s0 + s1;
}

template <int X>
__device__ __forceinline__ double pt_pairs(const double2 (&v)[16], bool im, uint32_t wtab) {
    if (im) return pt_pairs<X, true, true>(v, wtab);
    if (wtab) return pt_pairs<X, false, true>(v, wtab);
    return pt_pairs<X, false, false>(v, wtab);
}

__device__ __forceinline__ double pt_pairs_of(int x, const double2 (&v)[16], bool im, uint32_t wtab) {
    switch (x) {
        case 1: return pt_pairs<1>(v, im, wtab);
        case 2: return pt_pairs<2>(v, im, wtab);
        case 3: return pt_pairs<3>(v, im, wtab);
        case 4: return pt_pairs<4>(v, im, wtab);
        case 5: return pt_pairs<5>(v, im, wtab);
        case 6: return pt_pairs<6>(v, im, wtab);
        case 7: return pt_pairs<7>(v, im, wtab);
        case 8: return pt_pairs<8>(v, im, wtab);
        case 9: return pt_pairs<9>(v, im, wtab);
        case 10: return pt_pairs<10>(v, im, wtab);
        case 11: return pt_pairs<11>(v, im, wtab);
        case 12: return pt_pairs<12>(v, im, wtab);
        case 13: return pt_pairs<13>(v, im, wtab);
        case 14: return pt_pairs<14>(v, im, wtab);
        default: return pt_pairs<15>(v, im, wtab);
    }
}

// One bit per term (two words): parity of the thread's base & z, and the constant sign.
__device__ __forceinline__ void pt_thread_signs(uint32_t (&sg)[2], uint32_t g, const PtArgs& a) {
    sg[0] = sg[1] = 0;
    for (int r = 0; r < a.nruns; ++r) {
        const uint32_t base = pt_base(g, a.run[r]);
        for (int t = a.run[r].begin; t < a.run[r].end; ++t) {
            const uint32_t p = (__popc(base & a.term[t].zt) & 1u) ^ a.term[t].neg;
            if (t < 32) sg[0] |= p << t;
            else sg[1] |= p << (t - 32);
        }
    }
}

// One bit per term: parity of the tile's offset & z (every lane of the warp takes part).
__device__ __forceinline__ void pt_tile_signs(uint32_t (&tg)[2], uint64_t outer, const PtArgs& a) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const int t = lane + 32 * w;
        const uint32_t p = t < a.nterms ? uint32_t(__popcll(outer & a.term[t].z)) & 1u : 0u;
        tg[w] = __ballot_sync(0xffffffffu, p);
    }
}

__device__ __forceinline__ uint32_t pt_sign(const uint32_t (&sg)[2], int t) {
    return ((t < 32 ? sg[0] : sg[1]) << (31 - (t & 31))) & 0x80000000u;
}

// partials[(b * nslots + slot) * gridDim.x + blk]
__global__ void __launch_bounds__(kPtThreads, 2)
    pauli_tile_kernel(const double2* __restrict__ sv, const __grid_constant__ PtArgs a, int nslots,
                      double* __restrict__ partials) {
    constexpr int NT = kPtThreads, NW = kPtWarps;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t tl = 1u << a.m;
    double2* tile0 = reinterpret_cast<double2*>(smem);
    double* acc = reinterpret_cast<double*>(tile0 + 2 * size_t(tl < 16 ? 16 : tl));
    double* dsum = reinterpret_cast<double*>(acc + size_t(a.nterms) * NT);  // [term][warp]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t b = blockIdx.y;
    const double2* s = sv + b * int64_t(a.stride);
    const uint64_t goff = pt_gran_off(a);
    const bool on = uint32_t(tid) < (tl >> 4);
    for (int t = 0; t < a.nterms; ++t) acc[t * NT + tid] = 0.0;
    uint32_t tsg[2];
    pt_thread_signs(tsg, tid, a);
    uint64_t t = blockIdx.x;
    uint64_t outer = pt_outer(t, a);
    if (t < a.tiles) pt_load(tile0, s, goff, outer, a);
    asm volatile("cp.async.commit_group;" ::: "memory");
    int buf = 0;
    for (; t < a.tiles; t += gridDim.x) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this tile has landed; the other buffer's readers are done
        const double2* tile = tile0 + buf * size_t(tl);
        const uint64_t next = t + gridDim.x;
        const uint64_t outer_next = pt_outer(next < a.tiles ? next : t, a);
        if (next < a.tiles) pt_load(tile0 + (buf ^ 1) * size_t(tl), s, goff, outer_next, a);
        asm volatile("cp.async.commit_group;" ::: "memory");
        uint32_t sg[2];
        pt_tile_signs(sg, outer, a);
        sg[0] ^= tsg[0];
        sg[1] ^= tsg[1];
        if (on) {
            for (int r = 0; r < a.nruns; ++r) {
                const PtRun& run = a.run[r];
                const uint32_t sb = pt_swz(pt_base(tid, run));
                double2 v[16];
                {
                    uint32_t so[16];
                    pt_offsets(so, run);
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = tile[sb ^ so[c]];
                }
                int q = run.begin + run.dstart[16];
                if (q > run.begin) {
                    double p[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) p[c] = v[c].x * v[c].x + v[c].y * v[c].y;
#pragma unroll
                    for (int h = 1; h < 16; h <<= 1)
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            if (!(c & h)) {
                                const double u = p[c], w = p[c | h];
                                p[c] = u + w;
                                p[c | h] = u - w;
                            }
#pragma unroll
                    for (int z = 0; z < 16; ++z)
                        for (int k = run.begin + run.dstart[z]; k < run.begin + run.dstart[z + 1]; ++k)
                            acc[k * NT + tid] += flip(p[z], pt_sign(sg, k));
                }
                for (; q < run.end; ++q) {
                    const double p = pt_pairs_of(a.term[q].x, v, a.term[q].im, a.term[q].wtab);
                    acc[q * NT + tid] += flip(p, pt_sign(sg, q));
                }
            }
        }
        buf ^= 1;
        outer = outer_next;
    }
    for (int k0 = 0; k0 < a.nterms; k0 += 32) {  // a warp's sums, 32 terms a time
        double mine = 0.0;
        const int kn = a.nterms - k0 < 32 ? a.nterms - k0 : 32;
        for (int k = 0; k < kn; ++k) {
            double x = acc[(k0 + k) * NT + tid];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == k) mine = x;
        }
        if (lane < kn) dsum[(k0 + lane) * NW + warp] = mine;
    }
    __syncthreads();
    if (tid < a.nterms) {
        double x = 0.0;
        for (int w = 0; w < NW; ++w) x += dsum[tid * NW + w];
        partials[(b * nslots + a.term[tid].slot) * int64_t(gridDim.x) + blockIdx.x] = x * a.term[tid].coeff;
    }
}

// out += sum of the pass's terms applied to sv (accumulate = 0: out = ...). The
// tile of out stays in shared memory over the runs; every run adds its terms to
// the thread's 16 entries in registers. The diagonal terms are gathered into 16
// Walsh coefficients and transformed once, so they cost one complex-by-real
// product per amplitude however many there are.
template <int X>
__device__ __forceinline__ void pt_add(double2 (&o)[16], const double2 (&v)[16], double f, bool im, uint32_t wtab) {
    asm volatile("" : "+r"(wtab));
#pragma unroll
    for (int c = 0; c < 16; ++c) {  // out at c from x = c ^ X: the sign is x's
        const double2 x = v[c ^ X];
        const double g = flip(f, (wtab << (31 - (c ^ X))) & 0x80000000u);
        if (im) {
            o[c].x = fma(-g, x.y, o[c].x);
            o[c].y = fma(g, x.x, o[c].y);
        } else {
            o[c].x = fma(g, x.x, o[c].x);
            o[c].y = fma(g, x.y, o[c].y);
        }
    }
}

__device__ __forceinline__ void pt_add_of(int x, double2 (&o)[16], const double2 (&v)[16], double f, bool im, uint32_t w) {
    switch (x) {
        case 1: return pt_add<1>(o, v, f, im, w);
        case 2: return pt_add<2>(o, v, f, im, w);
        case 3: return pt_add<3>(o, v, f, im, w);
        case 4: return pt_add<4>(o, v, f, im, w);
        case 5: return pt_add<5>(o, v, f, im, w);
        case 6: return pt_add<6>(o, v, f, im, w);
        case 7: return pt_add<7>(o, v, f, im, w);
        case 8: return pt_add<8>(o, v, f, im, w);
        case 9: return pt_add<9>(o, v, f, im, w);
        case 10: return pt_add<10>(o, v, f, im, w);
        case 11: return pt_add<11>(o, v, f, im, w);
        case 12: return pt_add<12>(o, v, f, im, w);
        case 13: return pt_add<13>(o, v, f, im, w);
        case 14: return pt_add<14>(o, v, f, im, w);
        default: return pt_add<15>(o, v, f, im, w);
    }
}

__global__ void __launch_bounds__(kPtThreads, 2)
    pauli_tile_apply_kernel(const double2* __restrict__ sv, double2* __restrict__ out, const __grid_constant__ PtArgs a) {
    constexpr int NT = kPtThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t tl = 1u << a.m;
    double2* tile = reinterpret_cast<double2*>(smem);
    double2* ot = tile + tl;
    const int tid = threadIdx.x;
    const double2* s = sv + int64_t(blockIdx.y) * int64_t(a.stride);
    double2* os = out + int64_t(blockIdx.y) * int64_t(a.stride);
    const uint64_t goff = pt_gran_off(a);
    const bool on = uint32_t(tid) < (tl >> 4);
    uint32_t tsg[2];
    pt_thread_signs(tsg, tid, a);
    for (uint64_t t = blockIdx.x; t < a.tiles; t += gridDim.x) {
        const uint64_t outer = pt_outer(t, a);
        pt_load(tile, s, goff, outer, a);
        if (a.accumulate) pt_load(ot, os, goff, outer, a);
        asm volatile("cp.async.commit_group;" ::: "memory");
        uint32_t sg[2];
        pt_tile_signs(sg, outer, a);
        sg[0] ^= tsg[0];
        sg[1] ^= tsg[1];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        for (int r = 0; r < a.nruns; ++r) {
            const PtRun& run = a.run[r];
            if (on) {
                const uint32_t sb = pt_swz(pt_base(tid, run));
                uint32_t so[16];
                pt_offsets(so, run);
                double2 v[16], o[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    v[c] = tile[sb ^ so[c]];
                    o[c] = r == 0 && !a.accumulate ? make_double2(0.0, 0.0) : ot[sb ^ so[c]];
                }
                int q = run.begin + run.dstart[16];
                if (q > run.begin) {
                    double d[16];
#pragma unroll
                    for (int z = 0; z < 16; ++z) {
                        d[z] = 0.0;
                        for (int k = run.begin + run.dstart[z]; k < run.begin + run.dstart[z + 1]; ++k)
                            d[z] += flip(a.term[k].coeff, pt_sign(sg, k));
                    }
#pragma unroll
                    for (int h = 1; h < 16; h <<= 1)
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            if (!(c & h)) {
                                const double u = d[c], w = d[c | h];
                                d[c] = u + w;
                                d[c | h] = u - w;
                            }
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        o[c].x = fma(d[c], v[c].x, o[c].x);
                        o[c].y = fma(d[c], v[c].y, o[c].y);
                    }
                }
                for (; q < run.end; ++q)
                    pt_add_of(a.term[q].x, o, v, flip(a.term[q].coeff, pt_sign(sg, q)), a.term[q].im,
                                 a.term[q].wtab);
#pragma unroll
                for (int c = 0; c < 16; ++c) ot[sb ^ so[c]] = o[c];
            }
            __syncthreads();
        }
        const uint32_t grans = tl;
#pragma unroll
        for (int j = 0; j < (1 << kPtM) / NT; ++j) {
            const uint32_t g = tid + uint32_t(j) * NT;
            if (g >= grans) break;
            const uint64_t go = goff | (j & 1 ? a.high_off[0] : 0) | (j & 2 ? a.high_off[1] : 0) |
                                (j & 4 ? a.high_off[2] : 0) | (j & 8 ? a.high_off[3] : 0);
            *reinterpret_cast<float4*>(os + (outer | go)) = *reinterpret_cast<const float4*>(ot + pt_swz(g));
        }
        __syncthreads();  // the tile has been read before the next one is copied over it
    }
}

}  // namespace qgb

using namespace qgb;

namespace qgb_host {

namespace {

struct Plan {
    std::vector<PtArgs> passes;
};

// The state's bits of a tile, as a local mask.
uint16_t local_mask(uint64_t g, const PtArgs& a) {
    uint32_t o = uint32_t(g & ((uint64_t(1) << a.L) - 1));
    for (int j = 0; j < a.m - a.L; ++j) o |= uint32_t((g >> a.high_bits[j]) & 1) << (a.L + j);
    return uint16_t(o);
}

// One run being built: an echelon basis of its X masks.
struct RunPlan {
    std::vector<uint32_t> masks;                    // the masks taken (local)
    std::vector<uint32_t> basis;                    // independent masks, reduced
    std::vector<std::pair<int, uint32_t>> terms;    // (term, local X mask)
};

uint32_t reduce_by(uint32_t v, const std::vector<uint32_t>& basis) {
    for (uint32_t b : basis)
        if (v & (1u << (31 - __builtin_clz(b)))) v ^= b;
    return v;
}

void add_basis(std::vector<uint32_t>& basis, uint32_t v) {
    const int p = 31 - __builtin_clz(v);
    for (uint32_t& b : basis)
        if (b & (1u << p)) b ^= v;
    basis.push_back(v);
}

// Fills in the runs and terms of one pass whose geometry is set.
// expect: a pair is summed once (factor 2) as Re or Im of conj(v[y]) v[x]; i^ny times
// it has the real part Re, -Im, -Re, Im for ny = 0..3. Otherwise the terms are
// applied: 1, i, -1, -i.
bool build_pass(PtArgs& a, const std::vector<int>& taken, const PauliTerm* terms, bool expect) {
    std::vector<RunPlan> runs;
    std::vector<int> diag;
    for (int t : taken) {
        if (terms[t].x == 0) {
            diag.push_back(t);
            continue;
        }
        const uint32_t x = local_mask(terms[t].x, a);
        RunPlan* home = nullptr;
        for (RunPlan& r : runs)  // a run whose span has the mask
            if (reduce_by(x, r.basis) == 0) { home = &r; break; }
        if (!home)
            for (RunPlan& r : runs)
                if (r.basis.size() < 4) { home = &r; break; }
        if (!home) {
            runs.emplace_back();
            home = &runs.back();
        }
        const uint32_t red = reduce_by(x, home->basis);
        if (red) add_basis(home->basis, red);
        home->terms.emplace_back(t, x);
    }
    if (!diag.empty()) {
        if (runs.empty()) runs.emplace_back();
        for (int t : diag) runs[0].terms.emplace_back(t, 0u);
    }
    if (runs.size() > size_t(kPtMaxRuns)) return false;
    a.nruns = int(runs.size());
    a.nterms = 0;
    for (int r = 0; r < a.nruns; ++r) {
        RunPlan& rp = runs[r];
        for (int b = 0; b < a.m && rp.basis.size() < 4; ++b) {  // padded to four vectors with tile bits
            const uint32_t red = reduce_by(1u << b, rp.basis);
            if (red) add_basis(rp.basis, red);
        }
        std::sort(rp.basis.begin(), rp.basis.end(), [](uint32_t x, uint32_t y) {
            return __builtin_clz(x) > __builtin_clz(y);  // ascending leading bit
        });
        PtRun& run = a.run[r];
        for (int j = 0; j < 4; ++j) {
            run.basis[j] = uint16_t(rp.basis[j]);
            run.piv[j] = uint8_t(31 - __builtin_clz(rp.basis[j]));
        }
        auto zr_of = [&](int t) {
            const uint32_t zt = local_mask(terms[t].z, a);
            int zr = 0;
            for (int j = 0; j < 4; ++j) zr |= (__builtin_popcount(run.basis[j] & zt) & 1) << j;
            return zr;
        };
        std::stable_sort(rp.terms.begin(), rp.terms.end(), [&](const auto& p, const auto& q) {
            if ((p.second == 0) != (q.second == 0)) return p.second == 0;
            return p.second == 0 && zr_of(p.first) < zr_of(q.first);
        });
        run.begin = a.nterms;
        int nd = 0;
        for (int z = 0; z <= 16; ++z) run.dstart[z] = 0;
        for (const auto& [t, x] : rp.terms) {
            if (a.nterms >= kPtMaxTerms) return false;
            PtTerm& pt = a.term[a.nterms++];
            pt.z = terms[t].z;
            pt.slot = terms[t].slot;
            pt.coeff = terms[t].coeff * (x && expect ? 2.0 : 1.0);
            pt.zt = local_mask(terms[t].z, a);
            pt.zr = uint8_t(zr_of(t));
            pt.x = 0;
            for (int j = 0; j < 4; ++j) pt.x |= uint8_t(((x >> run.piv[j]) & 1u) << j);
            pt.wtab = 0;
            for (int c = 0; c < 16; ++c) pt.wtab |= uint16_t((__builtin_popcount(c & pt.zr) & 1) << c);
            pt.im = uint8_t(terms[t].ny & 1);
            pt.neg = uint8_t(((terms[t].ny + (expect ? 1 : 0)) >> 1) & 1);
            if (!x) {
                ++nd;
                for (int z = pt.zr + 1; z <= 16; ++z) run.dstart[z] = uint8_t(nd);
            }
        }
        run.end = a.nterms;
    }
    return true;
}

// Passes for the terms, or an empty plan when a term's X mask fits no tile.
Plan make_plan(int n, const PauliTerm* terms, int nterms, uint64_t stride, bool expect) {
    Plan plan;
    const int m = n < kPtM ? n : kPtM;
    const int L = n <= kPtM ? m : kPtLow;
    const int H = m - L;
    const uint64_t low = (uint64_t(1) << L) - 1;
    for (int t = 0; t < nterms; ++t)
        if (__builtin_popcountll(terms[t].x & ~low) > H) return plan;  // an X mask wider than a tile
    std::vector<int> left(nterms);
    for (int t = 0; t < nterms; ++t) left[t] = t;
    // masks in ascending order of their top bit, so that neighbouring bits share a pass
    std::stable_sort(left.begin(), left.end(), [&](int p, int q) { return terms[p].x < terms[q].x; });
    // (a full pass stops looking: what it passed over goes in front of the rest)
    for (size_t at = 0; at < left.size();) {
        uint64_t high = 0;
        std::vector<int> taken, over;
        size_t i = at;
        for (; i < left.size() && int(taken.size()) < kPtMaxTerms; ++i) {
            const uint64_t need = high | (terms[left[i]].x & ~low);
            if (__builtin_popcountll(need) <= H) {
                high = need;
                taken.push_back(left[i]);
            } else {
                over.push_back(left[i]);
            }
        }
        at = i - over.size();
        std::copy(over.begin(), over.end(), left.begin() + int64_t(at));
        for (int b = L; b < n && __builtin_popcountll(high) < H; ++b) high |= uint64_t(1) << b;
        plan.passes.emplace_back();
        PtArgs& a = plan.passes.back();
        a = PtArgs{};
        a.n = n;
        a.m = m;
        a.L = L;
        a.stride = stride;
        int h = 0;
        for (int b = L; b < n; ++b) {
            if ((high >> b) & 1) a.high_bits[h++] = b;
            else a.outer_bits[a.n_outer++] = uint8_t(b);
        }
        a.tiles = uint64_t(1) << (n - m);
        for (int j = 0; j < 4; ++j) {  // tile index bit log2(kPtThreads) + j
            const uint32_t e = uint32_t(kPtThreads) << j;
            if (e < (1u << m)) {
                const int tb = __builtin_ctz(e);
                a.high_off[j] = uint64_t(1) << (tb < L ? tb : a.high_bits[tb - L]);
            }
        }
        if (!build_pass(a, taken, terms, expect)) return Plan{};
    }
    return plan;
}

int expect_impl(const void* sv, int n, const PauliTerm* terms, int nterms, int64_t batch, int64_t stride, int max_blocks,
                double* partials, int* nblk, cudaStream_t st) {
    const Plan plan = make_plan(n, terms, nterms, uint64_t(stride), true);
    if (plan.passes.empty()) return QGB_EDECLINE;
    // one wave of two CTAs per SM; batches, whose states split unevenly over the SMs, in smaller pieces
    uint64_t bx = (uint64_t(sm_count()) * (batch == 1 ? 2 : 8) + uint64_t(batch) - 1) / uint64_t(batch);
    bx = std::min<uint64_t>(std::max<uint64_t>(bx, 1), std::min<uint64_t>(plan.passes[0].tiles, uint64_t(max_blocks)));
    for (const PtArgs& a : plan.passes) {
        const size_t smem = 2 * sizeof(double2) * (size_t(1) << a.m) + sizeof(double) * size_t(a.nterms) * kPtThreads +
                            sizeof(double) * size_t(a.nterms) * kPtWarps;
        constexpr int most = int(2 * sizeof(double2) * (size_t(1) << kPtM) +
                                 kPtMaxTerms * (sizeof(double) * kPtThreads + sizeof(double) * kPtWarps));
        static std::atomic<uint64_t> done{0};
        int rc = allow_smem(pauli_tile_kernel, most, done, "pauli tiles attribute");
        if (rc) return rc;
        pauli_tile_kernel<<<dim3(unsigned(bx), unsigned(batch)), kPtThreads, smem, st>>>((const double2*)sv, a, nterms,
                                                                                         partials);
        rc = check_launch("pauli tiles");
        if (rc) return rc;
    }
    *nblk = int(bx);
    return QGB_OK;
}

int apply_impl(const void* sv, void* out, int n, const PauliTerm* terms, int nterms, int64_t batch, int64_t stride,
               cudaStream_t st) {
    Plan plan = make_plan(n, terms, nterms, uint64_t(stride), false);
    if (plan.passes.empty()) return QGB_EDECLINE;
    bool first = true;
    for (PtArgs& a : plan.passes) {
        a.accumulate = first ? 0 : 1;
        first = false;
        const size_t smem = 2 * sizeof(double2) * (size_t(1) << a.m);
        static std::atomic<uint64_t> done{0};
        int rc = allow_smem(pauli_tile_apply_kernel, 2 * sizeof(double2) << kPtM, done, "pauli apply attribute");
        if (rc) return rc;
        uint64_t bx = (uint64_t(sm_count()) * 12 + uint64_t(batch) - 1) / uint64_t(batch);
        bx = std::min<uint64_t>(std::max<uint64_t>(bx, 1), a.tiles);
        pauli_tile_apply_kernel<<<dim3(unsigned(bx), unsigned(batch)), kPtThreads, smem, st>>>(
            (const double2*)sv, (double2*)out, a);
        rc = check_launch("pauli apply tiles");
        if (rc) return rc;
    }
    return QGB_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) % 16) == 0; }

// complex128 only: the complex64 kernels (reduce.cu) add float32 products in an
// order that fixes every bit of their float64 results, which callers compare
// between runs and builds; complex128 results move at the 1e-16 level only.
// From 5 bits up (two threads of 16 amplitudes).
bool eligible(const void* sv, int dtype, int n) { return dtype == QGB_C128 && n >= 5 && aligned16(sv); }

// Expectation values. Up to 11 bits one tile takes a pass of at most 44 terms, 57 us whatever its masks; the
// general kernel takes a launch for every run of up to 32 terms on one mask, 6 to 28 us at 8 bits. So at
// 9 bits and below sums of many terms a mask stay there (us, tiles / general: 8 bits, 1 term a mask 59 / 71, 4
// 123 / 105, 8 184 / 152, 32 331 / 219; 9 bits, 16 341 / 435, 32 333 / 271; 10 bits, 32 345 / 382; 14 bits,
// 1 110 / 162, 32 600 / 1071).
bool expect_pays(int n, const PauliTerm* terms, int nterms) {
    if (n > 9) return true;
    int runs = 0;
    for (int t = 0, k = 0; t < nterms; ++t, ++k)
        if (t == 0 || terms[t].x != terms[t - 1].x || k == 32) {
            ++runs;
            k = 0;
        }
    return n < 9 ? nterms < 4 * runs : nterms < 24 * runs;
}

// Applied sums. The general kernel is one launch that reads the state once a term, through the caches: a state
// in L1 or L2 costs it little, and it reads and writes `out` once. Tiles pay from 20 bits, and
// where all terms are diagonal, one pass for 44 of them, from 16 (us, tiles / general: Ising terms 12 bits 48 / 11,
// 17 bits 60 / 33, 20 bits 231 / 238, 22 bits 817 / 1010; 128 diagonal terms 14 bits 44 / 41, 17 bits
// 44 / 115, 20 bits 101 / 788; 128 dense terms 12 bits 376 / 48).
bool apply_pays(int n, const PauliTerm* terms, int nterms) {
    return n >= 20 || (n >= 16 && std::all_of(terms, terms + nterms, [](const PauliTerm& t) { return t.x == 0; }));
}

}  // namespace

int pauli_tiles_expect(const void* sv, int dtype, int n, const PauliTerm* terms, int nterms, int64_t batch,
                       int64_t stride, int max_blocks, double* partials, int* nblk, cudaStream_t st) {
    if (!eligible(sv, dtype, n) || !expect_pays(n, terms, nterms)) return QGB_EDECLINE;
    try {
        return expect_impl(sv, n, terms, nterms, batch, stride, max_blocks, partials, nblk, st);
    } catch (const std::exception&) {  // no memory for the plan: nothing has been launched
        return QGB_EDECLINE;
    }
}

int pauli_tiles_apply(const void* sv, void* out, int dtype, int n, const PauliTerm* terms, int nterms, int64_t batch,
                      int64_t stride, cudaStream_t st) {
    if (!eligible(sv, dtype, n) || !aligned16(out) || !apply_pays(n, terms, nterms)) return QGB_EDECLINE;
    try {
        return apply_impl(sv, out, n, terms, nterms, batch, stride, st);
    } catch (const std::exception&) {
        return QGB_EDECLINE;
    }
}

}  // namespace qgb_host
