// Adjoint reverse sweep with many gates per pass over the state and co-state.
//
// The reference differentiates a circuit through torch autograd, which stores
// every intermediate state (core/param_gates.py:21-49 builds the matrices,
// applications/compilation.py:73-133 calls backward). The adjoint method
// walks the gates backwards carrying phi (the state, uncomputed gate by gate)
// and lam (the co-state); qgb_adjoint_step does one HBM pass over both per
// gate. Here the host groups consecutive gates of the reverse order whose
// sites fit one tile (the geometry of the forward sweeps, sweep.cu): a CTA
// stages the tile of phi and of lam in shared memory (cp.async, double
// buffered), and for every op, in order (consecutive ops on the same sites in
// one register pass),
//   * for a rotation exp(-i theta P) whose derivative is wanted: adds
//     Im sum conj(lam) (P phi) over the tile's groups (float partial per
//     thread, a fixed xor-shuffle tree per warp, a compensated float
//     accumulator per (op, warp) in shared memory -- float64 for complex128);
//   * applies U^dagger to both tiles.
// Work is split into chunks of consecutive tiles, each inside one state; a
// chunk's accumulators are summed over the warps in order and stored as one
// partial per (chunk, op), and a second kernel adds the chunks of each state
// in order: bitwise reproducible, no atomics. The scratch size depends on the
// problem only (chunks per state fixed by the batch size).
#include <cstring>

#include "qgb_common.cuh"

namespace qgb {

constexpr int kAdjMaxThreads = 512;
constexpr int kAdjMaxWarps = kAdjMaxThreads / 32;

struct AdjSweepArgs {
    int n, L, H, m, n_ops;
    int high_bits[QGB_SWEEP_MAX_HIGH];
    int n_outer;
    int outer_bits[2 * QGB_MAX_QUBITS];
    int op_k[QGB_SWEEP_MAX_OPS];
    int op_pos[QGB_SWEEP_MAX_OPS][2];
    int64_t op_mat[QGB_SWEEP_MAX_OPS];
    int op_out[QGB_SWEEP_MAX_OPS];
    int gcol[QGB_SWEEP_MAX_OPS][4];
    float2 gval[QGB_SWEEP_MAX_OPS][4];  // entries of a Pauli product: 0, +-1, +-i (exact in float)
    int64_t mat_stride, batch, sv_stride;
    // register runs: consecutive ops on at most `rbits` tile bits, applied to groups of
    // 2^rbits amplitudes of both tiles held in registers (0: one shared-memory pass per op)
    int rbits;
    int n_runs;
    int run_len[QGB_SWEEP_MAX_OPS];     // at a run's first op: its op count (0 elsewhere)
    int run_pos[QGB_SWEEP_MAX_OPS][4];  // at a run's first op: the tile bit of each local bit of the run
    int op_lpos[QGB_SWEEP_MAX_OPS][2];  // every op's sites as local bits of its run
    int op_gcls[QGB_SWEEP_MAX_OPS];     // generator class of a wanted derivative (kGenNone: none)
    uint64_t tiles;        // tiles per state, 2^tile_shift
    uint64_t chunk_tiles;  // tiles per chunk, 2^chunk_shift
    int tile_shift, chunk_shift;
    uint64_t chunks;       // chunks over all states
};

__host__ __device__ inline int adj_chunks_per_state(uint64_t tiles, int64_t batch) {
    // ~2048 chunks in all (several per CTA on 152 SMs), a power of two per state
    uint64_t want = 2048 / uint64_t(batch > 0 ? batch : 1);
    uint64_t c = 1;
    while (c * 2 <= want && c * 2 <= tiles) c *= 2;
    return int(c);
}

__device__ __forceinline__ void cp_async16_adj(void* smem_dst, const void* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src)
                 : "memory");
}

constexpr int kAdjMaxRun = 4;  // consecutive ops on the same sites handled in one register pass

// A run of R consecutive ops on the same K sites (R <= kAdjMaxRun): per group
// of partner amplitudes, one load and one store of the staged tiles; for each
// op of the run in order, the derivative (if wanted) at the op's output, then
// U^dagger on both (diagonal ones by one product per amplitude). A single op
// without derivative whose U^dagger permutes (CNOT, SWAP, X) is a copy from the
// permuted tile offsets. threads tid = 0..nthr-1 of the CTA.
template <typename T, int K, int R>
__device__ __forceinline__ void adj_tile_run(cplx<T>* __restrict__ pt, cplx<T>* __restrict__ lt, int m,
                                             const AdjSweepArgs& a, int op0, const cplx<T>* __restrict__ ush,
                                             typename WAccOf<T>::type* __restrict__ red, int tid, int nthr) {
    constexpr int D = 1 << K;
    using C = cplx<T>;
    int pos[K], srt[K];
#pragma unroll
    for (int j = 0; j < K; ++j) pos[j] = srt[j] = a.op_pos[op0][j];
    if constexpr (K == 2) {
        if (srt[0] > srt[1]) {
            const int t = srt[0];
            srt[0] = srt[1];
            srt[1] = t;
        }
    }
    uint32_t soff[D];
#pragma unroll
    for (int r = 0; r < D; ++r) {
        uint32_t o = 0;
#pragma unroll
        for (int j = 0; j < K; ++j) o |= uint32_t((r >> (K - 1 - j)) & 1) << pos[j];
        soff[r] = swz<T>(o);
    }
    C ud[R][D * D];
    bool want[R];
    C gv[R][D];
    int gc[R][D];
#pragma unroll
    for (int q = 0; q < R; ++q) {
#pragma unroll
        for (int e = 0; e < D * D; ++e) ud[q][e] = ush[(op0 + q) * 16 + e];  // U^dagger, staged per state
        want[q] = a.op_out[op0 + q] >= 0;
#pragma unroll
        for (int r = 0; r < D; ++r) {
            gv[q][r] = mk<T>(T(a.gval[op0 + q][r].x), T(a.gval[op0 + q][r].y));
            gc[q][r] = a.gcol[op0 + q][r];
        }
    }
    // U^dagger diagonal (e.g. RZ, CZ): two complex products per row instead of a row of the matrix
    bool diag[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        bool d = true;
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
            for (int c = 0; c < D; ++c)
                if (r != c) d = d && ud[q][r * D + c].x == T(0) && ud[q][r * D + c].y == T(0);
        diag[q] = d;
    }
    const uint32_t groups = 1u << (m - K);
    if constexpr (R == 1) {
        // a single op without derivative whose U^dagger is a permutation with unit entries
        // (CNOT, SWAP, X): out[r] = in[col(r)], read straight from the permuted tile offsets
        if (!want[0]) {
            int col[D];
            bool perm = true;
#pragma unroll
            for (int r = 0; r < D; ++r) {
                int nz = 0;
                col[r] = 0;
#pragma unroll
                for (int c = 0; c < D; ++c) {
                    const C u = ud[0][r * D + c];
                    if (u.x != T(0) || u.y != T(0)) {
                        ++nz;
                        col[r] = c;
                        perm = perm && u.x == T(1) && u.y == T(0);
                    }
                }
                perm = perm && nz == 1;
            }
            if (perm) {
                uint32_t poff[D];
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    uint32_t o = 0;
#pragma unroll
                    for (int j = 0; j < K; ++j) o |= uint32_t((col[r] >> (K - 1 - j)) & 1) << pos[j];
                    poff[r] = swz<T>(o);
                }
                for (uint32_t g = tid; g < groups; g += nthr) {
                    uint32_t base = g;
#pragma unroll
                    for (int j = 0; j < K; ++j)
                        base = ((base >> srt[j]) << (srt[j] + 1)) | (base & ((1u << srt[j]) - 1));
                    const uint32_t sb = swz<T>(base);
                    C p[D], l[D];
#pragma unroll
                    for (int r = 0; r < D; ++r) {
                        p[r] = pt[sb ^ poff[r]];
                        l[r] = lt[sb ^ poff[r]];
                    }
#pragma unroll
                    for (int r = 0; r < D; ++r) {
                        pt[sb ^ soff[r]] = p[r];
                        lt[sb ^ soff[r]] = l[r];
                    }
                }
                return;
            }
        }
    }
    T s[R];
#pragma unroll
    for (int q = 0; q < R; ++q) s[q] = T(0);
    for (uint32_t g = tid; g < groups; g += nthr) {
        uint32_t base = g;
#pragma unroll
        for (int j = 0; j < K; ++j) base = ((base >> srt[j]) << (srt[j] + 1)) | (base & ((1u << srt[j]) - 1));
        const uint32_t sb = swz<T>(base);
        C p[D], l[D];
#pragma unroll
        for (int c = 0; c < D; ++c) {
            p[c] = pt[sb ^ soff[c]];
            l[c] = lt[sb ^ soff[c]];
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (want[q]) {
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    C pc = p[0];  // p[gc[r]] by selects (no dynamic register indexing)
#pragma unroll
                    for (int c = 1; c < D; ++c)
                        if (gc[q][r] == c) pc = p[c];
                    C w = mk<T>(0, 0);
                    cfma(w, gv[q][r], pc);
                    s[q] += l[r].x * w.y - l[r].y * w.x;  // Im(conj(l) w)
                }
            }
            if (diag[q]) {
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    C x = mk<T>(0, 0), y = mk<T>(0, 0);
                    cfma(x, ud[q][r * D + r], p[r]);
                    cfma(y, ud[q][r * D + r], l[r]);
                    p[r] = x;
                    l[r] = y;
                }
            } else {
                C pn[D], ln[D];
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    C x = mk<T>(0, 0), y = mk<T>(0, 0);
#pragma unroll
                    for (int c = 0; c < D; ++c) {
                        cfma(x, ud[q][r * D + c], p[c]);
                        cfma(y, ud[q][r * D + c], l[c]);
                    }
                    pn[r] = x;
                    ln[r] = y;
                }
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    p[r] = pn[r];
                    l[r] = ln[r];
                }
            }
        }
#pragma unroll
        for (int r = 0; r < D; ++r) {
            pt[sb ^ soff[r]] = p[r];
            lt[sb ^ soff[r]] = l[r];
        }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        if (want[q]) {  // uniform over the CTA: every lane reaches the shuffles
            T v = s[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((tid & 31) == 0) wacc_add(red[op0 + q], v);
        }
    }
}

// ---- register runs -------------------------------------------------------
// An op of a run acts on a group of 2^R amplitudes of phi and lam held in
// registers; local bit P of the group <-> tile bit run_pos[P]. Positions are
// runtime values: each (R, positions) case is its own fully unrolled instance,
// chosen by a switch. For each op: the derivative (if wanted) at the op's
// output, Im sum_r conj(l_r) (gval_r p_{gcol_r}), then U^dagger on both --
// dense, diagonal (two products per row) or a permutation with unit entries
// (register moves), as classified when the state's matrices were staged.
constexpr int kAdjDense = 0, kAdjDiag = 1, kAdjPerm = 2, kAdjReal = 3;  // kAdjReal: a dense real matrix (RY)
// permutations of a two-site U^dagger known at compile time (register renaming, no selects):
// rows (0, 1, 2, 3) <- columns (0, 1, 3, 2) [CNOT, control on the first site], (0, 3, 2, 1)
// [CNOT, control on the second site], (0, 2, 1, 3) [SWAP]
constexpr int kAdjPermCX = 4, kAdjPermXC = 5, kAdjPermSwap = 6;
// generator classes of a wanted derivative (host-classified Pauli-product rows): none, diagonal
// (row r reads column r), flipped (one site: row r reads r ^ 1; two sites: 3 - r), any other
constexpr int kGenNone = 0, kGenDiag = 1, kGenFlip = 2, kGenAny = 3;
// one-site generators with real (Z, X) or imaginary (Y) entries need one component of each sum
constexpr int kGenDiagRe = 4, kGenFlipRe = 5, kGenFlipIm = 6;

// A staged one-site op uses 4 of its 16 slots; slots 4 and 5 repeat a real U^dagger's (a, b), (c, d)
// or a diagonal one's entries, so that one 16-byte load fetches them (complex64), slot 6 holds
// the two generator entries' nonzero components.
__device__ __forceinline__ void adj_load2(const float2* u, float2& a, float2& b) {
    const float4 q = *reinterpret_cast<const float4*>(u + 4);
    a = make_float2(q.x, q.y);
    b = make_float2(q.z, q.w);
}
__device__ __forceinline__ void adj_load2(const double2* u, double2& a, double2& b) {
    a = u[4];
    b = u[5];
}

// The derivative Im sum_r conj(l_r) (g_r p_{col r}) of one op over a group: complex sums
// W_r = sum conj(l_r) q_r per generator row r, combined once per op as Im(g_r W_r) =
// g_r.x W_r.y + g_r.y W_r.x (g_r in {+-1, +-i}).
template <typename T, typename C>
__device__ __forceinline__ void wacc(C& w, const C& l, const C& q) {
    w.x = fmaf(l.x, q.x, fmaf(l.y, q.y, w.x));
    w.y = fmaf(l.x, q.y, fmaf(-l.y, q.x, w.y));
}
template <>
__device__ __forceinline__ void wacc<double, double2>(double2& w, const double2& l, const double2& q) {
    w.x = fma(l.x, q.x, fma(l.y, q.y, w.x));
    w.y = fma(l.x, q.y, fma(-l.y, q.x, w.y));
}

// one component of wacc's sum
template <bool IM, typename C, typename T>
__device__ __forceinline__ void wacc1(T& w, const C& l, const C& q) {
    if constexpr (IM) w = fma(l.x, q.y, fma(-l.y, q.x, w));
    else w = fma(l.x, q.x, fma(l.y, q.y, w));
}

template <int R, int P, int MODE, int GEN, typename C, typename T>
__device__ __forceinline__ void adj_reg1(C (&p)[1 << R], C (&l)[1 << R], const C* __restrict__ u,
                                         const float2* gv, T& s) {
    constexpr int D = 1 << R, bit = 1 << P;
    constexpr bool one = GEN == kGenDiagRe || GEN == kGenFlipRe || GEN == kGenFlipIm;
    C u0, u1, u2, u3;
    if constexpr (MODE == kAdjReal) {
        C ab, cd;
        adj_load2(u, ab, cd);
        u0.x = ab.x;
        u1.x = ab.y;
        u2.x = cd.x;
        u3.x = cd.y;
    } else if constexpr (MODE == kAdjDiag) {
        adj_load2(u, u0, u3);
    } else if constexpr (MODE == kAdjDense) {
        u0 = u[0];
        u1 = u[1];
        u2 = u[2];
        u3 = u[3];
    }
    C w0 = mk<T>(T(0), T(0)), w1 = mk<T>(T(0), T(0));
    T v0 = T(0), v1 = T(0);
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if (c & bit) continue;
        const C p0 = p[c], p1 = p[c | bit], l0 = l[c], l1 = l[c | bit];
        if constexpr (GEN == kGenDiag) {
            wacc<T>(w0, l0, p0);
            wacc<T>(w1, l1, p1);
        } else if constexpr (GEN == kGenDiagRe) {
            wacc1<true>(v0, l0, p0);
            wacc1<true>(v1, l1, p1);
        } else if constexpr (GEN == kGenFlipRe || GEN == kGenFlipIm) {
            wacc1<GEN == kGenFlipRe>(v0, l0, p1);
            wacc1<GEN == kGenFlipRe>(v1, l1, p0);
        } else if constexpr (GEN != kGenNone) {  // one site: off-diagonal rows (X, Y)
            wacc<T>(w0, l0, p1);
            wacc<T>(w1, l1, p0);
        }
        if constexpr (MODE == kAdjReal) {
            const T a = u0.x, b = u1.x, cc = u2.x, d = u3.x;
            p[c] = mk<T>(a * p0.x + b * p1.x, a * p0.y + b * p1.y);
            p[c | bit] = mk<T>(cc * p0.x + d * p1.x, cc * p0.y + d * p1.y);
            l[c] = mk<T>(a * l0.x + b * l1.x, a * l0.y + b * l1.y);
            l[c | bit] = mk<T>(cc * l0.x + d * l1.x, cc * l0.y + d * l1.y);
        } else if constexpr (MODE == kAdjDiag) {
            C x = mk<T>(0, 0), y = mk<T>(0, 0), z = mk<T>(0, 0), t = mk<T>(0, 0);
            cfma(x, u0, p0);
            cfma(y, u3, p1);
            cfma(z, u0, l0);
            cfma(t, u3, l1);
            p[c] = x;
            p[c | bit] = y;
            l[c] = z;
            l[c | bit] = t;
        } else if constexpr (MODE == kAdjPerm) {  // one site: a unit permutation that is not the identity swaps
            p[c] = p1;
            p[c | bit] = p0;
            l[c] = l1;
            l[c | bit] = l0;
        } else {
            C x = mk<T>(0, 0), y = mk<T>(0, 0), z = mk<T>(0, 0), t = mk<T>(0, 0);
            cfma(x, u0, p0);
            cfma(x, u1, p1);
            cfma(y, u2, p0);
            cfma(y, u3, p1);
            cfma(z, u0, l0);
            cfma(z, u1, l1);
            cfma(t, u2, l0);
            cfma(t, u3, l1);
            p[c] = x;
            p[c | bit] = y;
            l[c] = z;
            l[c | bit] = t;
        }
    }
    if constexpr (one) {
        const C g = u[6];
        s = fma(g.y, v1, g.x * v0);
    } else if constexpr (GEN != kGenNone)
        s += T(gv[0].x) * w0.y + T(gv[0].y) * w0.x + T(gv[1].x) * w1.y + T(gv[1].y) * w1.x;
}

// matrix bit 1 (most significant) <-> local bit P0 (the op's first site), bit 0 <-> P1
template <int R, int P0, int P1, int MODE, int GEN, typename C, typename T>
__device__ __forceinline__ void adj_reg2(C (&p)[1 << R], C (&l)[1 << R], const C* __restrict__ u,
                                         const uint8_t* __restrict__ col, const float2* gv, const int* gc, T& s) {
    constexpr int D = 1 << R, b0 = 1 << P0, b1 = 1 << P1;
    int gcr[4], colr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        gcr[r] = GEN == kGenAny ? gc[r] : 0;
        colr[r] = MODE == kAdjPerm ? col[r] : 0;
    }
    C w[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) w[r] = mk<T>(T(0), T(0));
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if ((c & b0) || (c & b1)) continue;
        const int ix[4] = {c, c | b1, c | b0, c | b0 | b1};
        C x[4], y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            x[r] = p[ix[r]];
            y[r] = l[ix[r]];
        }
        if constexpr (GEN == kGenDiag) {
#pragma unroll
            for (int r = 0; r < 4; ++r) wacc<T>(w[r], y[r], x[r]);
        } else if constexpr (GEN == kGenFlip) {
#pragma unroll
            for (int r = 0; r < 4; ++r) wacc<T>(w[r], y[r], x[3 - r]);
        } else if constexpr (GEN == kGenAny) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                C q = x[0];  // x[gc[r]] by selects (no dynamic register indexing)
#pragma unroll
                for (int e = 1; e < 4; ++e)
                    if (gcr[r] == e) q = x[e];
                wacc<T>(w[r], y[r], q);
            }
        }
        if constexpr (MODE == kAdjDiag) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const C d = u[5 * r];
                C a = mk<T>(0, 0), b = mk<T>(0, 0);
                cfma(a, d, x[r]);
                cfma(b, d, y[r]);
                p[ix[r]] = a;
                l[ix[r]] = b;
            }
        } else if constexpr (MODE == kAdjPermCX || MODE == kAdjPermXC || MODE == kAdjPermSwap) {
            constexpr int s1 = MODE == kAdjPermCX ? 1 : (MODE == kAdjPermXC ? 3 : 2);
            constexpr int s2 = MODE == kAdjPermCX ? 3 : (MODE == kAdjPermXC ? 2 : 1);
            constexpr int s3 = MODE == kAdjPermCX ? 2 : (MODE == kAdjPermXC ? 1 : 3);
            p[ix[1]] = x[s1];
            p[ix[2]] = x[s2];
            p[ix[3]] = x[s3];
            l[ix[1]] = y[s1];
            l[ix[2]] = y[s2];
            l[ix[3]] = y[s3];
        } else if constexpr (MODE == kAdjPerm) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                C a = x[0], b = y[0];
#pragma unroll
                for (int e = 1; e < 4; ++e)
                    if (colr[r] == e) {
                        a = x[e];
                        b = y[e];
                    }
                p[ix[r]] = a;
                l[ix[r]] = b;
            }
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                C a = mk<T>(0, 0), b = mk<T>(0, 0);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const C m = u[4 * r + e];
                    cfma(a, m, x[e]);
                    cfma(b, m, y[e]);
                }
                p[ix[r]] = a;
                l[ix[r]] = b;
            }
        }
    }
    if constexpr (GEN != kGenNone) {
#pragma unroll
        for (int r = 0; r < 4; ++r) s += T(gv[r].x) * w[r].y + T(gv[r].y) * w[r].x;
    }
}

template <int R, int P0, int P1, int GEN, typename C, typename T>
__device__ __forceinline__ void adj_reg2_mode(C (&p)[1 << R], C (&l)[1 << R], const C* u, int mode,
                                              const uint8_t* col, const float2* gv, const int* gc, T& s) {
    switch (mode) {
        case kAdjDiag: adj_reg2<R, P0, P1, kAdjDiag, GEN>(p, l, u, col, gv, gc, s); break;
        case kAdjPermCX: adj_reg2<R, P0, P1, kAdjPermCX, GEN>(p, l, u, col, gv, gc, s); break;
        case kAdjPermXC: adj_reg2<R, P0, P1, kAdjPermXC, GEN>(p, l, u, col, gv, gc, s); break;
        case kAdjPermSwap: adj_reg2<R, P0, P1, kAdjPermSwap, GEN>(p, l, u, col, gv, gc, s); break;
        case kAdjPerm: adj_reg2<R, P0, P1, kAdjPerm, GEN>(p, l, u, col, gv, gc, s); break;
        default: adj_reg2<R, P0, P1, kAdjDense, GEN>(p, l, u, col, gv, gc, s); break;
    }
}

template <int R, int P0, int P1, typename C, typename T>
__device__ __forceinline__ void adj_reg2_any(C (&p)[1 << R], C (&l)[1 << R], const C* u, int mode, int gen,
                                             const uint8_t* col, const float2* gv, const int* gc, T& s) {
    switch (gen) {
        case kGenNone: adj_reg2_mode<R, P0, P1, kGenNone>(p, l, u, mode, col, gv, gc, s); break;
        case kGenDiag: adj_reg2_mode<R, P0, P1, kGenDiag>(p, l, u, mode, col, gv, gc, s); break;
        case kGenFlip: adj_reg2_mode<R, P0, P1, kGenFlip>(p, l, u, mode, col, gv, gc, s); break;
        default: adj_reg2_mode<R, P0, P1, kGenAny>(p, l, u, mode, col, gv, gc, s); break;
    }
}

template <int R, int CODE, typename C, typename T>
__device__ __forceinline__ void adj_apply2_case(C (&p)[1 << R], C (&l)[1 << R], const C* u, int mode, int gen,
                                                const uint8_t* col, const float2* gv, const int* gc, T& s) {
    constexpr int P0 = CODE / 4, P1 = CODE % 4;
    if constexpr (P0 < R && P1 < R && P0 != P1) adj_reg2_any<R, P0, P1>(p, l, u, mode, gen, col, gv, gc, s);
}

template <int R, typename C, typename T>
__device__ __forceinline__ void adj_apply2(C (&p)[1 << R], C (&l)[1 << R], int P0, int P1, const C* u, int mode,
                                           int gen, const uint8_t* col, const float2* gv, const int* gc, T& s) {
    switch (P0 * 4 + P1) {
        case 1: adj_apply2_case<R, 1>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 2: adj_apply2_case<R, 2>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 3: adj_apply2_case<R, 3>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 4: adj_apply2_case<R, 4>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 6: adj_apply2_case<R, 6>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 7: adj_apply2_case<R, 7>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 8: adj_apply2_case<R, 8>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 9: adj_apply2_case<R, 9>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 11: adj_apply2_case<R, 11>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 12: adj_apply2_case<R, 12>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 13: adj_apply2_case<R, 13>(p, l, u, mode, gen, col, gv, gc, s); break;
        case 14: adj_apply2_case<R, 14>(p, l, u, mode, gen, col, gv, gc, s); break;
    }
}

// Every op of a run is one case of one switch (its own unrolled code): a one-site op by its local bit,
// U^dagger class and generator class, two consecutive one-site ops Z-like then Y-like on the same bit (the
// RZ, RY pair of a reversed ansatz) as one, any two-site op through adj_apply2.
constexpr int kCodeTwo = 0, kCodePair = 1, kCodeOne = 4;  // kCodePair + P; kCodeOne + (P * 4 + mode) * 6 + gen
__device__ __forceinline__ int adj_gen_index(int gen) {  // kGenNone, DiagRe, FlipRe, FlipIm, Diag, Flip -> 0..5
    return gen == kGenNone ? 0 : gen == kGenDiagRe ? 1 : gen == kGenFlipRe ? 2 : gen == kGenFlipIm ? 3
           : gen == kGenDiag ? 4 : 5;
}

// The derivative sums of a tile's ops, reduced over a warp 32 ops at a time. Op t's 32 per-thread sums are
// added by the xor tree 16, 8, 4, 2, 1, the additions of different ops sharing the lanes: two ops waiting at a
// level are merged by one shuffle (the upper lanes go on with the later op), so an op costs one shuffle
// instead of five and a level's latency is paid once for all. The sums of an op are added in the same
// tree as one op at a time.
__device__ __forceinline__ int adj_gen1(const AdjSweepArgs& a, int op) {  // a one-site op's generator class
    const int cls = a.op_gcls[op];
    if (cls == kGenNone) return kGenNone;
    const float2 g0 = a.gval[op][0], g1 = a.gval[op][1];
    const bool re = g0.y == 0.f && g1.y == 0.f, im = g0.x == 0.f && g1.x == 0.f;
    if (cls == kGenDiag) return re ? kGenDiagRe : kGenDiag;
    return re ? kGenFlipRe : (im ? kGenFlipIm : kGenFlip);
}

template <typename T>
__device__ __forceinline__ T adj_merge(T a, T b, int o, int lane) {  // a: the earlier op
    const bool up = lane & o;
    const T keep = up ? b : a, send = up ? a : b;
    return keep + __shfl_xor_sync(0xffffffffu, send, o);
}

template <typename T>
struct AdjTree {
    T s[5];
    int t;
    __device__ __forceinline__ void add_to(typename WAccOf<T>::type* red, const uint8_t* dlist, int nd, T x, int lane) {
        const int at = (t & ~31) + int(__brev(uint32_t(lane)) >> 27);
        if (at < nd) wacc_add(red[dlist[at]], x);
    }
    // the next derivative op's per-thread sum; red: this warp's accumulators, dlist: op of each derivative
    __device__ __forceinline__ void push(T x, typename WAccOf<T>::type* red, const uint8_t* dlist, int nd, int lane) {
        const int t0 = t;
        bool out = true;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            if (out) {
                if ((t0 >> k) & 1) {
                    x = adj_merge(s[k], x, 16 >> k, lane);
                } else {
                    s[k] = x;
                    out = false;
                }
            }
        }
        if (out) add_to(red, dlist, nd, x, lane);
        t = t0 + 1;
    }
    // two in a row
    __device__ __forceinline__ void push2(T x, T y, typename WAccOf<T>::type* red, const uint8_t* dlist, int nd,
                                          int lane) {
        if (t & 1) {
            push(x, red, dlist, nd, lane);
            push(y, red, dlist, nd, lane);
            return;
        }
        x = adj_merge(x, y, 16, lane);
        const int t0 = t >> 1;
        t += 2;
        if (!(t0 & 1)) {
            s[1] = x;
            return;
        }
        x = adj_merge(s[1], x, 8, lane);
        if (!(t0 & 2)) {
            s[2] = x;
            return;
        }
        x = adj_merge(s[2], x, 4, lane);
        if (!(t0 & 4)) {
            s[3] = x;
            return;
        }
        x = adj_merge(s[3], x, 2, lane);
        if (!(t0 & 8)) {
            s[4] = x;
            return;
        }
        x = adj_merge(s[4], x, 1, lane);
        t -= 1;  // add_to names the block of the last op
        add_to(red, dlist, nd, x, lane);
        t += 1;
    }
    // the ops still waiting at the end of a tile
    __device__ __forceinline__ void finish(typename WAccOf<T>::type* red, const uint8_t* dlist, int nd, int lane) {
        if (t & 31) {
            T x = T(0);
            bool have = false;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                if ((t >> k) & 1) {
                    x = adj_merge(s[k], have ? x : T(0), 16 >> k, lane);
                    have = true;
                } else if (have) {
                    x = adj_merge(x, T(0), 16 >> k, lane);
                }
            }
            add_to(red, dlist, nd, x, lane);
        }
        t = 0;
    }
};

// A run as the kernel executes it. Permutations without derivative at a run's start or end (the CNOT ladder of
// an ansatz) move no data: the pass keeps the linear map from a tile's logical index to the place of
// its amplitude in shared memory, and such an op only changes the map. A run's thread then addresses its group
// through the images of the index bits: off[P] of the run's bits, base[j] of the j-th other bit, all XORed.
constexpr int kAdjMaxTile = QGB_SWEEP_MAX_TILE_BITS;
struct AdjRun {
    uint32_t off[3];  // byte offsets
    uint16_t base[kAdjMaxTile - 3];
    uint16_t flip;   // image of 0 (X gates)
    uint8_t first, count;  // its ops
};
struct AdjMap {  // of the whole tile, after the pass's last op
    uint16_t bit[kAdjMaxTile];
    uint16_t flip;
    uint16_t nruns;
};

// Builds the runs and the final map from the ops' classes; called by one whole warp.
template <typename T>
__device__ void adj_build_runs(AdjRun* runs, AdjMap* map, const AdjSweepArgs& a, const uint8_t* umode, uint8_t* prog,
                               const uint8_t* ucode, int lane) {
    const int m = a.m;
    uint32_t col = lane < m ? swz<T>(1u << lane) : 0u, flip = 0u;  // lane j: the image of index bit j
    // each lane describes two ops (the loops below then wait for shuffles, not for tables): how the map
    // moves (0: not at all, 1: X, 2, 3: CNOT either way, 4: SWAP), the sites, and at a run's first op its length
    uint32_t info[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int op = lane + 32 * h;
        info[h] = 0;
        if (op < a.n_ops) {
            const int mode = umode[op], p0 = a.op_pos[op][0], two = a.op_k[op] == 2;
            uint32_t kind = 0;
            if (a.op_gcls[op] == kGenNone) {
                if (!two) kind = mode == kAdjPerm ? 1 : 0;
                else kind = mode == kAdjPermCX ? 2 : mode == kAdjPermXC ? 3 : mode == kAdjPermSwap ? 4 : 0;
            }
            info[h] = kind | uint32_t(p0) << 4 | uint32_t(two ? a.op_pos[op][1] : p0) << 8 | uint32_t(a.run_len[op]) << 12;
        }
    }
    auto info_of = [&](int op) { return __shfl_sync(0xffffffffu, op < 32 ? info[0] : info[1], op & 31); };
    auto move = [&](uint32_t f) {  // new[x] = old[pi(x)]: the image of x becomes that of pi(x)
        const int kind = f & 15, p0 = (f >> 4) & 15, p1 = (f >> 8) & 15;
        const uint32_t c0 = __shfl_sync(0xffffffffu, col, p0), c1 = __shfl_sync(0xffffffffu, col, p1);
        if (kind == 1) flip ^= c0;
        else if (kind == 2) col ^= lane == p0 ? c1 : 0u;
        else if (kind == 3) col ^= lane == p1 ? c0 : 0u;
        else col = lane == p0 ? c1 : (lane == p1 ? c0 : col);
    };
    int nruns = 0;
    for (int i0 = 0; i0 < a.n_ops;) {
        const int end = i0 + int(info_of(i0) >> 12);
        int b = i0, e = end;
        for (; b < end; ++b) {
            const uint32_t f = info_of(b);
            if (!(f & 15)) break;
            move(f);
        }
        while (e > b && (info_of(e - 1) & 15)) --e;
        if (b < e) {
            AdjRun& r = runs[nruns];
            const int r0 = a.run_pos[i0][0], r1 = a.run_pos[i0][1], r2 = a.run_pos[i0][2];
            const uint32_t own = 1u << r0 | 1u << r1 | 1u << r2;
            if (lane == r0) r.off[0] = col * uint32_t(sizeof(cplx<T>));
            if (lane == r1) r.off[1] = col * uint32_t(sizeof(cplx<T>));
            if (lane == r2) r.off[2] = col * uint32_t(sizeof(cplx<T>));
            if (lane < m && !((own >> lane) & 1u)) r.base[__popc(~own & ((1u << lane) - 1u))] = uint16_t(col);
            if (lane == 0) {
                r.flip = uint16_t(flip);
                r.first = uint8_t(b);
                r.count = uint8_t(e - b);
                // only pairs, on bits 0, 1, .. in order: a program of its own (1 to 3 pairs)
                int np = (e - b) % 2 == 0 && e - b <= 6 ? (e - b) / 2 : 0;
                for (int j = 0; j < np; ++j)
                    if (ucode[b + 2 * j] != kCodePair + j) np = 0;
                prog[nruns] = uint8_t(np);
            }
            ++nruns;
        }
        for (; e < end; ++e) move(info_of(e));
        i0 = end;
    }
    if (lane < m) map->bit[lane] = uint16_t(col);
    if (lane == 0) {
        map->flip = uint16_t(flip);
        map->nruns = uint16_t(nruns);
    }
}

// The pair Z-like then Y-like on bit P, straight-line.
template <int P, typename C, typename T>
__device__ __forceinline__ void adj_pair(C (&p)[8], C (&l)[8], const C* __restrict__ u, T& s0, T& s1) {
    adj_reg1<3, P, kAdjDiag, kGenDiagRe>(p, l, u, nullptr, s0);
    adj_reg1<3, P, kAdjReal, kGenFlipIm>(p, l, u + 16, nullptr, s1);
}

// Any run, an op at a time. one: a single group per thread (its sums join the tree).
template <typename T>
__device__ __forceinline__ void adj_run_ops(cplx<T> (&p)[8], cplx<T> (&l)[8], int first, int count, bool one,
                                            const AdjSweepArgs& a, const cplx<T>* __restrict__ ush,
                                            const uint8_t* __restrict__ ucode, const uint8_t* __restrict__ umode,
                                            const uint8_t* __restrict__ ucol, AdjTree<T>& tree,
                                            const uint8_t* __restrict__ dlist, int nd,
                                            typename WAccOf<T>::type* __restrict__ red, int lane) {
    using C = cplx<T>;
    constexpr int R = 3;
    for (int q = 0; q < count; ++q) {
        const int op = first + q;
        const C* u = ush + op * 16;
        T sd = T(0), sd2 = T(0);
        const int code = ucode[op];
        switch (code) {
#define QGB_ADJ_G(P, M, B)                                                                                  \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 0: adj_reg1<R, P, M, kGenNone>(p, l, u, a.gval[op], sd); break;   \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 1: adj_reg1<R, P, M, kGenDiagRe>(p, l, u, a.gval[op], sd); break; \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 2: adj_reg1<R, P, M, kGenFlipRe>(p, l, u, a.gval[op], sd); break; \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 3: adj_reg1<R, P, M, kGenFlipIm>(p, l, u, a.gval[op], sd); break; \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 4: adj_reg1<R, P, M, kGenDiag>(p, l, u, a.gval[op], sd); break;   \
    case kCodeOne + ((P) * 4 + (B)) * 6 + 5: adj_reg1<R, P, M, kGenFlip>(p, l, u, a.gval[op], sd); break;
#define QGB_ADJ_P(P)                                                        \
    case kCodePair + (P): adj_pair<P>(p, l, u, sd, sd2); break;             \
        QGB_ADJ_G(P, kAdjDense, 0) QGB_ADJ_G(P, kAdjDiag, 1) QGB_ADJ_G(P, kAdjPerm, 2) QGB_ADJ_G(P, kAdjReal, 3)
            QGB_ADJ_P(0)
            QGB_ADJ_P(1)
            QGB_ADJ_P(2)
#undef QGB_ADJ_P
#undef QGB_ADJ_G
            default:
                adj_apply2<R>(p, l, a.op_lpos[op][0], a.op_lpos[op][1], u, umode[op], a.op_gcls[op], ucol + op * 4,
                              a.gval[op], a.gcol[op], sd);
                break;
        }
        const bool pair = code >= kCodePair && code < kCodeOne;
        if (a.op_gcls[op] != kGenNone) {  // uniform over the CTA: every lane reaches the shuffles
            if (one) {
                if (pair) tree.push2(sd, sd2, red, dlist, nd, lane);
                else tree.push(sd, red, dlist, nd, lane);
            } else {  // several groups per thread: each is added by itself
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    sd += __shfl_xor_sync(0xffffffffu, sd, o);
                    sd2 += __shfl_xor_sync(0xffffffffu, sd2, o);
                }
                if (lane == 0) {
                    wacc_add(red[op], sd);
                    if (pair) wacc_add(red[op + 1], sd2);
                }
            }
        }
        q += pair;
    }
}

// Every run of the pass on one staged pair of tiles: groups of 8 amplitudes,
// one group per thread at a time, a barrier after each run. ucode / umode / ucol:
// each op's case, U^dagger class and, for a permutation, its source column per row.
template <typename T>
__device__ __forceinline__ void adj_tile_runs(uint32_t tile, int m, const AdjSweepArgs& a,
                                              const cplx<T>* __restrict__ ush, const AdjRun* __restrict__ runs,
                                              int nruns, const uint16_t* __restrict__ sbase,
                                              const uint8_t* __restrict__ prog, const uint8_t* __restrict__ ucode,
                                              const uint8_t* __restrict__ umode, const uint8_t* __restrict__ ucol,
                                              const uint8_t* __restrict__ dlist, int nd,
                                              typename WAccOf<T>::type* __restrict__ red, int tid, int nthr) {
    using C = cplx<T>;
    constexpr int D = 8;
    const int lane = tid & 31;
    const uint32_t groups = 1u << (m - 3);
    const bool one = groups <= uint32_t(nthr);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t lam = uint32_t(sizeof(C)) << m;  // the co-state's tile follows the state's
    AdjTree<T> tree;
    tree.t = 0;
    for (int i = 0; i < nruns; ++i) {
        const AdjRun& run = runs[i];
        uint32_t soff[D];
        soff[0] = 0;
        soff[1] = run.off[0];
        soff[2] = run.off[1];
        soff[4] = run.off[2];
        soff[3] = soff[1] ^ soff[2];
        soff[5] = soff[1] ^ soff[4];
        soff[6] = soff[2] ^ soff[4];
        soff[7] = soff[3] ^ soff[4];
        for (uint32_t gb = 0; gb < groups; gb += uint32_t(nthr)) {  // every thread the same trip count
            const uint32_t g = gb + uint32_t(tid);
            const bool ok = g < groups;
            uint32_t sb = sbase[i * nthr + tid];
            if (!one)  // the bits above the thread's
                for (int j = 31 - __clz(nthr); j < m - 3; ++j) sb ^= (g >> j) & 1u ? uint32_t(run.base[j]) : 0u;
            sb *= uint32_t(sizeof(C));
            C p[D], l[D];
#pragma unroll
            for (int c = 0; c < D; ++c) {
                const unsigned char* at = smem_raw + (tile + (sb ^ soff[c]));
                p[c] = ok ? *reinterpret_cast<const C*>(at) : mk<T>(T(0), T(0));
                l[c] = ok ? *reinterpret_cast<const C*>(at + lam) : mk<T>(T(0), T(0));
            }
            const int np = one ? prog[i] : 0;
            if (np > 0) {
                const C* u = ush + int(run.first) * 16;
                T s0, s1;
                adj_pair<0>(p, l, u, s0, s1);
                tree.push2(s0, s1, red, dlist, nd, lane);
                if (np > 1) {
                    adj_pair<1>(p, l, u + 32, s0, s1);
                    tree.push2(s0, s1, red, dlist, nd, lane);
                    if (np > 2) {
                        adj_pair<2>(p, l, u + 64, s0, s1);
                        tree.push2(s0, s1, red, dlist, nd, lane);
                    }
                }
            } else {
                adj_run_ops<T>(p, l, run.first, run.count, one, a, ush, ucode, umode, ucol, tree, dlist, nd, red, lane);
            }
            if (ok) {
#pragma unroll
                for (int c = 0; c < D; ++c) {
                    unsigned char* at = smem_raw + (tile + (sb ^ soff[c]));
                    *reinterpret_cast<C*>(at) = p[c];
                    *reinterpret_cast<C*>(at + lam) = l[c];
                }
            }
        }
        __syncthreads();
    }
    tree.finish(red, dlist, nd, lane);
}

// Length of the run of ops starting at op0 on the same sites (same k and tile bits, in order).
__device__ __forceinline__ int adj_run_length(const AdjSweepArgs& a, int op0) {
    int r = 1;
    while (op0 + r < a.n_ops && r < kAdjMaxRun && a.op_k[op0 + r] == a.op_k[op0] &&
           a.op_pos[op0 + r][0] == a.op_pos[op0][0] && (a.op_k[op0] == 1 || a.op_pos[op0 + r][1] == a.op_pos[op0][1]))
        ++r;
    return r;
}

template <typename T, int K>
__device__ __forceinline__ int adj_tile_ops(cplx<T>* pt, cplx<T>* lt, int m, const AdjSweepArgs& a, int op0,
                                            const cplx<T>* ush, typename WAccOf<T>::type* red, int tid, int nthr) {
    // longest run kept in registers without spilling under the 512-thread register cap
    constexpr int kMax = sizeof(T) == 4 ? (K == 1 ? 4 : 2) : (K == 1 ? 2 : 1);
    int r = adj_run_length(a, op0);
    if (r > kMax) r = kMax;
    if (r == 1) adj_tile_run<T, K, 1>(pt, lt, m, a, op0, ush, red, tid, nthr);
    else if (r == 2) { if constexpr (kMax >= 2) adj_tile_run<T, K, 2>(pt, lt, m, a, op0, ush, red, tid, nthr); }
    else if (r == 3) { if constexpr (kMax >= 3) adj_tile_run<T, K, 3>(pt, lt, m, a, op0, ush, red, tid, nthr); }
    else { if constexpr (kMax >= 4) adj_tile_run<T, K, 4>(pt, lt, m, a, op0, ush, red, tid, nthr); }
    return r;
}

// bytes of the kernel's shared memory before the runs, and in all
template <typename T>
__host__ __device__ inline size_t adj_runs_offset(int m, int H, int n_ops, int nbuf) {
    const size_t o = sizeof(cplx<T>) * ((size_t(2 * nbuf) << m) + size_t(n_ops) * 16) + sizeof(uint64_t) * (size_t(1) << H) +
                     sizeof(double) * size_t(n_ops) * kAdjMaxWarps + size_t(n_ops) * 8;
    return (o + 15) & ~size_t(15);
}
template <typename T>
__host__ __device__ inline size_t adj_smem_bytes(int m, int H, int n_ops, int n_runs, int threads, int nbuf) {
    return adj_runs_offset<T>(m, H, n_ops, nbuf) + (sizeof(AdjRun) + sizeof(uint16_t) * threads) * size_t(n_runs) +
           sizeof(AdjMap);
}

// complex64: 256 threads and 2 CTAs per SM (128 registers): the straight-line programs spill at the 80
// registers of a third CTA (64 sets of 20 qubits, 28 passes: 38.2 ms with three, 34.8 ms with two, 74.5 ms
// before the map and the programs); complex128 keeps 128 registers (up to 512 threads when one CTA fits).
// Bound by instruction issue: two thirds of it the two-by-two products and derivative sums, the rest
// addresses, reductions and the copies; HBM is at a quarter.
template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 256 : kAdjMaxThreads, sizeof(T) == 4 ? 2 : 1) adjoint_sweep_kernel(cplx<T>* __restrict__ phi,
                                                                       cplx<T>* __restrict__ lam,
                                                                       const cplx<T>* __restrict__ mats,
                                                                       const __grid_constant__ AdjSweepArgs a,
                                                                       double* __restrict__ partials, int nbuf) {
    using C = cplx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = a.L, H = a.H, m = a.m;
    const int nwarps = blockDim.x >> 5;
    // layout: nbuf x (phi tile, lam tile) | ush (n_ops x 16 complex: U^dagger of the current state) |
    //         hoff (2^H uint64) | red (kAdjMaxWarps x n_ops accumulators, 8 bytes) | umode, ucode, dlist (n_ops each) | ucol (n_ops x 4) |
    //         prog (n_ops) | runs (n_runs) | map | sbase (n_runs x threads)
    C* bufs = reinterpret_cast<C*>(smem_raw);
    C* ush = bufs + (size_t(2 * nbuf) << m);
    uint64_t* hoff = reinterpret_cast<uint64_t*>(ush + size_t(a.n_ops) * 16);
    auto* red = reinterpret_cast<typename WAccOf<T>::type*>(hoff + (size_t(1) << H));
    uint8_t* umode = reinterpret_cast<uint8_t*>(red + size_t(a.n_ops) * kAdjMaxWarps);
    uint8_t* ucode = umode + a.n_ops;
    uint8_t* dlist = ucode + a.n_ops;
    uint8_t* ucol = dlist + a.n_ops;
    uint8_t* prog = ucol + 4 * a.n_ops;
    AdjRun* runs = reinterpret_cast<AdjRun*>(smem_raw + adj_runs_offset<T>(m, H, a.n_ops, nbuf));
    AdjMap* map = reinterpret_cast<AdjMap*>(runs + a.n_runs);
    uint16_t* sbase = reinterpret_cast<uint16_t*>(map + 1);  // [run][thread]: the thread's group, images XORed
    uint32_t out0 = 0;                                       // image of this thread's first amplitude at the end
    auto* myred = red + size_t(threadIdx.x >> 5) * a.n_ops;  // this warp's accumulators
    int nd = 0;                                              // derivatives, in order
    for (int i = 0; i < a.n_ops; ++i)
        if (a.op_gcls[i] != kGenNone) {
            if (threadIdx.x == 0) dlist[nd] = uint8_t(i);
            ++nd;
        }
    int64_t staged = -1;  // state whose matrices sit in ush
    for (uint32_t h = threadIdx.x; h < (1u << H); h += blockDim.x) {
        uint64_t o = 0;
        for (int j = 0; j < H; ++j) o |= uint64_t((h >> j) & 1u) << a.high_bits[j];
        hoff[h] = o;
    }
    for (int i = threadIdx.x; i < a.n_ops * kAdjMaxWarps; i += blockDim.x) wacc_zero(red[i]);
    __syncthreads();
    const uint32_t lmask = (1u << L) - 1;
    constexpr uint32_t per16 = 16 / sizeof(C);
    // this CTA's tiles: chunks blockIdx.x, blockIdx.x + gridDim.x, ..., each chunk_tiles consecutive tiles
    const uint64_t my_chunks = a.chunks > blockIdx.x ? (a.chunks - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const uint64_t my_tiles = my_chunks * a.chunk_tiles;
    auto tile_of = [&](uint64_t i) -> uint64_t {
        return ((uint64_t(blockIdx.x) + (i >> a.chunk_shift) * gridDim.x) << a.chunk_shift) + (i & (a.chunk_tiles - 1));
    };
    auto base_of = [&](uint64_t w) -> uint64_t {
        // the tile's bits at the outer positions, a bit per lane (called by whole warps)
        const uint64_t b = w >> a.tile_shift, o = w & (a.tiles - 1);
        uint32_t lo = 0, hi = 0;
        for (int j = threadIdx.x & 31; j < a.n_outer; j += 32)
            if ((o >> j) & 1ull) {
                const int ob = a.outer_bits[j];
                if (ob < 32) lo |= 1u << ob;
                else hi |= 1u << (ob - 32);
            }
        lo = __reduce_or_sync(0xffffffffu, lo);
        if (a.n > 32) hi = __reduce_or_sync(0xffffffffu, hi);
        return b * uint64_t(a.sv_stride) + ((uint64_t(hi) << 32) | lo);
    };
    auto load_async = [&](uint64_t w, C* dp, C* dl) {
        const uint64_t base = base_of(w);
        for (uint32_t e = per16 * threadIdx.x; e < (1u << m); e += per16 * blockDim.x) {
            const uint64_t src = base + (hoff[e >> L] | (e & lmask));
            cp_async16_adj(dp + swz<T>(e), phi + src);
            cp_async16_adj(dl + swz<T>(e), lam + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (my_tiles > 0) load_async(tile_of(0), bufs, bufs + (size_t(1) << m));
    for (uint64_t i = 0; i < my_tiles; ++i) {
        const uint64_t w = tile_of(i);
        const int slot = nbuf == 2 ? int(i & 1) : 0;
        C* pt = bufs + (size_t(2 * slot) << m);
        C* lt = pt + (size_t(1) << m);
        if (nbuf == 2 && i + 1 < my_tiles) {
            C* np_ = bufs + (size_t(2 * (slot ^ 1)) << m);
            load_async(tile_of(i + 1), np_, np_ + (size_t(1) << m));
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        const int64_t b = int64_t(w >> a.tile_shift);
        if (b != staged) {  // once per chunk: every op's U^dagger for this state (previous readers done: loop-end barrier)
            const C* mb = mats + b * a.mat_stride;
            for (int e = threadIdx.x; e < a.n_ops * 16; e += blockDim.x) {
                const int op = e >> 4, rc = e & 15, d = 1 << a.op_k[op];
                if (rc < d * d) {
                    const int r = rc / d, c = rc - r * d;
                    const C u = mb[a.op_mat[op] + c * d + r];
                    ush[e] = mk<T>(u.x, -u.y);
                }
            }
            if (a.rbits > 0) {
                __syncthreads();
                // classify each op's U^dagger: diagonal, a permutation with unit entries, or dense
                for (int op = threadIdx.x; op < a.n_ops; op += blockDim.x) {
                    const int d = 1 << a.op_k[op];
                    const C* u = ush + op * 16;
                    bool diag = true, perm = true, real = true;
                    for (int r = 0; r < d; ++r) {
                        int nz = 0, cc = 0;
                        for (int c = 0; c < d; ++c) {
                            const C v = u[r * d + c];
                            const bool z = v.x == T(0) && v.y == T(0);
                            if (v.y != T(0)) real = false;
                            if (r != c && !z) diag = false;
                            if (!z) {
                                ++nz;
                                cc = c;
                                perm = perm && v.x == T(1) && v.y == T(0);
                            }
                        }
                        perm = perm && nz == 1;
                        ucol[op * 4 + r] = uint8_t(cc);
                    }
                    int mode = diag ? kAdjDiag : (perm ? kAdjPerm : ((real && d == 2) ? kAdjReal : kAdjDense));
                    if (mode == kAdjPerm && d == 4) {
                        const uint8_t* c4 = ucol + op * 4;
                        if (c4[0] == 0 && c4[1] == 1 && c4[2] == 3 && c4[3] == 2) mode = kAdjPermCX;
                        else if (c4[0] == 0 && c4[1] == 3 && c4[2] == 2 && c4[3] == 1) mode = kAdjPermXC;
                        else if (c4[0] == 0 && c4[1] == 2 && c4[2] == 1 && c4[3] == 3) mode = kAdjPermSwap;
                    }
                    umode[op] = uint8_t(mode);
                    int code = kCodeTwo;
                    if (d == 2) {
                        C* w = ush + op * 16;
                        const int gen = adj_gen1(a, op);
                        if (mode == kAdjReal) {
                            w[4] = mk<T>(u[0].x, u[1].x);
                            w[5] = mk<T>(u[2].x, u[3].x);
                        } else {
                            w[4] = u[0];
                            w[5] = u[3];
                        }
                        const bool im = gen == kGenFlipIm;
                        w[6] = mk<T>(T(im ? a.gval[op][0].y : a.gval[op][0].x), T(im ? a.gval[op][1].y : a.gval[op][1].x));
                        code = kCodeOne + (a.op_lpos[op][0] * 4 + mode) * 6 + adj_gen_index(gen);
                    }
                    ucode[op] = uint8_t(code);
                }
                __syncthreads();
                // the Z-like, Y-like pairs: both ops of a pair in one run (each op looks at its successor only)
                for (int op = threadIdx.x; op + 1 < a.n_ops; op += blockDim.x) {
                    const int P = a.op_lpos[op][0];
                    const int first = kCodeOne + (P * 4 + kAdjDiag) * 6 + 1, second = kCodeOne + (P * 4 + kAdjReal) * 6 + 3;
                    if (a.run_len[op + 1] == 0 && ucode[op] == first && ucode[op + 1] == second)
                        ucode[op] = uint8_t(kCodePair + P);
                }
                __syncthreads();
                if (threadIdx.x < 32) adj_build_runs<T>(runs, map, a, umode, prog, ucode, threadIdx.x);
                __syncthreads();
                const int tb = min(m - 3, 31 - __clz(int(blockDim.x)));  // group bits that the thread number gives
                for (int i = 0; i < map->nruns; ++i) {
                    uint32_t sb = runs[i].flip;
                    for (int j = 0; j < tb; ++j) sb ^= (threadIdx.x >> j) & 1u ? uint32_t(runs[i].base[j]) : 0u;
                    sbase[i * int(blockDim.x) + int(threadIdx.x)] = uint16_t(sb);
                }
                out0 = map->flip;
                for (int j = 0; j < m; ++j) out0 ^= ((per16 * threadIdx.x) >> j) & 1u ? uint32_t(map->bit[j]) : 0u;
            }
            staged = b;
        }
        __syncthreads();
        if (a.rbits == 3) {
            adj_tile_runs<T>(uint32_t(sizeof(C)) * (uint32_t(2 * slot) << m), m, a, ush, runs, map->nruns, sbase, prog, ucode, umode, ucol, dlist, nd, myred, threadIdx.x,
                             blockDim.x);
        } else {
            for (int op = 0; op < a.n_ops;) {
                op += a.op_k[op] == 1 ? adj_tile_ops<T, 1>(pt, lt, m, a, op, ush, myred, threadIdx.x, blockDim.x)
                                      : adj_tile_ops<T, 2>(pt, lt, m, a, op, ush, myred, threadIdx.x, blockDim.x);
                __syncthreads();
            }
        }
        const uint64_t base = base_of(w);
        if (a.rbits == 3) {  // through the map: the two amplitudes of a 16-byte store may lie apart
            const int lg = 31 - __clz(int(per16 * blockDim.x));
            uint32_t s1 = out0, it = 0;
            for (uint32_t e = per16 * threadIdx.x; e < (1u << m); e += per16 * blockDim.x, ++it) {
                const uint64_t dst = base + (hoff[e >> L] | (e & lmask));
                for (uint32_t x = it & ~(it - 1), j = 0; it != 0 && (1u << j) <= x; ++j) s1 ^= map->bit[lg + j];
                if constexpr (per16 == 2) {
                    const uint32_t s2 = s1 ^ map->bit[0];
                    const C a0 = pt[s1], a1 = pt[s2], b0 = lt[s1], b1 = lt[s2];
                    *reinterpret_cast<float4*>(phi + dst) = make_float4(a0.x, a0.y, a1.x, a1.y);
                    *reinterpret_cast<float4*>(lam + dst) = make_float4(b0.x, b0.y, b1.x, b1.y);
                } else {
                    phi[dst] = pt[s1];
                    lam[dst] = lt[s1];
                }
            }
        } else for (uint32_t e = per16 * threadIdx.x; e < (1u << m); e += per16 * blockDim.x) {
            const uint64_t dst = base + (hoff[e >> L] | (e & lmask));
            *reinterpret_cast<float4*>(phi + dst) = *reinterpret_cast<const float4*>(pt + swz<T>(e));
            *reinterpret_cast<float4*>(lam + dst) = *reinterpret_cast<const float4*>(lt + swz<T>(e));
        }
        if ((i & (a.chunk_tiles - 1)) == a.chunk_tiles - 1) {  // chunk done: one partial per op, accumulators reset
            __syncthreads();  // every warp's sums of this tile are in
            const uint64_t chunk = w >> a.chunk_shift;
            for (int op = threadIdx.x; op < a.n_ops; op += blockDim.x) {
                if (a.op_out[op] < 0) continue;
                double t = 0.0;
                for (int wp = 0; wp < nwarps; ++wp) {
                    auto& r = red[size_t(wp) * a.n_ops + op];
                    t += wacc_value(r);
                    wacc_zero(r);
                }
                partials[chunk * a.n_ops + op] = t;
            }
        }
        __syncthreads();  // buffers free for the copy issued next; accumulators reset before the next tile
        if (nbuf == 1 && i + 1 < my_tiles) load_async(tile_of(i + 1), bufs, bufs + (size_t(1) << m));
    }
}

// grad_out[op_out[op] * batch + b] = sum over the state's chunks (in order) of partials[chunk * n_ops + op]
__global__ void adjoint_sweep_finish_kernel(const double* __restrict__ partials, int n_ops, int64_t batch, int cps,
                                            const __grid_constant__ AdjSweepArgs a, double* __restrict__ out) {
    const int64_t item = int64_t(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (item >= batch * n_ops) return;
    const int64_t b = item / n_ops;
    const int op = int(item - b * n_ops);
    if (a.op_out[op] < 0) return;
    double s = 0.0;
#pragma unroll 16  // loads ahead of the (ordered) additions: 24 qubits 20.7 us a sweep one after the other, 11.9 so
    for (int j = lane; j < cps; j += 32) s += partials[(b * cps + j) * n_ops + op];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[int64_t(a.op_out[op]) * batch + b] = s;
}

}  // namespace qgb

using namespace qgb;
using namespace qgb_host;

namespace {

template <typename T>
int launch_adj(void* phi, void* lam, const void* mats, const AdjSweepArgs& a, double* partials, cudaStream_t st) {
    auto kern = adjoint_sweep_kernel<T>;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
            return check_launch("adjoint sweep attribute");
        attr = true;
    }
    for (int nbuf = 2; nbuf >= 1; --nbuf) {
        // (the table for 512 threads where a block may get them)
        const size_t smem = adj_smem_bytes<T>(a.m, a.H, a.n_ops, a.n_runs, sizeof(T) == 8 ? 512 : 256, nbuf);
        if (smem > 227 * 1024) continue;
        int per_sm = 0, threads = 256;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem) != cudaSuccess)
            return check_launch("adjoint sweep occupancy");
        if (per_sm < 1) continue;
        if (per_sm == 1 && sizeof(T) == 8) {
            int p512 = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p512, kern, 512, smem) != cudaSuccess)
                return check_launch("adjoint sweep occupancy");
            if (p512 >= 1) threads = 512;
        }
        uint64_t grid = uint64_t(per_sm) * sm_count();
        if (grid > a.chunks) grid = a.chunks;
        kern<<<unsigned(grid), threads, smem, st>>>((cplx<T>*)phi, (cplx<T>*)lam, (const cplx<T>*)mats, a, partials,
                                                    nbuf);
        return check_launch("adjoint sweep kernel");
    }
    return set_error(QGB_EINVAL, "adjoint sweep tile of 2^%d amplitudes does not fit in shared memory", a.m);
}

int g_adj_run_bits = -1;  // register runs: -1 default (on), 0 per-op passes

// Register runs span 3 tile bits (8-amplitude groups of both tiles); 16-amplitude
// groups measured slower (more registers and code per op) and are not built.
int adj_run_bits(int dtype) {
    (void)dtype;
    return g_adj_run_bits == 0 ? 0 : 3;
}

}  // namespace

extern "C" int qgb_set_adjoint_runs(int bits) {
    if (bits != -1 && bits != 0 && bits != 3)
        return set_error(QGB_EINVAL, "adjoint register-run width %d (-1 default, 0 off, 3)", bits);
    g_adj_run_bits = bits;
    return QGB_OK;
}

extern "C" size_t qgb_adjoint_sweep_scratch_bytes(int n, int tile_bits, int n_ops, int64_t batch) {
    if (n < 1 || n > QGB_MAX_QUBITS || tile_bits < 1 || tile_bits > n || n_ops < 1 || n_ops > QGB_SWEEP_MAX_OPS ||
        batch < 1)
        return 0;
    const uint64_t tiles = uint64_t(1) << (n - tile_bits);
    return sizeof(double) * size_t(batch) * size_t(adj_chunks_per_state(tiles, batch)) * size_t(n_ops);
}

extern "C" int qgb_adjoint_sweep_step(void* phi, void* lam, int dtype, int n, const qgb_adjoint_sweep* sweep,
                                      const void* mats, int64_t mat_stride, int64_t batch, int64_t sv_stride,
                                      double* grad_out, void* scratch, size_t scratch_bytes, void* stream) {
    if (!phi || !lam || !sweep || !mats) return set_error(QGB_EINVAL, "null pointer");
    if (dtype != QGB_C64 && dtype != QGB_C128) return set_error(QGB_EINVAL, "dtype %d unknown", dtype);
    if (n < 1 || n > QGB_MAX_QUBITS) return set_error(QGB_EINVAL, "n=%d invalid", n);
    if (batch < 1) return set_error(QGB_EINVAL, "batch %lld < 1", (long long)batch);
    if (batch > 1 && sv_stride < (int64_t(1) << n)) return set_error(QGB_EINVAL, "state stride too small");
    if (mat_stride < 0) return set_error(QGB_EINVAL, "negative matrix stride");
    const int64_t esz = dtype == QGB_C64 ? 8 : 16;
    if ((reinterpret_cast<uintptr_t>(phi) & 15) || (reinterpret_cast<uintptr_t>(lam) & 15) ||
        (batch > 1 && (sv_stride * esz) % 16))
        return set_error(QGB_EINVAL, "state pointers and stride must be 16-byte aligned");
    if (reinterpret_cast<uintptr_t>(mats) % esz) return set_error(QGB_EINVAL, "matrix buffer misaligned");
    const int64_t span = (batch - 1) * (batch > 1 ? sv_stride : 0) + (int64_t(1) << n);
    const char* pb = static_cast<const char*>(phi);
    const char* lb = static_cast<const char*>(lam);
    if (pb < lb + span * esz && lb < pb + span * esz) return set_error(QGB_EINVAL, "the two batches overlap");
    const qgb_adjoint_sweep& sw = *sweep;
    const int L = sw.low_bits, H = sw.n_high, m = L + H;
    if (L < 1 || H < 0 || H > QGB_SWEEP_MAX_HIGH || m > n || m > QGB_SWEEP_MAX_TILE_BITS)
        return set_error(QGB_EINVAL, "tile geometry L=%d H=%d invalid for n=%d", L, H, n);
    if (sw.n_ops < 1 || sw.n_ops > QGB_SWEEP_MAX_OPS) return set_error(QGB_EINVAL, "n_ops=%d out of range", sw.n_ops);
    AdjSweepArgs a{};
    a.n = n;
    a.L = L;
    a.H = H;
    a.m = m;
    a.n_ops = sw.n_ops;
    uint64_t in_tile = (1ull << L) - 1;
    int prev = L - 1;
    for (int h = 0; h < H; ++h) {
        const int b = sw.high_bits[h];
        if (b <= prev || b >= n) return set_error(QGB_EINVAL, "high bits must be ascending, >= L and < n");
        in_tile |= 1ull << b;
        a.high_bits[h] = b;
        prev = b;
    }
    a.n_outer = 0;
    for (int b = 0; b < n; ++b)
        if (!((in_tile >> b) & 1ull)) a.outer_bits[a.n_outer++] = b;
    bool any_out = false;
    for (int i = 0; i < sw.n_ops; ++i) {
        const int k = sw.op_k[i];
        if (k < 1 || k > 2) return set_error(QGB_EINVAL, "adjoint sweep op %d has width %d (1 or 2)", i, k);
        if (k > m) return set_error(QGB_EINVAL, "adjoint sweep op %d wider than the tile", i);
        uint32_t seen = 0;
        for (int j = 0; j < k; ++j) {
            const int p = sw.op_pos[i][j];
            if (p < 0 || p >= m || ((seen >> p) & 1u))
                return set_error(QGB_EINVAL, "adjoint sweep op %d has bad tile bit %d", i, p);
            seen |= 1u << p;
            a.op_pos[i][j] = p;
        }
        if (sw.op_mat[i] < 0) return set_error(QGB_EINVAL, "adjoint sweep op %d has negative matrix offset", i);
        a.op_k[i] = k;
        a.op_mat[i] = sw.op_mat[i];
        a.op_out[i] = sw.op_out[i] < 0 ? -1 : sw.op_out[i];
        a.op_gcls[i] = kGenNone;
        if (a.op_out[i] >= 0) {
            any_out = true;
            const int d = 1 << k;
            uint32_t cols = 0;
            bool gdiag = true, gflip = true;
            for (int r = 0; r < d; ++r) {
                const int c = sw.op_gen_col[i][r];
                const double re = sw.op_gen_val[i][r][0], im = sw.op_gen_val[i][r][1];
                const bool unit = (re == 0.0 && (im == 1.0 || im == -1.0)) || (im == 0.0 && (re == 1.0 || re == -1.0));
                if (c < 0 || c >= d || !unit)
                    return set_error(QGB_EINVAL, "adjoint sweep op %d: generator row %d is not a Pauli-product row", i, r);
                a.gcol[i][r] = c;
                a.gval[i][r] = make_float2(float(re), float(im));
                cols |= 1u << c;
                gdiag = gdiag && c == r;
                gflip = gflip && c == d - 1 - r;
            }
            if (cols != (1u << d) - 1u)
                return set_error(QGB_EINVAL, "adjoint sweep op %d: generator rows are not a permutation", i);
            a.op_gcls[i] = gdiag ? kGenDiag : (gflip ? kGenFlip : kGenAny);
        }
    }
    if (any_out && !grad_out) return set_error(QGB_EINVAL, "derivatives requested without an output");
    // register runs: greedy, consecutive ops while their sites fit rbits tile bits
    a.rbits = adj_run_bits(dtype);
    if (a.rbits > m) a.rbits = m;
    if (a.rbits >= 3) {
        for (int i0 = 0; i0 < sw.n_ops;) {
            uint32_t bits = 0;
            int i = i0;
            for (; i < sw.n_ops; ++i) {
                uint32_t nb = bits;
                for (int j = 0; j < a.op_k[i]; ++j) nb |= 1u << a.op_pos[i][j];
                if (__builtin_popcount(nb) > a.rbits) break;
                bits = nb;
            }
            // the run's local bits: its own tile bits ascending, then the lowest unused ones
            int nrp = 0;
            for (int b = 0; b < m && nrp < a.rbits; ++b)
                if ((bits >> b) & 1u) a.run_pos[i0][nrp++] = b;
            for (int b = 0; b < m && nrp < a.rbits; ++b)
                if (!((bits >> b) & 1u)) a.run_pos[i0][nrp++] = b;
            a.run_len[i0] = i - i0;
            ++a.n_runs;
            for (int o = i0; o < i; ++o)
                for (int j = 0; j < a.op_k[o]; ++j)
                    for (int r = 0; r < a.rbits; ++r)
                        if (a.run_pos[i0][r] == a.op_pos[o][j]) a.op_lpos[o][j] = r;
            i0 = i;
        }
    } else {
        a.rbits = 0;
    }
    a.mat_stride = batch > 1 ? mat_stride : 0;
    a.batch = batch;
    a.sv_stride = batch > 1 ? sv_stride : 0;
    a.tiles = uint64_t(1) << (n - m);
    const int cps = adj_chunks_per_state(a.tiles, batch);
    a.chunk_tiles = a.tiles / uint64_t(cps);
    a.chunks = uint64_t(batch) * uint64_t(cps);
    a.tile_shift = n - m;
    a.chunk_shift = __builtin_ctzll(a.chunk_tiles);
    const size_t need = sizeof(double) * size_t(a.chunks) * size_t(a.n_ops);
    if (any_out && (!scratch || scratch_bytes < need))
        return set_error(QGB_ESCRATCH, "scratch of %zu bytes needed (qgb_adjoint_sweep_scratch_bytes)", need);
    cudaStream_t st = (cudaStream_t)stream;
    double* part = (double*)scratch;
    const int rc = dtype == QGB_C64 ? launch_adj<float>(phi, lam, mats, a, part, st)
                                    : launch_adj<double>(phi, lam, mats, a, part, st);
    if (rc || !any_out) return rc;
    const int64_t items = batch * a.n_ops;
    adjoint_sweep_finish_kernel<<<unsigned((items + 7) / 8), 256, 0, st>>>(part, a.n_ops, batch, cps, a, grad_out);
    return check_launch("adjoint sweep finish");
}
