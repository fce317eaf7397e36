// Noisy trajectories in one persistent launch.
//
// The reference samples noisy circuits one at a time on the CPU (MonteCarloSim,
// tensorQ/monte_carlo_sim.py:14-35, one statevector run per sample). Here one
// launch runs every trajectory through the whole circuit:
//
//  * each CTA takes the next trajectory from a work counter (an atomic ticket,
//    nobody waits on anybody) and owns it to the end: the circuit is cut on the
//    host into tile sweeps (ops whose bits fit one shared-memory tile: the low
//    L bits times H chosen high bits), and the CTA streams the trajectory's
//    state through shared memory once per sweep -- cp.async double buffering,
//    every op of the sweep applied to the staged tile -- ping-ponging between
//    the trajectory's own slot and a per-CTA scratch vector;
//  * after every gate, on each of its sites, a depolarising channel (I, or X,
//    Y, Z with p/3 each, sampled from Philox with the same counters as the
//    gate-by-gate kernel, so both paths draw the same Paulis) and amplitude
//    damping (Kraus K0 = diag(1, sqrt(1 - gamma)), K1 = sqrt(gamma) |0><1|);
//  * amplitude damping is unravelled exactly by the no-jump norm: the state
//    is advanced with K0 unnormalised; its squared norm after channel m,
//    N_m = N_{m-1} - gamma W_m (W_m the weight of the site's |1> component
//    just before the channel), is the probability of no jump up to m; with a
//    uniform threshold r the first jump is at the first m with N_m < r, which
//    has probability N_{m-1} - N_m = gamma W_m, as the sequential rule. The
//    W_m of a sweep are summed over its tiles; at the sweep's end the CTA walks
//    the channels, and if a jump falls inside the sweep it runs the sweep again
//    from its (untouched) input with K1 at that channel, renormalised, and a
//    fresh threshold. Without a jump the threshold carries over as r / N_end
//    (the conditional law) and the next sweep's first op rescales the state by
//    1 / sqrt(N_end). A last pass writes the normalised state to the
//    trajectory's slot.
//
// What bounds it: instructions, on 16 warps an SM (one CTA; the tile buffers fill shared memory).
// An op of a 16-amplitude group takes 96 to 128 FP32 instructions (op, K0, weights); the rest was
// overhead, 400 instructions an op in all: a select per damped component for a jump that hardly
// ever happens, a shuffle butterfly and a single lane's update per channel, moves of the group
// where the switches on positions join, and index arithmetic per tile and run. Now one switch per
// op into straight-line cases, jumps apart, weights summed 16 channels at a time through shared
// memory in the butterfly's order, half the products for x rotations and real ops, diagonal ops by
// a factor per local index, offsets from per-run tables: 230 instructions an op, and 152
// trajectories of the 20-qubit Ising circuit, 3 Trotter steps, from 20.0 to 12.2 ms; every
// rounding stays, so the states are the same bit for bit.
//
// Random numbers: Philox4x32-10 (philox.cuh). Pauli of site j after gate g:
// counter (g, trajectory, 2j, 0), as the gate-by-gate kernel; jump threshold
// number i of a trajectory: counter (i, trajectory, 0, 2).
#include "philox.cuh"
#include "qgb_common.cuh"

namespace qgb {

using TrajSweepDesc = qgb_traj_sweep;
using TrajOpDesc = qgb_traj_op;

constexpr int kTrajMaxOps = 128;    // ops per sweep
constexpr int kTrajMaxSmem = 222 * 1024;  // dynamic shared memory of a CTA
constexpr int kTrajMaxJumps = 16;   // jumps inside one sweep of one trajectory
constexpr int kTrajThreads = 512;  // 16 warps, one register group each at a time (100 registers): 15 % faster than
                                    // 8 warps with two groups each (215 registers), the latency-bound runs

struct TrajRunArgs {
    int n;
    int64_t ntraj, stride;
    int nsweeps;
    double p_dep, gamma;
    uint32_t seed0, seed1;
    int nbuf;            // tile buffers (2: the next tile's copy overlaps the ops)
    int mmax;            // largest tile bits of any sweep
    int max_log;         // jump log entries per trajectory
};

__device__ int g_traj_status = 0;

__device__ __forceinline__ void traj_cp16(void* smem_dst, const void* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src)
                 : "memory");
}

template <typename T> __device__ __forceinline__ uint32_t tswz(uint32_t e);
template <> __device__ __forceinline__ uint32_t tswz<float>(uint32_t e) { return swz<float>(e); }
template <> __device__ __forceinline__ uint32_t tswz<double>(uint32_t e) { return swz<double>(e); }

// ---- ops on a register group ------------------------------------------------
// A run of consecutive ops whose sites lie within R tile bits is applied to
// groups of 2^R amplitudes held in registers: local index bit P <-> the run's
// tile position run_pos[P]. Positions are runtime values; each (width,
// positions) case is its own fully unrolled instance, chosen by a switch, so
// the group never leaves registers.

template <typename C> __device__ __forceinline__ C cmul(const C& a, const C& b) {
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// A matrix entry pair in one 16-byte load (complex64).
__device__ __forceinline__ void ld_pair(const float2* m, float2& a, float2& b) {
    const float4 t = *reinterpret_cast<const float4*>(m);
    a = make_float2(t.x, t.y);
    b = make_float2(t.z, t.w);
}
__device__ __forceinline__ void ld_pair(const double2* m, double2& a, double2& b) {
    a = m[0];
    b = m[1];
}

// Diagonal op: m holds the factor of every local index, so no position is needed.
template <int R, typename C>
__device__ __forceinline__ void reg_diag(C (&v)[1 << R], const C* __restrict__ m) {
#pragma unroll
    for (int c = 0; c < (1 << R); c += 2) {
        C a, b;
        ld_pair(m + c, a, b);
        v[c] = cmul(v[c], a);
        v[c + 1] = cmul(v[c + 1], b);
    }
}

template <int R, int P, typename C>
__device__ __forceinline__ void reg_op1(C (&v)[1 << R], const C* __restrict__ m) {
    constexpr int D = 1 << R, bit = 1 << P;
    C m00, m01, m10, m11;
    ld_pair(m, m00, m01);
    ld_pair(m + 2, m10, m11);
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if (c & bit) continue;
        const C a = v[c], b = v[c | bit];
        C x = cmul(m00, a), y = cmul(m10, a);
        cfma(x, m01, b);
        cfma(y, m11, b);
        v[c] = x;
        v[c | bit] = y;
    }
}

// matrix index bit 1 (most significant) <-> local position P0 (the op's first site), bit 0 <-> P1
template <int R, int P0, int P1, typename C>
__device__ __forceinline__ void reg_op2(C (&v)[1 << R], const C* __restrict__ m) {
    constexpr int D = 1 << R, b0 = 1 << P0, b1 = 1 << P1;
    C mm[16];
#pragma unroll
    for (int e = 0; e < 16; e += 2) ld_pair(m + e, mm[e], mm[e + 1]);
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if ((c & b0) || (c & b1)) continue;
        const C x[4] = {v[c], v[c | b1], v[c | b0], v[c | b0 | b1]};
        C y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            y[r] = cmul(mm[4 * r], x[0]);
#pragma unroll
            for (int k = 1; k < 4; ++k) cfma(y[r], mm[4 * r + k], x[k]);
        }
        v[c] = y[0];
        v[c | b1] = y[1];
        v[c | b0] = y[2];
        v[c | b0 | b1] = y[3];
    }
}

// One-site op whose entries are real on the diagonal and imaginary off it (ROT: x
// rotations), or all real: half the products. The products left out are by an exact zero.
template <int R, int P, bool ROT, typename C>
__device__ __forceinline__ void reg_op1_half(C (&v)[1 << R], const C* __restrict__ m) {
    constexpr int D = 1 << R, bit = 1 << P;
    C m00, m01, m10, m11;
    ld_pair(m, m00, m01);
    ld_pair(m + 2, m10, m11);
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if (c & bit) continue;
        const C a = v[c], b = v[c | bit];
        if (ROT) {
            v[c].x = fma(-m01.y, b.y, m00.x * a.x);
            v[c].y = fma(m01.y, b.x, m00.x * a.y);
            v[c | bit].x = fma(m11.x, b.x, -(m10.y * a.y));
            v[c | bit].y = fma(m11.x, b.y, m10.y * a.x);
        } else {
            v[c].x = fma(m01.x, b.x, m00.x * a.x);
            v[c].y = fma(m01.x, b.y, m00.x * a.y);
            v[c | bit].x = fma(m11.x, b.x, m10.x * a.x);
            v[c | bit].y = fma(m11.x, b.y, m10.x * a.y);
        }
    }
}

// Both components times s; complex64 in one packed instruction (each rounded as alone).
__device__ __forceinline__ void scale2(float2& v, float s) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(v.x), "+f"(v.y)
        : "f"(s));
}
__device__ __forceinline__ void scale2(double2& v, double s) {
    v.x *= s;
    v.y *= s;
}

// Amplitude damping of the site at local position P: w += weight of its |1>
// components; then K0 (|1> components times s0) or a replayed jump (the |1>
// components times sj move to |0>, |1> cleared).
template <int R, int P, bool JUMP, typename C, typename T>
__device__ __forceinline__ void reg_damp(C (&v)[1 << R], T s, T& w) {
    constexpr int D = 1 << R, bit = 1 << P;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        if (!(c & bit)) continue;
        w = fma(v[c].x, v[c].x, w);
        w = fma(v[c].y, v[c].y, w);
        if (JUMP) {
            v[c ^ bit].x = s * v[c].x;
            v[c ^ bit].y = s * v[c].y;
            v[c].x = T(0);
            v[c].y = T(0);
        } else {
            scale2(v[c], s);
        }
    }
}

// Kinds of ops: one site general / real diagonal and imaginary off it / real; diagonal on one
// or two sites (a factor per local index); two sites general.
enum TrajKind : int { kOp1 = 0, kRot1 = 1, kReal1 = 2, kDiag1 = 3, kDiag2 = 4, kOp2 = 5 };

// Where an op's channels leave the lanes' weights: complex64 in the next rows of shared memory
// (TrajSweepSmem::rows), complex128 straight in the accumulators.
constexpr int kTrajRows = 16, kTrajRow = 36;

template <typename T> struct WeightSink;
template <> struct WeightSink<float> {
    float* at;  // the lane's element of the next row
    __device__ __forceinline__ void put(float w) {
        *at = w;
        at += kTrajRow;
    }
};
template <> struct WeightSink<double> {
    double* at;  // the next channel's accumulator
    __device__ __forceinline__ void put(double w) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if ((threadIdx.x & 31) == 0) wacc_add(*at, w);
        ++at;
    }
};

// An op and the K0 damping of its sites, straight-line.
template <int R, int KIND, int P0, int P1, bool DAMP, typename C, typename T>
__device__ __forceinline__ void reg_case(C (&v)[1 << R], const C* m, T s0, WeightSink<T>& sink) {
    constexpr bool two = KIND == kDiag2 || KIND == kOp2;
    if constexpr (P0 < R && (!two || (P1 < R && P0 != P1))) {
        if constexpr (KIND == kOp1) reg_op1<R, P0>(v, m);
        else if constexpr (KIND == kRot1) reg_op1_half<R, P0, true>(v, m);
        else if constexpr (KIND == kReal1) reg_op1_half<R, P0, false>(v, m);
        else if constexpr (KIND == kOp2) reg_op2<R, P0, P1>(v, m);
        else reg_diag<R>(v, m);
        if constexpr (DAMP) {
            T w = T(0);  // the state's precision: the jump and renormalisation factors come from these
            reg_damp<R, P0, false>(v, s0, w);
            sink.put(w);
            if constexpr (two) {
                w = T(0);
                reg_damp<R, P1, false>(v, s0, w);
                sink.put(w);
            }
        }
    }
}

// One switch per op: with one for the op and one per damped site the group changed
// registers at each join.
template <int R, bool DAMP, typename C, typename T>
__device__ __forceinline__ void reg_op(C (&v)[1 << R], int code, const C* m, T s0, WeightSink<T>& sink) {
#define QGB_ONE(K, P) case K * 16 + P * 4: reg_case<R, K, P, 0, DAMP>(v, m, s0, sink); break;
#define QGB_ONES(K) QGB_ONE(K, 0) QGB_ONE(K, 1) QGB_ONE(K, 2) QGB_ONE(K, 3)
#define QGB_TWO(K, P, Q) case K * 16 + P * 4 + Q: reg_case<R, K, P, Q, DAMP>(v, m, s0, sink); break;
#define QGB_TWOS(K)                                                                                              \
    QGB_TWO(K, 0, 1) QGB_TWO(K, 0, 2) QGB_TWO(K, 0, 3) QGB_TWO(K, 1, 0) QGB_TWO(K, 1, 2) QGB_TWO(K, 1, 3)       \
    QGB_TWO(K, 2, 0) QGB_TWO(K, 2, 1) QGB_TWO(K, 2, 3) QGB_TWO(K, 3, 0) QGB_TWO(K, 3, 1) QGB_TWO(K, 3, 2)
    switch (code) {
        QGB_ONES(kOp1)
        QGB_ONES(kRot1)
        QGB_ONES(kReal1)
        QGB_ONES(kDiag1)
        QGB_TWOS(kDiag2)
        QGB_TWOS(kOp2)
    }
#undef QGB_ONE
#undef QGB_ONES
#undef QGB_TWO
#undef QGB_TWOS
}

// Damping of one site, with or without a jump (only ops where a jump is replayed come here).
template <int R, typename C, typename T>
__device__ __forceinline__ void reg_damp_at(C (&v)[1 << R], int P, bool jump, T s0, T sj, T& w) {
    switch (P + (jump ? 4 : 0)) {
        case 0: reg_damp<R, 0, false>(v, s0, w); break;
        case 1: if constexpr (R > 1) reg_damp<R, 1, false>(v, s0, w); break;
        case 2: if constexpr (R > 2) reg_damp<R, 2, false>(v, s0, w); break;
        case 3: if constexpr (R > 3) reg_damp<R, 3, false>(v, s0, w); break;
        case 4: reg_damp<R, 0, true>(v, sj, w); break;
        case 5: if constexpr (R > 1) reg_damp<R, 1, true>(v, sj, w); break;
        case 6: if constexpr (R > 2) reg_damp<R, 2, true>(v, sj, w); break;
        case 7: if constexpr (R > 3) reg_damp<R, 3, true>(v, sj, w); break;
    }
}

// Per-warp accumulators of the damping weights (WAccOf, qgb_common.cuh): for
// complex64 a compensated float sum -- a float64 add per warp, op and tile kept
// GB300's narrow FP64 pipe 38 % busy -- for complex128 a double.
// Per-sweep, per-trajectory state in dynamic shared memory.
template <typename T> struct TrajSweepSmem {
    cplx<T>* msh;     // [op][16]: the op's matrix with its sampled Paulis folded in (first op: times the prescale)
    typename WAccOf<T>::type* chw_w;  // [warp][2 * kTrajMaxOps]: per-warp weights of |1> before each damping, by channel
    T* rows;          // [warp][kTrajRows][kTrajRow]: the lanes' weights of the last channels (complex64)
    T* djump;         // [op][2]: jump factor sqrt(gamma) / sqrt(gamma W) where a jump is replayed
    uint32_t* desc;   // [op]: kind, local positions, width, replayed jumps and first channel (TrajDesc)
    uint4* runs;      // [op][2]: at a run's first op, the swizzled byte offset of every local position; the bits
                      // below the run's ascending positions (16 bits each) and the run's length
};

// Op descriptor bits: the local positions of its sites and its kind (the case of reg_op), ...
enum TrajDesc : uint32_t { kDescP0 = 2, kDescP1 = 0, kDescKind = 4, kDescCode = 127, kDescTwo = 1u << 7,
                           kDescJump0 = 1u << 8, kDescJumps = 3u << 8, kDescChan = 10 };

// A channel's weights of the 32 lanes wait in a row of shared memory; when kTrajRows channels have
// one, lane j sums row j in the order of a shuffle butterfly and adds the sum to the channel's
// accumulator: 31 additions and 8 loads for 16 channels, where a butterfly per channel took 5
// shuffles, 5 additions and an update by a single lane each. The row pitch keeps the 16-byte loads
// of different rows on different banks.
__device__ __forceinline__ void traj_flush(const float* __restrict__ rows, int count, WAccF* __restrict__ acc, int lane) {
    __syncwarp();
    if (lane < count) {
        float x[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 q = *reinterpret_cast<const float4*>(rows + lane * kTrajRow + 4 * j);
            x[4 * j] = q.x;
            x[4 * j + 1] = q.y;
            x[4 * j + 2] = q.z;
            x[4 * j + 3] = q.w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int l = 0; l < o; ++l) x[l] = __fadd_rn(x[l], x[l + o]);
        wacc_add(acc[lane], x[0]);
    }
    __syncwarp();
}

// Every run of a sweep on one staged tile, a group of 2^R amplitudes per thread
// at a time, a barrier after each run.
template <typename T, int R, bool DAMP>
__device__ __forceinline__ void traj_tile_runs(cplx<T>* __restrict__ tile, int m, int nops,
                                               const TrajSweepSmem<T>& sm, T s0, int tid, int nthr) {
    using C = cplx<T>;
    constexpr int D = 1 << R;
    const int warp = tid >> 5, lane = tid & 31;
    auto* myw = sm.chw_w + size_t(warp) * (2 * kTrajMaxOps);
    T* rows = sm.rows + warp * (kTrajRows * kTrajRow);
    for (int i0 = 0; i0 < nops;) {
        const uint4 r0 = sm.runs[2 * i0], r1 = sm.runs[2 * i0 + 1];
        const uint32_t bit[4] = {r0.x, r0.y, r0.z, r0.w};
        const uint32_t below[4] = {r1.x & 0xffffu, r1.x >> 16, r1.y & 0xffffu, r1.y >> 16};
        const int nr = int(r1.z);
        const uint32_t groups = 1u << (m - R);
        for (uint32_t gb = 0; gb < groups; gb += uint32_t(nthr)) {
            C v[D];
            const uint32_t g = gb + uint32_t(tid);
            const bool ok = g < groups;
            uint32_t base = ok ? g : 0u;
#pragma unroll
            for (int j = 0; j < R; ++j) base += base & ~below[j];  // a zero bit at the position
            uint32_t at[D];  // byte offsets of the group; the swizzle is linear over XOR
            at[0] = tswz<T>(base) * uint32_t(sizeof(C));
#pragma unroll
            for (int j = 0; j < R; ++j)
#pragma unroll
                for (int l = 0; l < (1 << j); ++l) at[l + (1 << j)] = at[l] ^ bit[j];
#pragma unroll
            for (int l = 0; l < D; ++l)
                v[l] = ok ? *reinterpret_cast<const C*>(reinterpret_cast<const char*>(tile) + at[l]) : mk<T>(T(0), T(0));
            auto* acc = myw + (sm.desc[i0] >> kDescChan);  // of the next channel without a sum
            WeightSink<T> sink;
            if constexpr (sizeof(T) == 4) sink.at = rows + lane;
            else sink.at = acc;
            const C* mm = sm.msh + size_t(i0) * 16;
            const uint32_t* dp = sm.desc + i0;
            uint32_t next = *dp;
            for (int left = nr; left > 0; --left, mm += 16) {
                const uint32_t d = next;
                next = *++dp;  // one past the last op is the table after it
                if (!DAMP || !(d & kDescJumps)) {
                    reg_op<R, DAMP>(v, int(d & kDescCode), mm, s0, sink);
                } else {
                    const T* dj = sm.djump + 2 * (dp - 1 - sm.desc);
                    reg_op<R, false>(v, int(d & kDescCode), mm, s0, sink);
                    T w = T(0);
                    reg_damp_at<R>(v, (d >> kDescP0) & 3, (d & kDescJump0) != 0, s0, dj[0], w);
                    sink.put(w);
                    if (d & kDescTwo) {
                        w = T(0);
                        reg_damp_at<R>(v, (d >> kDescP1) & 3, (d & (kDescJump0 << 1)) != 0, s0, dj[1], w);
                        sink.put(w);
                    }
                }
                if constexpr (DAMP && sizeof(T) == 4) {
                    if (left == 1 || sink.at > rows + lane + (kTrajRows - 2) * kTrajRow) {
                        const int count = int(sink.at - (rows + lane)) / kTrajRow;
                        traj_flush(rows, count, acc, lane);
                        acc += count;
                        sink.at = rows + lane;
                    }
                }
            }
            if (ok)
#pragma unroll
                for (int l = 0; l < D; ++l) *reinterpret_cast<C*>(reinterpret_cast<char*>(tile) + at[l]) = v[l];
        }
        __syncthreads();
        i0 += nr;
    }
}

template <typename T, int RMAX, bool DAMP>
__device__ __forceinline__ void traj_tile_dispatch(cplx<T>* tile, int m, int nops, const TrajSweepSmem<T>& sm, T s0,
                                                   int tid, int nthr) {
    const int R = m < RMAX ? m : RMAX;
    switch (R) {
        case 1: traj_tile_runs<T, 1, DAMP>(tile, m, nops, sm, s0, tid, nthr); break;
        case 2: traj_tile_runs<T, 2, DAMP>(tile, m, nops, sm, s0, tid, nthr); break;
        case 3: traj_tile_runs<T, 3, DAMP>(tile, m, nops, sm, s0, tid, nthr); break;
        default: if constexpr (RMAX >= 4) traj_tile_runs<T, 4, DAMP>(tile, m, nops, sm, s0, tid, nthr); break;
    }
}

template <typename T> constexpr int traj_rmax() { return sizeof(T) == 4 ? 4 : 3; }

template <typename T> constexpr size_t traj_row_elems() {
    return sizeof(T) == 4 ? size_t(kTrajThreads / 32) * kTrajRows * kTrajRow : 0;
}

// dynamic shared memory: tile buffers | high-bit offsets | folded matrices | per-warp weights | lanes' weights |
// jump factors | op descriptors | run positions
template <typename T> __host__ __device__ constexpr size_t traj_aux_bytes() {
    return sizeof(uint32_t) * (size_t(1) << QGB_SWEEP_MAX_HIGH) + sizeof(cplx<T>) * kTrajMaxOps * 16 +
           sizeof(typename WAccOf<T>::type) * (kTrajThreads / 32) * 2 * kTrajMaxOps + sizeof(T) * traj_row_elems<T>() +
           sizeof(T) * 2 * kTrajMaxOps + (sizeof(uint32_t) + 2 * sizeof(uint4)) * kTrajMaxOps;
}

template <typename T>
__global__ void __launch_bounds__(kTrajThreads) traj_run_kernel(cplx<T>* __restrict__ states,
                                                                cplx<T>* __restrict__ pingpong,
                                                                const TrajSweepDesc* __restrict__ sweeps,
                                                                const TrajOpDesc* __restrict__ ops,
                                                                const cplx<T>* __restrict__ mats, int* queue,
                                                                int* __restrict__ jump_count, int* __restrict__ jump_log,
                                                                const __grid_constant__ TrajRunArgs a) {
    using C = cplx<T>;
    extern __shared__ __align__(16) unsigned char traj_smem[];
    C* bufs = reinterpret_cast<C*>(traj_smem);
    uint32_t* hoff = reinterpret_cast<uint32_t*>(bufs + (size_t(a.nbuf) << a.mmax));
    TrajSweepSmem<T> sm;
    sm.msh = reinterpret_cast<C*>(hoff + (size_t(1) << QGB_SWEEP_MAX_HIGH));
    sm.chw_w = reinterpret_cast<typename WAccOf<T>::type*>(sm.msh + kTrajMaxOps * 16);
    sm.rows = reinterpret_cast<T*>(sm.chw_w + (kTrajThreads / 32) * 2 * kTrajMaxOps);
    sm.djump = sm.rows + traj_row_elems<T>();
    sm.desc = reinterpret_cast<uint32_t*>(sm.djump + 2 * kTrajMaxOps);
    sm.runs = reinterpret_cast<uint4*>(sm.desc + kTrajMaxOps);
    __shared__ double chw[2 * kTrajMaxOps];  // per (op, site): weight of |1> before damping, summed over the tiles
    __shared__ uint8_t pk[kTrajMaxOps][2];   // sampled Paulis
    __shared__ int jop[kTrajMaxJumps], jsite[kTrajMaxJumps];
    __shared__ double jscale[kTrajMaxJumps];
    __shared__ int s_traj, s_njump, s_replay;
    __shared__ double s_r, s_prescale;
    __shared__ int s_jumps_total;
    const int tid = threadIdx.x, nthr = blockDim.x, nwarps = blockDim.x >> 5;
    const uint64_t dim = uint64_t(1) << a.n;
    C* scratch = pingpong + uint64_t(blockIdx.x) * dim;
    const T s0 = T(sqrt(1.0 - a.gamma));
    const bool damp = a.gamma > 0;
    constexpr uint32_t per16 = 16 / sizeof(C);
    while (true) {
        if (tid == 0) {
            s_traj = atomicAdd(queue, 1);
            s_r = Philox::uniform4(0u, uint32_t(s_traj), 0u, 2u, a.seed0, a.seed1);
            s_prescale = 1.0;
            s_jumps_total = 0;
        }
        __syncthreads();
        const int64_t t = s_traj;
        if (t >= a.ntraj) break;
        C* own = states + t * a.stride;
        C* src = nullptr;  // null: the sweep starts from |0...0>
        C* dst = scratch;
        for (int s = 0; s < a.nsweeps; ++s) {
            const TrajSweepDesc sw = sweeps[s];
            const int L = sw.L, H = sw.H, m = L + H, nops = sw.op_end - sw.op_begin;
            const TrajOpDesc* sops = ops + sw.op_begin;
            const uint32_t lmask = (1u << L) - 1u;
            // tile-index -> global offset of the high bits; the outer bits enumerate tiles
            for (uint32_t h = tid; h < (1u << H); h += nthr) {
                uint32_t o = 0;
                for (int j = 0; j < H; ++j) o |= ((h >> j) & 1u) << sw.high_bits[j];
                hoff[h] = o;
            }
            uint32_t in_tile = lmask;
            for (int j = 0; j < H; ++j) in_tile |= 1u << sw.high_bits[j];
            // the Paulis of the sweep's channels (state independent, the gate-by-gate kernel's counters)
            for (int c = tid; c < 2 * nops; c += nthr) {
                const int i = c >> 1, j = c & 1;
                int p = 0;
                if (a.p_dep > 0 && j < sops[i].k) {
                    const double u = Philox::uniform(uint32_t(sops[i].gate), uint32_t(t), 2u * j, a.seed0, a.seed1);
                    if (u >= 1.0 - a.p_dep) p = 1 + min(2, int((u - (1.0 - a.p_dep)) / (a.p_dep / 3.0)));
                }
                pk[i][j] = uint8_t(p);
            }
            if (tid == 0) s_njump = 0;
            __syncthreads();
            // each op's matrix with its Paulis folded into the rows (X swaps, Y swaps with -i / i, Z negates
            // the |1> row of its site); the first op of the sweep also carries the prescale 1 / sqrt(N_end)
            for (int i = tid; i < nops; i += nthr) {
                const TrajOpDesc& op = sops[i];
                const int D = 1 << op.k;
                C M[16];
                const T ps = i == 0 ? T(s_prescale) : T(1);
                for (int e = 0; e < D * D; ++e) {
                    const C x = mats[op.mat + e];
                    M[e] = mk<T>(x.x * ps, x.y * ps);
                }
                bool diag = (op.flags & 1) != 0;
                for (int j = 0; j < op.k; ++j) {
                    const int pj = pk[i][j];
                    if (pj == 0) continue;
                    if (pj != 3) diag = false;
                    const int bit = 1 << (op.k - 1 - j);
                    for (int r = 0; r < D; ++r) {
                        if (r & bit) continue;
                        for (int c = 0; c < D; ++c) {
                            const C lo = M[r * D + c], hi = M[(r | bit) * D + c];
                            if (pj == 1) {
                                M[r * D + c] = hi;
                                M[(r | bit) * D + c] = lo;
                            } else if (pj == 2) {
                                M[r * D + c] = mk<T>(hi.y, -hi.x);
                                M[(r | bit) * D + c] = mk<T>(-lo.y, lo.x);
                            } else {
                                M[(r | bit) * D + c] = mk<T>(-hi.x, -hi.y);
                            }
                        }
                    }
                }
                C* out = sm.msh + size_t(i) * 16;
                if (diag) {  // the factor of every local index of the run's group
                    const int r = m < traj_rmax<T>() ? m : traj_rmax<T>();
                    for (int c = 0; c < (1 << r); ++c) {
                        int e = (c >> op.lpos[0]) & 1;
                        if (op.k == 2) e = 2 * e + ((c >> op.lpos[1]) & 1);
                        out[c] = M[e * (D + 1)];
                    }
                } else {
                    for (int e = 0; e < D * D; ++e) out[e] = M[e];
                }
                uint32_t chan = 0;
                for (int x = 0; x < i; ++x) chan += uint32_t(sops[x].k);
                int kind = op.k == 1 ? (diag ? kDiag1 : kOp1) : (diag ? kDiag2 : kOp2);
                if (kind == kOp1) {
                    if (M[0].y == T(0) && M[3].y == T(0) && M[1].x == T(0) && M[2].x == T(0)) kind = kRot1;
                    else if (M[0].y == T(0) && M[3].y == T(0) && M[1].y == T(0) && M[2].y == T(0)) kind = kReal1;
                }
                sm.desc[i] = uint32_t(kind) << kDescKind | uint32_t(op.lpos[0]) << kDescP0 |
                             (op.k == 2 ? uint32_t(op.lpos[1]) << kDescP1 | kDescTwo : 0u) | chan << kDescChan;
                if (op.run > 0) {
                    const int r = m < traj_rmax<T>() ? m : traj_rmax<T>();
                    uint32_t b[4] = {0, 0, 0, 0}, low[4] = {0, 0, 0, 0};
                    for (int x = 0; x < r; ++x) {
                        int rank = 0;
                        for (int y = 0; y < r; ++y) rank += op.run_pos[y] < op.run_pos[x];
                        b[x] = tswz<T>(1u << op.run_pos[x]) * uint32_t(sizeof(C));
                        low[rank] = (1u << op.run_pos[x]) - 1u;
                    }
                    sm.runs[2 * i] = make_uint4(b[0], b[1], b[2], b[3]);
                    sm.runs[2 * i + 1] = make_uint4(low[0] | low[1] << 16, low[2] | low[3] << 16, uint32_t(op.run), 0u);
                }
            }
            const uint64_t tiles = uint64_t(1) << (a.n - m);
            // bases of successive tiles: a count over the bits outside the tile
            auto after = [&](uint32_t base) -> uint32_t { return ((base | in_tile) + 1u) & ~in_tile; };
            // Offsets of the thread's 16-byte pieces: offset and swizzle are linear over disjoint bits, so a
            // piece's are the thread's, once a sweep, and the step's, the same for all threads.
            const uint32_t step = per16 * nthr, e_t = per16 * tid;
            uint32_t off_t = e_t & lmask;
            for (int j = 0; j < H; ++j) off_t |= (((e_t & ((1u << m) - 1u)) >> (L + j)) & 1u) << sw.high_bits[j];
            const uint32_t sw_t = tswz<T>(e_t);
            auto load = [&](uint32_t base, C* buf) {
                if (src) {
#pragma unroll 4
                    for (uint32_t e = 0; e + e_t < (1u << m); e += step)
                        traj_cp16(buf + (sw_t ^ tswz<T>(e)), src + (base + off_t + hoff[e >> L] + (e & lmask)));
                } else {
                    for (uint32_t e = tid; e < (1u << m); e += nthr) {
                        const uint32_t gi = base + hoff[e >> L] + (e & lmask);
                        buf[tswz<T>(e)] = mk<T>(gi == 0 ? T(1) : T(0), T(0));
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            for (int pass = 0; pass <= kTrajMaxJumps; ++pass) {
                // damping of every (op, site): K0, or the replayed jumps of this sweep
                for (int c = tid; c < 2 * nops; c += nthr) sm.djump[c] = T(0);
                for (int c = tid; c < nwarps * 2 * nops; c += nthr)
                    wacc_zero(sm.chw_w[size_t(c / (2 * nops)) * (2 * kTrajMaxOps) + (c % (2 * nops))]);
                __syncthreads();
                if (tid == 0)
                    for (int q = 0; q < s_njump; ++q) {
                        sm.desc[jop[q]] |= kDescJump0 << jsite[q];
                        sm.djump[2 * jop[q] + jsite[q]] = T(sqrt(a.gamma) * jscale[q]);
                    }
                __syncthreads();
                uint32_t base = 0, base_next = after(0);
                load(0, bufs);
                for (uint64_t w = 0; w < tiles; ++w) {
                    C* cur = bufs + (size_t(a.nbuf == 2 ? (w & 1) : 0) << m);
                    if (a.nbuf == 2 && w + 1 < tiles) {
                        load(base_next, bufs + (size_t((w + 1) & 1) << m));
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                    } else {
                        asm volatile("cp.async.wait_group 0;" ::: "memory");
                    }
                    __syncthreads();
                    if (damp) traj_tile_dispatch<T, traj_rmax<T>(), true>(cur, m, nops, sm, s0, tid, nthr);
                    else traj_tile_dispatch<T, traj_rmax<T>(), false>(cur, m, nops, sm, s0, tid, nthr);
#pragma unroll 4
                    for (uint32_t e = 0; e + e_t < (1u << m); e += step)
                        *reinterpret_cast<float4*>(dst + (base + off_t + hoff[e >> L] + (e & lmask))) =
                            *reinterpret_cast<const float4*>(cur + (sw_t ^ tswz<T>(e)));
                    __syncthreads();  // the buffer is free for the copy issued two tiles later
                    if (a.nbuf == 1 && w + 1 < tiles) load(base_next, bufs);
                    base = base_next;
                    base_next = after(base);
                }
                // the weights, summed over the warps in a fixed order
                for (int c = tid; c < 2 * nops; c += nthr) {
                    const uint32_t d = sm.desc[c >> 1];
                    if ((c & 1) && !(d & kDescTwo)) continue;
                    const size_t ch = (d >> kDescChan) + (c & 1);
                    double x = 0.0;
                    for (int wp = 0; wp < nwarps; ++wp) x += wacc_value(sm.chw_w[size_t(wp) * (2 * kTrajMaxOps) + ch]);
                    chw[c] = x;
                }
                __syncthreads();
                // the sweep's channels in order: where does the no-jump norm fall below the threshold?
                if (tid == 0) {
                    s_replay = 0;
                    double N = 1.0;
                    if (damp) {
                        // channels up to the last jump recorded in this sweep are decided; after it the
                        // replay renormalised the state, so the walk restarts there with N = 1
                        int i0 = 0, j0 = 0;
                        if (s_njump > 0) {
                            i0 = jop[s_njump - 1];
                            j0 = jsite[s_njump - 1] + 1;
                        }
                        for (int i = i0; i < nops && !s_replay; ++i) {
                            const int k = sops[i].k;
                            for (int j = (i == i0 ? j0 : 0); j < k; ++j) {
                                const double Wc = chw[2 * i + j];
                                const double Nn = N - a.gamma * Wc;
                                if (Nn < s_r) {
                                    if (s_njump >= kTrajMaxJumps) {
                                        atomicExch(&g_traj_status, 1);  // too many jumps in one sweep: not replayed
                                        i = nops;
                                        break;
                                    }
                                    jop[s_njump] = i;
                                    jsite[s_njump] = j;
                                    jscale[s_njump] = 1.0 / sqrt(a.gamma * Wc);
                                    ++s_njump;
                                    const int idx = s_jumps_total++;
                                    if (idx < a.max_log && jump_log) {
                                        jump_log[(t * a.max_log + idx) * 2] = sops[i].gate;
                                        jump_log[(t * a.max_log + idx) * 2 + 1] = j;
                                    }
                                    s_r = Philox::uniform4(uint32_t(idx + 1), uint32_t(t), 0u, 2u, a.seed0, a.seed1);
                                    s_replay = 1;
                                    break;
                                }
                                N = Nn;
                            }
                        }
                    }
                    if (!s_replay) {
                        s_r = s_r / N;
                        s_prescale = 1.0 / sqrt(N);
                    }
                }
                __syncthreads();
                if (!s_replay) break;
            }
            src = dst;
            dst = (dst == own) ? scratch : own;
        }
        // the normalised state into the trajectory's slot
        {
            const T sc = T(s_prescale);
            if (src) {
                {
#pragma unroll 4
                    for (uint64_t e = uint64_t(per16) * tid; e < dim; e += per16 * nthr) {
                        float4 q = *reinterpret_cast<const float4*>(src + e);
                        T* x = reinterpret_cast<T*>(&q);
#pragma unroll
                        for (int j = 0; j < int(2 * per16); ++j) x[j] *= sc;
                        *reinterpret_cast<float4*>(own + e) = q;
                    }
                }
            } else {
                for (uint64_t e = tid; e < dim; e += nthr) own[e] = mk<T>(e == 0 ? T(1) : T(0), T(0));
            }
        }
        if (tid == 0 && jump_count) jump_count[t] = s_jumps_total;
        __syncthreads();
    }
}

}  // namespace qgb

using namespace qgb;
using namespace qgb_host;

namespace {

template <typename T>
size_t traj_smem_bytes(int mmax, int hmax, int nbuf) {
    (void)hmax;
    return sizeof(cplx<T>) * (size_t(nbuf) << mmax) + traj_aux_bytes<T>();
}

template <typename T>
int traj_grid(int mmax, int hmax, int64_t ntraj, int* nbuf_out, size_t* smem_out) {
    auto kern = traj_run_kernel<T>;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrajMaxSmem) != cudaSuccess)
            return check_launch("trajectory kernel attribute");
        attr = true;
    }
    for (int nbuf = 2; nbuf >= 1; --nbuf) {
        const size_t smem = traj_smem_bytes<T>(mmax, hmax, nbuf);
        if (smem > kTrajMaxSmem) continue;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTrajThreads, smem) != cudaSuccess)
            return check_launch("trajectory kernel occupancy");
        if (per_sm < 1) continue;
        int64_t grid = int64_t(per_sm) * sm_count();
        if (grid > ntraj) grid = ntraj;
        *nbuf_out = nbuf;
        *smem_out = smem;
        return int(grid);
    }
    return set_error(QGB_EINVAL, "trajectory tile of 2^%d amplitudes does not fit in shared memory", mmax);
}

int traj_check_tables(int n, const TrajSweepDesc* sweeps, int nsweeps, const TrajOpDesc* ops, int nops_total,
                      int64_t mat_elems, int* mmax, int* hmax, int dtype) {
    *mmax = 1;
    *hmax = 0;
    const int lmin = dtype == QGB_C64 ? 1 : 0;
    for (int s = 0; s < nsweeps; ++s) {
        const TrajSweepDesc& sw = sweeps[s];
        const int m = sw.L + sw.H;
        if (sw.L < lmin || sw.H < 0 || sw.H > QGB_SWEEP_MAX_HIGH || m > n || m > 14)
            return set_error(QGB_EINVAL, "sweep %d: tile geometry L=%d H=%d invalid for n=%d", s, sw.L, sw.H, n);
        int prev = sw.L - 1;
        for (int j = 0; j < sw.H; ++j) {
            if (sw.high_bits[j] <= prev || sw.high_bits[j] >= n)
                return set_error(QGB_EINVAL, "sweep %d: high bits must be ascending, >= L and < n", s);
            prev = sw.high_bits[j];
        }
        if (sw.op_begin < 0 || sw.op_end < sw.op_begin || sw.op_end > nops_total || sw.op_end - sw.op_begin > kTrajMaxOps ||
            sw.op_end == sw.op_begin)
            return set_error(QGB_EINVAL, "sweep %d: op range [%d, %d) invalid", s, sw.op_begin, sw.op_end);
        if (m > *mmax) *mmax = m;
        if (sw.H > *hmax) *hmax = sw.H;
        const int R = m < (dtype == QGB_C64 ? 4 : 3) ? m : (dtype == QGB_C64 ? 4 : 3);
        int run_left = 0;
        const int32_t* rpos = nullptr;
        for (int i = sw.op_begin; i < sw.op_end; ++i) {
            const TrajOpDesc& op = ops[i];
            if (run_left == 0) {
                if (op.run < 1 || i + op.run > sw.op_end)
                    return set_error(QGB_EINVAL, "op %d: run length %d invalid in its sweep", i, op.run);
                uint32_t seen = 0;
                for (int j = 0; j < R; ++j) {
                    const int p = op.run_pos[j];
                    if (p < 0 || p >= m || ((seen >> p) & 1u)) return set_error(QGB_EINVAL, "op %d: run positions invalid", i);
                    seen |= 1u << p;
                }
                run_left = op.run;
                rpos = op.run_pos;
            } else if (op.run != 0) {
                return set_error(QGB_EINVAL, "op %d opens a run inside another run", i);
            }
            --run_left;
            if (op.k < 1 || op.k > 2 || op.k > m) return set_error(QGB_EINVAL, "op %d: width %d invalid", i, op.k);
            for (int j = 0; j < op.k; ++j) {
                if (op.pos[j] < 0 || op.pos[j] >= m) return set_error(QGB_EINVAL, "op %d: tile position out of range", i);
                if (op.lpos[j] < 0 || op.lpos[j] >= R || rpos[op.lpos[j]] != op.pos[j])
                    return set_error(QGB_EINVAL, "op %d: local position does not match its run", i);
            }
            if (op.k == 2 && op.pos[0] == op.pos[1]) return set_error(QGB_EINVAL, "op %d: repeated tile position", i);
            if (op.gate < 0 || op.mat < 0 || op.mat + (int64_t(1) << (2 * op.k)) > mat_elems)
                return set_error(QGB_EINVAL, "op %d: gate index or matrix offset out of range", i);
        }
    }
    return QGB_OK;
}

}  // namespace

extern "C" size_t qgb_traj_sweep_bytes(void) { return sizeof(TrajSweepDesc); }
extern "C" size_t qgb_traj_op_bytes(void) { return sizeof(TrajOpDesc); }

extern "C" size_t qgb_traj_run_scratch_bytes(int dtype, int n, int tile_bits, int64_t ntraj) {
    if ((dtype != QGB_C64 && dtype != QGB_C128) || n < 1 || n > 30 || tile_bits < 1 || tile_bits > 14 || ntraj < 1)
        return 0;
    const int m = tile_bits < n ? tile_bits : n;
    int nbuf = 0;
    size_t smem = 0;
    const int grid = dtype == QGB_C64 ? traj_grid<float>(m, QGB_SWEEP_MAX_HIGH, ntraj, &nbuf, &smem)
                                      : traj_grid<double>(m, QGB_SWEEP_MAX_HIGH, ntraj, &nbuf, &smem);
    if (grid <= 0) return 0;
    const size_t isz = dtype == QGB_C64 ? 8 : 16;
    return 256 + size_t(grid) * (size_t(1) << n) * isz;
}

extern "C" int qgb_traj_run(void* sv, int dtype, int n, int64_t ntraj, int64_t stride, const qgb_traj_sweep* sweeps_host,
                            const qgb_traj_sweep* sweeps_dev, int nsweeps, const qgb_traj_op* ops_host,
                            const qgb_traj_op* ops_dev, int nops, const void* mats, int64_t mat_elems, double p_dep, double gamma, uint64_t seed, int* jump_count,
                            int* jump_log, int max_log, void* scratch, size_t scratch_bytes, void* stream) {
    if (!sv || !sweeps_host || !sweeps_dev || !ops_host || !ops_dev || !mats || !scratch)
        return set_error(QGB_EINVAL, "null pointer");
    if (dtype != QGB_C64 && dtype != QGB_C128) return set_error(QGB_EINVAL, "dtype %d unknown", dtype);
    if (n < 1 || n > 30) return set_error(QGB_EINVAL, "n=%d invalid (trajectories of 1 to 30 qubits)", n);
    if (ntraj < 1 || ntraj > (int64_t(1) << 30)) return set_error(QGB_EINVAL, "ntraj %lld out of range", (long long)ntraj);
    if (ntraj > 1 && stride < (int64_t(1) << n)) return set_error(QGB_EINVAL, "trajectory stride too small");
    if (nsweeps < 0 || nops < 0) return set_error(QGB_EINVAL, "negative table size");
    if (p_dep < 0 || p_dep > 1 || gamma < 0 || gamma >= 1) return set_error(QGB_EINVAL, "noise parameters out of range");
    if (max_log < 0 || (max_log > 0 && !jump_log)) return set_error(QGB_EINVAL, "jump log missing");
    const size_t isz = dtype == QGB_C64 ? 8 : 16;
    if ((reinterpret_cast<uintptr_t>(sv) & 15) || (ntraj > 1 && (stride * int64_t(isz)) % 16) ||
        (reinterpret_cast<uintptr_t>(scratch) & 15))
        return set_error(QGB_EINVAL, "state, stride and scratch must be 16-byte aligned");
    if (reinterpret_cast<uintptr_t>(mats) % isz) return set_error(QGB_EINVAL, "matrix buffer misaligned");
    int mmax = 1, hmax = 0;
    int rc = traj_check_tables(n, reinterpret_cast<const TrajSweepDesc*>(sweeps_host), nsweeps,
                               reinterpret_cast<const TrajOpDesc*>(ops_host), nops, mat_elems, &mmax, &hmax, dtype);
    if (rc) return rc;
    int nbuf = 0;
    size_t smem = 0;
    // shared memory sized for the largest high-bit table, as qgb_traj_run_scratch_bytes assumes
    (void)hmax;
    const int grid = dtype == QGB_C64 ? traj_grid<float>(mmax, QGB_SWEEP_MAX_HIGH, ntraj, &nbuf, &smem)
                                      : traj_grid<double>(mmax, QGB_SWEEP_MAX_HIGH, ntraj, &nbuf, &smem);
    if (grid <= 0) return grid < 0 ? grid : set_error(QGB_ECUDA, "no trajectory CTA fits on an SM");
    const size_t need = 256 + size_t(grid) * (size_t(1) << n) * isz;
    if (scratch_bytes < need) return set_error(QGB_ESCRATCH, "trajectory scratch of %zu bytes needed", need);
    cudaStream_t st = (cudaStream_t)stream;
    int* queue = static_cast<int*>(scratch);
    if (cudaMemsetAsync(queue, 0, sizeof(int), st) != cudaSuccess) return check_launch("trajectory queue reset");
    void* ping = static_cast<unsigned char*>(scratch) + 256;
    TrajRunArgs a{};
    a.n = n;
    a.ntraj = ntraj;
    a.stride = ntraj > 1 ? stride : 0;
    a.nsweeps = nsweeps;
    a.p_dep = p_dep;
    a.gamma = gamma;
    a.seed0 = uint32_t(seed);
    a.seed1 = uint32_t(seed >> 32);
    a.nbuf = nbuf;
    a.mmax = mmax;
    a.max_log = max_log;
    const TrajSweepDesc* sd = reinterpret_cast<const TrajSweepDesc*>(sweeps_dev);
    const TrajOpDesc* od = reinterpret_cast<const TrajOpDesc*>(ops_dev);
    if (dtype == QGB_C64)
        traj_run_kernel<float><<<grid, kTrajThreads, smem, st>>>((float2*)sv, (float2*)ping, sd, od,
                                                                  (const float2*)mats, queue, jump_count, jump_log, a);
    else
        traj_run_kernel<double><<<grid, kTrajThreads, smem, st>>>((double2*)sv, (double2*)ping, sd, od,
                                                                   (const double2*)mats, queue, jump_count, jump_log, a);
    return check_launch("trajectory kernel");
}

namespace qgb_host {
int traj_status_read_clear() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, qgb::g_traj_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) {
        const int z = 0;
        cudaMemcpyToSymbol(qgb::g_traj_status, &z, sizeof(int));
    }
    return v;
}
}  // namespace qgb_host
