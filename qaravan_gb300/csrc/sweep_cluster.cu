// Tile sweeps of small vectors: one tile spread over a thread-block cluster.
//
// The sweep kernels (sweep.cu, sweep_df.cu) give each tile to one CTA and each
// thread whole groups of partner amplitudes. A vector of a few tiles leaves the
// chip idle, and in a tile of few groups most threads wait while some form all
// 2^k output rows of an op: an op then costs 2-8 us whatever the arithmetic
// (12 qubits, 3-qubit blocks in double-float: 8 us an op on one SM). Here
//   * a cluster of R CTAs (R a power of two up to 16) holds the tile, CTA `rank`
//     the amplitudes whose top log2(R) tile bits equal its rank;
//   * a thread forms as few output rows as there are threads for (one, in a
//     CTA's part of up to 512 amplitudes), reading the 2^k inputs from the shared
//     memory of the CTAs that hold them (distributed shared memory where the op
//     acts on a rank bit);
//   * the tile is kept twice and an op writes to the other copy, so an op costs
//     one barrier: of the cluster when it or its neighbour reads other CTAs'
//     parts, else of the CTA;
//   * ops' geometry and matrices (in the tile's number format) are staged for many
//     ops at once.
// The rows are summed in the order of the other kernels and with their
// arithmetic (float32, or double-float for complex128), so the results are
// theirs bit for bit.
//
// What bounds it: the FP32 issue rate of one row per thread for double-float
// (about 550 instructions an op of 3 qubits and thread) and latency for float32
// (the barriers, remote loads and the sum chain of a row). Depth-20 brickwork
// against one CTA per tile, complex128: 12 qubits 901 -> 171 us, 16 qubits 2479 ->
// 510 us; 4-qubit blocks of complex64: 12 qubits 133 -> 86 us, 6 sites of a
// density matrix 130 -> 105 us.
#include "sweep_df.cuh"

namespace qgb {

constexpr int kClBits = 9;
constexpr int kClThreads = 1 << kClBits;
constexpr int kClMaxRankBits = 4;  // 16 CTAs (more than 8 need the non-portable attribute)
constexpr int kClSmem = 220 * 1024;
constexpr int kClMats = 4096;  // staged matrix entries: 64 ops of 3 qubits, 16 of 4

template <typename T> struct ClAmp;
template <> struct ClAmp<float> { using type = float2; };
template <> struct ClAmp<double> { using type = dfc; };

__device__ __forceinline__ float2 cl_in(float2 v) { return v; }
__device__ __forceinline__ dfc cl_in(double2 v) {
    dfc y;
    df_split(v.x, y.rh, y.rl);
    df_split(v.y, y.ih, y.il);
    return y;
}
__device__ __forceinline__ float2 cl_out(float2 v) { return v; }
__device__ __forceinline__ double2 cl_out(const dfc& v) { return make_double2(df_join(v.rh, v.rl), df_join(v.ih, v.il)); }

__device__ __forceinline__ void cl_load(float2& v, uint32_t addr) {
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cl_load(dfc& v, uint32_t addr) {
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.rh), "=f"(v.rl), "=f"(v.ih), "=f"(v.il)
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One output row: sum over the columns in order.
template <int D>
__device__ __forceinline__ float2 cl_row(const float2* __restrict__ mrow, const float2 (&v)[D]) {
    float2 acc = make_float2(0.f, 0.f);
    const float4* m4 = reinterpret_cast<const float4*>(mrow);
#pragma unroll
    for (int c = 0; c < D; c += 2) {
        const float4 q = m4[c >> 1];
        cfma(acc, make_float2(q.x, q.y), v[c]);
        cfma(acc, make_float2(q.z, q.w), v[c + 1]);
    }
    return acc;
}
template <int D>
__device__ __forceinline__ dfc cl_row(const dfc* __restrict__ mrow, const dfc (&v)[D]) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < D; ++c) dfc_mac(s, mrow[c], v[c]);
    return dfc_finish(s);
}

// An op as one CTA of the cluster sees it, worked out once per launch.
// Matrix bit b (value 1 << b) is tile bit pos[k - 1 - b]: a local one (its
// amplitude offset in lbit[b]) or a rank bit (in rbit[b]).
struct ClOp {
    uint32_t lbit[QGB_MAX_K - 1], rbit[QGB_MAX_K - 1];
    uint32_t taken;   // the local bits
    uint32_t rk;      // the rank bits
    uint32_t mine;    // the matrix rows' bits fixed by the rank
    int nl, k;
    int moff;         // its matrix in the staged chunk
};

// One op on this CTA's part of the tile: src -> dst, ml local tile bits.
template <typename T, int K>
__device__ __forceinline__ void cl_op(const typename ClAmp<T>::type* __restrict__ src,
                                      typename ClAmp<T>::type* __restrict__ dst, int ml, uint32_t rank,
                                      const ClOp& op, const typename ClAmp<T>::type* __restrict__ msh) {
    constexpr int D = 1 << K;
    using A = typename ClAmp<T>::type;
    uint32_t lbit[K];
#pragma unroll
    for (int b = 0; b < K; ++b) lbit[b] = op.lbit[b];
    const uint32_t taken = op.taken, rk = op.rk, mine = op.mine;
    const int nl = op.nl, lg = ml - nl;  // 2^lg groups in this part
    // rows per thread: the part's outputs over the threads, at most a group's local rows
    int lr = ml > kClBits ? ml - kClBits : 0;
    if (lr > nl) lr = nl;
    const uint32_t items = 1u << (ml - lr);
    for (uint32_t it = threadIdx.x; it < items; it += kClThreads) {
        const uint32_t chunk = it >> lg;
        uint32_t base = it & ((1u << lg) - 1u);  // the group's bits at the free local positions
        uint32_t left = taken;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const uint32_t low = left & (0u - left);  // 0 once all bits are in: base stays
            const uint32_t keep = base & (low - 1u);
            base = base + (base - keep);
            if (low == 0u) base = keep;
            left ^= low;
        }
        const uint32_t sb = swz<T>(base);
        A v[D];
        if (rk == 0) {
            uint32_t so[D];
            so[0] = sb;
#pragma unroll
            for (int b = 0; b < K; ++b) {
                const uint32_t w = swz<T>(lbit[b]);
#pragma unroll
                for (int c = 0; c < (1 << b); ++c) so[(1 << b) + c] = so[c] ^ w;
            }
#pragma unroll
            for (int c = 0; c < D; ++c) v[c] = src[so[c]];
        } else {
            // the same per rank: the offset in the part and the rank that holds it, by doubling
            uint32_t so[D], sr[D];
            so[0] = sb;
            sr[0] = rank & ~rk;
#pragma unroll
            for (int b = 0; b < K; ++b) {
                const uint32_t w = swz<T>(lbit[b]), r = op.rbit[b];
#pragma unroll
                for (int c = 0; c < (1 << b); ++c) {
                    so[(1 << b) + c] = so[c] ^ w;
                    sr[(1 << b) + c] = sr[c] | r;
                }
            }
            const uint32_t sbase = uint32_t(__cvta_generic_to_shared(src));
#pragma unroll
            for (int c = 0; c < D; ++c) cl_load(v[c], cl_map(sbase + so[c] * uint32_t(sizeof(A)), sr[c]));
        }
        const uint32_t rows = 1u << lr;
        for (uint32_t i = 0; i < rows; ++i) {
            // local row number -> matrix row (bits of the op's local positions, lowest first) and offset
            uint32_t q = (chunk << lr) | i, row = mine, o = 0;
#pragma unroll
            for (int b = 0; b < K; ++b)
                if (lbit[b]) {
                    if (q & 1u) {
                        row |= 1u << b;
                        o |= lbit[b];
                    }
                    q >>= 1;
                }
            dst[sb ^ swz<T>(o)] = cl_row<D>(msh + row * D, v);
        }
    }
}

template <typename T, int KMAX>
__global__ void __launch_bounds__(kClThreads, 1)
    sweep_cluster_kernel(cplx<T>* __restrict__ sv, const cplx<T>* __restrict__ mats,
                         const __grid_constant__ SweepArgs a, int rbits) {
    using A = typename ClAmp<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ClOp ops[QGB_SWEEP_MAX_OPS];
    const int L = a.sw.low_bits, H = a.sw.n_high, m = L + H, ml = m - rbits, nops = a.sw.n_ops;
    const uint32_t rank = blockIdx.x & ((1u << rbits) - 1u);
    const uint64_t w = blockIdx.x >> rbits;
    const uint32_t part = 1u << ml;
    A* tile = reinterpret_cast<A*>(smem_raw);  // two copies
    A* msh = tile + 2 * size_t(part);          // kClMats matrix entries
    const uint64_t gbase = sweep_tile_base(w, a);
    const cplx<T>* mb = mats + int64_t(w / a.tiles) * a.mat_stride;
    auto offset = [&](uint32_t e) {  // global offset of this part's amplitude e
        const uint32_t u = (rank << ml) | e;
        uint64_t o = u & ((1u << L) - 1u);
        const uint32_t h = u >> L;
        for (int j = 0; j < H; ++j) o |= uint64_t((h >> j) & 1u) << a.sw.high_bits[j];
        return gbase + o;  // (the part's bits are disjoint from the tile's, not from the vector's start)
    };
    if (int(threadIdx.x) < nops) {
        ClOp o;
        const int i = threadIdx.x;
        o.k = a.sw.op_k[i];
        o.taken = o.rk = o.mine = 0;
        o.nl = 0;
        o.moff = 0;
#pragma unroll
        for (int b = 0; b < QGB_MAX_K - 1; ++b) {
            o.lbit[b] = o.rbit[b] = 0;
            if (b < o.k) {
                const int p = a.sw.op_pos[i][o.k - 1 - b];
                if (p < ml) {
                    o.lbit[b] = 1u << p;
                    ++o.nl;
                } else {
                    o.rbit[b] = 1u << (p - ml);
                }
                o.taken |= o.lbit[b];
                o.rk |= o.rbit[b];
                if (rank & o.rbit[b]) o.mine |= 1u << b;
            }
        }
        ops[i] = o;
    }
    for (uint32_t e = threadIdx.x; e < part; e += kClThreads) tile[swz<T>(e)] = cl_in(sv[offset(e)]);
    __syncthreads();
    int cur = 0, staged = 0;
    bool prev = true;  // every CTA of the cluster has started and filled its part before the first remote read
    for (int i = 0; i < nops; ++i) {
        if (i == staged) {  // the matrices of the next ops, as many as fit
            __syncthreads();  // the previous chunk has been used
            int n = 0;
            while (staged < nops) {
                const int dd = 1 << (2 * ops[staged].k);
                if (n + dd > kClMats) break;
                if (threadIdx.x == 0) ops[staged].moff = n;
                n += dd;
                ++staged;
            }
            __syncthreads();
            for (int j = i + int(threadIdx.x >> 5); j < staged; j += kClThreads / 32) {  // a warp per op
                const int dd = 1 << (2 * ops[j].k);
                const cplx<T>* mat = mb + a.sw.op_mat[j];
                A* to = msh + ops[j].moff;
#pragma unroll 2
                for (int e = threadIdx.x & 31; e < dd; e += 32) to[e] = cl_in(__ldg(mat + e));
            }
            __syncthreads();
        }
        const ClOp& op = ops[i];
        const bool x = op.rk != 0;
        // other CTAs' parts are read, or were read by the op that used the copy written now
        if (x || (prev && rbits > 0)) cl_barrier();
        else __syncthreads();
        prev = x;
        const A* src = tile + cur * size_t(part);
        A* dst = tile + (cur ^ 1) * size_t(part);
        const A* mat = msh + op.moff;
        switch (op.k) {
            case 1: cl_op<T, 1>(src, dst, ml, rank, op, mat); break;
            case 2: cl_op<T, 2>(src, dst, ml, rank, op, mat); break;
            case 3: if constexpr (KMAX >= 3) cl_op<T, 3>(src, dst, ml, rank, op, mat); break;
            case 4: if constexpr (KMAX >= 4) cl_op<T, 4>(src, dst, ml, rank, op, mat); break;
            default: if constexpr (KMAX >= 5) cl_op<T, 5>(src, dst, ml, rank, op, mat); break;
        }
        cur ^= 1;
    }
    if (rbits > 0) cl_barrier();  // no CTA leaves while another reads its part
    else __syncthreads();
    const A* last = tile + cur * size_t(part);
    for (uint32_t e = threadIdx.x; e < part; e += kClThreads) sv[offset(e)] = cl_out(last[swz<T>(e)]);
}

}  // namespace qgb

using namespace qgb;

namespace {

// How many clusters of 2^r CTAs, an SM each, the device runs at a time (0: none, or not known), asked once per
// kernel instance and device.
template <typename T, int KMAX>
int cluster_room(int r) {
    auto kern = sweep_cluster_kernel<T, KMAX>;
    static std::atomic<int> known[64][kClMaxRankBits + 1];  // 1 + the answer
    std::atomic<int>& k = known[qgb_host::current_device()][r];
    const int hit = k.load(std::memory_order_relaxed);
    if (hit > 0) return hit - 1;
    int n = 0;
    if (r == 0) {
        n = qgb_host::sm_count();
    } else if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmem) == cudaSuccess &&
               cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1u << r);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = kClSmem;  // one CTA an SM
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 1u << r;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) n = 0;
    }
    if (n <= 0) {
        n = 0;
        cudaGetLastError();  // a size that this device does not take is no error of the caller's
    }
    k.store(1 + n, std::memory_order_relaxed);
    return n;
}

template <typename T, int KMAX>
int launch_cluster(void* sv, const void* mats, const SweepArgs& a, cudaStream_t st) {
    const int m = a.sw.low_bits + a.sw.n_high;
    const uint64_t total = uint64_t(a.batch) * a.tiles;
    // One wave: as many CTAs per tile as leave every cluster an SM per CTA (152 SMs hold 7, 15, 36 and
    // 76 clusters of 16, 8, 4 and 2 CTAs; one too many costs a second wave: 17 qubits complex128,
    // 16 tiles: 8 CTAs 1228 us, 4 CTAs 943 us), each with at least 128 amplitudes
    // (9 qubits complex128: 128 of 4 CTAs 78 us, 256 of 2 CTAs 92 us).
    if (total > uint64_t(cluster_room<T, KMAX>(0))) return qgb_host::QGB_EDECLINE;
    int rbits = 0;
    while (rbits < kClMaxRankBits && m - (rbits + 1) >= 7 && total <= uint64_t(cluster_room<T, KMAX>(rbits + 1))) ++rbits;
    // float32 rows are cheap enough for one CTA to keep up on large parts (20-qubit sweeps of 13-bit
    // tiles: 518 us with 2 CTAs a tile, 467 us with one CTA of sweep.cu; 12 bits alone 177 against
    // 133 us, 11 bits 104 against 113 us); double-float rows are not (2 CTAs 1.8x faster)
    if (sizeof(T) == 4 && rbits < 2 && m - rbits > 11) return qgb_host::QGB_EDECLINE;
    // and so are ops of at most two qubits on small tiles (here / one CTA of sweep.cu: 4 bits 13 / 10 us, 8 bits
    // 25 / 18, 10 bits 35 / 30, 11 bits 40 / 41, 12 bits 51 / 66; of three qubits 8 bits 17 / 25)
    if (sizeof(T) == 4 && KMAX <= 2 && m <= 10) return qgb_host::QGB_EDECLINE;
    const size_t smem = sizeof(typename ClAmp<T>::type) * ((size_t(2) << (m - rbits)) + kClMats);
    if (smem > size_t(kClSmem)) return qgb_host::QGB_EDECLINE;  // the tile twice
    auto kern = sweep_cluster_kernel<T, KMAX>;
    static std::atomic<uint64_t> done{0};
    const int rc = qgb_host::allow_smem(kern, kClSmem, done, "cluster sweep attribute");
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(total << rbits));
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1u << rbits;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (cplx<T>*)sv, (const cplx<T>*)mats, a, rbits);
    if (e == cudaErrorInvalidClusterSize || e == cudaErrorLaunchOutOfResources) {  // nothing was launched
        cudaGetLastError();
        return qgb_host::QGB_EDECLINE;
    }
    return qgb_host::check_launch("cluster sweep");
}

}  // namespace

namespace qgb_host {

int launch_sweep_cluster(int dtype, void* sv, const void* mats, const SweepArgs& a, int kmax, cudaStream_t st) {
    if (dtype == QGB_C64) switch (kmax) {
        case 1:
        case 2: return launch_cluster<float, 2>(sv, mats, a, st);
        case 3: return launch_cluster<float, 3>(sv, mats, a, st);
        case 4: return launch_cluster<float, 4>(sv, mats, a, st);
        case 5: return launch_cluster<float, 5>(sv, mats, a, st);
    } else switch (kmax) {
        case 1:
        case 2: return launch_cluster<double, 2>(sv, mats, a, st);
        case 3: return launch_cluster<double, 3>(sv, mats, a, st);
        case 4: return launch_cluster<double, 4>(sv, mats, a, st);
    }
    return QGB_EDECLINE;
}

}  // namespace qgb_host
