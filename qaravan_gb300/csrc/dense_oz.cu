// Dense 5-qubit blocks of a complex128 state on the 5th-generation tensor cores
// (tcgen05, sm_103a), in fixed point: the digits of both operands are multiplied
// exactly in fp16 and summed exactly in fp32.
//
// Replaces the reference's per-gate `op_action` (tensorQ/statevector_sim.py:124-140)
// for fused blocks of a complex128 statevector. The double-float tile sweeps
// (sweep_df.cu) spend 48 FP32 instructions per complex multiply-add and are bound
// by that pipe; here the data warps only split and reassemble numbers (about 150
// instructions per amplitude and 5-qubit block, against about 1000) and the products
// run on the tensor cores.
//
// Method (error-free splitting for matrix products: Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines of
// matrix multiplication and its applications", Numer. Algorithms 59, 2012). Every group row
// (the 32 amplitudes that differ in the target bits, 64 reals) is scaled by the
// power of two of its largest component to integers of up to 50 bits, the
// operator to 51 bits, and each integer is written in 6 signed digits of 9 bits,
// base 512, |digit| <= 256: exact in fp16. The product of digits i and j of two rows,
// summed over 64 reals, is below 2^22, so the sums of all digit pairs with the same
// i + j = s are exact in one fp32 accumulator for s <= 3; for s = 4 to 6, whose weight is
// 2^-36 and less, fp32 rounding does not matter, and pairs with i + j >= 7 (2^-55 of
// the row) are dropped (with those of 6 dropped too the error was 2e-14 a block). 26
// digit pairs; a digit of the state meets the operator's digits side by side, N = 224
// down to 64 columns, so 4096 amplitudes take 48 MMAs (one pair at a time, N = 64,
// the tensor pipe idled half of each). The seven accumulators are reassembled in a 64-bit integer and rounded to float64 by integer
// instructions (the FP64 pipe would cost more than the products). Errors are
// relative to the row's largest component, about 2^-50: against 64-bit arithmetic
// 1.1e-15 to 1.5e-15 of the norm per block, and 7.1e-15 after a 24-qubit circuit of depth 5 where
// the double-float sweeps leave 4.9e-14.
//
// Small amplitudes. An error relative to the row's largest component M is worse than
// double-float's, which is relative to B_i = sum_j |U_ij| |x_j| of the output, wherever
// B_i is much smaller than M: phases, permutations, small rotations beside a large
// amplitude. So an output is left to the products only when B_i >= M / 32 is certain
// (one product |U_ij| |x_j| of M / 32, or four of M / 128, by bit masks of the entries of
// at least 1/16, 1/8, 1/4 and of the components within 1, 2, 3 binades of M), or, in a row of at most
// 8 components that all lie within 3 binades, when one product of M / 128 is (what is
// rounded is then as large as what is summed). The other outputs are formed in
// double-float from the staged tile, the products with nonzero entries of the block only,
// as the tile sweeps form them (sweep_df.cu), while the MMAs run. The certificate costs 6 % of a
// pass; recomputed outputs, in passes that meet product-like rows and in narrow blocks, up to the
// pass once more: 25 qubits depth 8 17.8 ms without either, 18.9 with the certificate, 22.1 in all
// (20.3 with the last narrow blocks in a tile sweep, compiler._narrow_tail).
//
// Data path per CTA (one per SM, 16 warps): a tile is 4096 amplitudes (64 KB: the 5
// target bits and the 7 lowest others), copied by cp.async one tile ahead; four
// warps share a lane quarter's rows, 8 components each; digits go to shared memory
// as K-major core matrices (96 KB), where both operands are read by the MMAs; results
// come back through that space for coalesced stores, or go straight to memory where a thread's
// rows are runs of 128 bytes (no target among the three lowest bits: 19.2 to 17.8 ms at 25 qubits).
// What bounds it: the integer instructions that split and reassemble (24 qubits: ALU pipe 60 % busy, 2660
// instructions a warp and tile of 20,100 cycles); the products (tensor pipe 17 %, the first half
// overlapped with nothing) come next, memory (20 %) last: the seven accumulators fill tensor memory, so
// two tiles cannot be in flight.
// Measured, brickwork against the double-float sweeps: 17 qubits depth 20 1.00 to 0.80 ms, 20 qubits
// depth 20 3.49 to 1.89 ms, 22 qubits depth 8 6.20 to 2.79 ms, 25 qubits depth 8 48.4 to 20.3 ms.
#include "sweep_df.cuh"
#include "tc_common.cuh"

namespace qgb {

__device__ int g_oz_status = 0;

constexpr int kOzK = 5, kOzD = 32, kOzR = 64;   // components, reals per group row
constexpr int kOzTileBits = 12, kOzTile = 1 << kOzTileBits;
constexpr int kOzThreads = 512;
constexpr int kOzDigits = 6;
constexpr int kOzSums = 7;                      // digit pairs i + j = 0 .. 6, an accumulator each
constexpr int kOzXBytes = 128 * kOzR * 2;       // one digit of 128 rows
constexpr int kOzHalf = kOzR / 2;               // output columns of half the components
constexpr int kOzWRows = kOzSums * kOzHalf;     // B rows of a half: the digits one after the other, then zeros
constexpr int kOzWBytes = kOzWRows * kOzR * 2;  // the operator's digits for one half
constexpr size_t kOzSmem = size_t(kOzDigits) * kOzXBytes + 2 * kOzWBytes + sizeof(double2) * kOzTile +
                           sizeof(double2) * kOzThreads + 128;
// kind::f16, fp32 accumulator, K-major fp16 operands, M = 128, N columns
__host__ __device__ constexpr uint32_t oz_idesc(int n) {
    return (1u << 4) | (uint32_t(n >> 3) << 17) | (uint32_t(128 >> 4) << 24);
}
constexpr unsigned long long kOzBias = 256ull | 256ull << 9 | 256ull << 18 | 256ull << 27 | 256ull << 36 | 256ull << 45;

struct OzArgs {
    int tile_bits[kOzTileBits];  // global bit of each tile bit, ascending
    int pos_g[7];                // tile positions of the group bits, ascending
    int pos_t[kOzK];             // tile positions of the target bits, ascending
    int perm_in[kOzD], perm_out[kOzD];  // memory-order component -> matrix column / row
    uint64_t tiles;
    int reverse;
    int direct;                  // no target among the three lowest bits: rows are written straight from registers
};

// The certificate (see above): this many products of entries of at least 1/16 and components of at least 1/8
// of the row's largest (2 binades); one where the row has at most 8 components, all that large.
constexpr int kOzNear = 2, kOzCount = 4, kOzSparse = 8;

// 16-byte element swizzle of the staged tile (linear over XOR).
__host__ __device__ __forceinline__ uint32_t oz_swz(uint32_t e) { return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u); }

// round(|x| 2^(bits - (emax - 1022))) with x's sign, biased so that all base-512 digits are
// non-negative fields; emax >= x's biased exponent.
__device__ __forceinline__ unsigned long long oz_fixed(double x, int emax, int bits) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = int((b >> 52) & 0x7ff);
    unsigned long long m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const int sh = emax - E + 53 - bits;  // >= 1
    m = E == 0 || sh > 60 ? 0ull : ((m >> (sh - 1)) + 1ull) >> 1;
    return kOzBias + (((long long)b) < 0 ? 0ull - m : m);
}

// Digit i (0: most significant) of two fields as packed fp16 integers in [-256, 255].
__device__ __forceinline__ uint32_t oz_digits(unsigned long long re, unsigned long long im, int i) {
    const int s = 9 * (kOzDigits - 1 - i);
    const uint32_t a = uint32_t(re >> s), c = uint32_t(im >> s);
    const uint32_t f = (__byte_perm(a, c, 0x5410) & 0x01ff01ffu) | 0x64006400u;  // 1024 + field
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&f), __floats2half2_rn(1280.f, 1280.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// v = sum_s acc_s 512^(5 - s) as a float64 scaled so that a v of bit length 64 gets the biased exponent e.
// The shifts wrap modulo 2^64; the sum itself stays below 2^62.
__device__ __forceinline__ double oz_join(const float* a, int e) {
    const int a0 = __float2int_rn(a[0]), a1 = __float2int_rn(a[1]), a2 = __float2int_rn(a[2]), a3 = __float2int_rn(a[3]);
    const int a4 = __float2int_rn(a[4]), a5 = __float2int_rn(fmaf(a[6], 1.f / 512.f, a[5]));
    long long v = ((long long)a2 << 27) + ((long long)a3 << 18) + ((long long)a4 << 9) + a5;
    v += (long long)((unsigned long long)(uint32_t(a0) << 13) << 32) + ((long long)a1 << 36);
    const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ull;
    unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    if (m == 0) return 0.0;
    const int lz = __clzll((long long)m);
    m <<= lz;                                      // leading bit at 63
    m = (m >> 11) + ((m >> 10) & 1ull);            // 53 bits, half up; a carry moves into the exponent below
    const int ex = e - lz;
    if (ex <= 0) return __longlong_as_double((long long)sign);
    const unsigned long long r = ((unsigned long long)(ex - 1) << 52) + m;  // the implicit bit adds 1 to ex - 1
    return ex >= 0x7ff ? __longlong_as_double((long long)(sign | 0x7ff0000000000000ull)) : __longlong_as_double((long long)(sign | r));
}

__device__ __forceinline__ void oz_ld8(uint32_t taddr, float (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// The loaded registers are valid only after the wait: tying them to it keeps every use behind it.
__device__ __forceinline__ void oz_ld_wait(float (&r)[kOzSums][8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int s = 0; s < kOzSums; ++s)
#pragma unroll
        for (int j = 0; j < 8; ++j) asm volatile("" : "+f"(r[s][j]));
}

__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0; "
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// The outputs of one row in `unsure` (bit c: output 8 h + c) in double-float, as the tile sweeps form
// them: the products with the nonzero entries of the block's row, in order. Called by whole warps, a row
// per lane; tile: the staged tile in double-float, scaled by 2^(896 - bias) a row; urow: the warp's 32 entries.
__device__ __noinline__ void oz_redo(double2 (&v)[8], uint32_t unsure, int bias, const double2* __restrict__ op,
                                     const dfc* tile, uint32_t row, const uint32_t* toff, dfc* urow, const OzArgs& a,
                                     int h, int lane) {
    const double scale = __hiloint2double((bias + 127) << 20, 0);  // 2^(bias - 896)
    uint32_t todo = __reduce_or_sync(0xffffffffu, unsure);
    while (todo) {
        const int c = __ffs(todo) - 1;
        todo &= todo - 1;
        const double2 u = op[a.perm_out[8 * h + c] * kOzD + a.perm_in[lane]];
        dfc m;
        df_split(u.x, m.rh, m.rl);
        df_split(u.y, m.ih, m.il);
        urow[lane] = m;
        uint32_t nz = __ballot_sync(0xffffffffu, u.x != 0.0 || u.y != 0.0);
        __syncwarp();
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        dfc w = {0.f, 0.f, 0.f, 0.f}, y = w;
        while (nz) {  // an entry's loads ahead of the previous one's product
            const int j = __ffs(nz) - 1;
            nz &= nz - 1;
            const dfc wj = urow[j], yj = tile[row ^ toff[j]];
            dfc_mac(s, w, y);
            w = wj;
            y = yj;
        }
        dfc_mac(s, w, y);
        __syncwarp();
        const dfc r = dfc_finish(s);
        v[c] = make_double2(df_join(r.rh, r.rl) * scale, df_join(r.ih, r.il) * scale);
    }
}

__global__ void __launch_bounds__(kOzThreads, 1) dense_oz_kernel(double2* __restrict__ sv, const double2* __restrict__ op,
                                                                 const __grid_constant__ OzArgs a) {
    extern __shared__ unsigned char oz_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(oz_smem_raw) + 127) & ~uintptr_t(127));
    unsigned char* W = base;                                // [half][b_off(digit * 32 + n, k, kOzWRows)]
    unsigned char* X = W + 2 * kOzWBytes;                   // [digit][b_off(row, k, 128)]
    double2* tile = reinterpret_cast<double2*>(X + kOzDigits * kOzXBytes);
    dfc* urow = reinterpret_cast<dfc*>(tile + kOzTile) + (threadIdx.x & ~31u);  // the warp's row of the block (oz_redo)
    double2* out = reinterpret_cast<double2*>(X);           // the results, once the MMAs have read the digits
    __shared__ __align__(8) uint64_t done[2];  // the accumulators of a half are complete
    __shared__ uint32_t tmem_slot;
    __shared__ int wexp;
    __shared__ uint32_t row_exp[4][128];               // a thread's largest exponent and how far below it its components are
    __shared__ __align__(16) uint32_t heavy[3][kOzD];  // bit j: entry (i, j) of the block is at least 1/16, 1/8, 1/4, memory order
    __shared__ uint32_t toff[kOzD];                    // component -> its offset in the staged tile
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, h = warp >> 2;  // lane quarter, quarter of the components
    const int rown = 32 * q + lane;

    // ---- operator digits
    if (tid == 0) wexp = 0;
    if (tid < 3 * kOzD) heavy[tid / kOzD][tid % kOzD] = 0;
    __syncthreads();
    {
        double2 v[2];
        int e = 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int w = tid + t * kOzThreads, i = w & 31, j = w >> 5;
            v[t] = op[a.perm_out[i] * kOzD + a.perm_in[j]];
            e = max(e, max((__double2hiint(v[t].x) >> 20) & 0x7ff, (__double2hiint(v[t].y) >> 20) & 0x7ff));
            const float a1 = fabsf(float(v[t].x)) + fabsf(float(v[t].y));  // up to sqrt(2) times the entry
#pragma unroll
            for (int l = 0; l < 3; ++l)
                if (a1 >= 0.08838835f * float(1 << l)) atomicOr(&heavy[l][i], 1u << j);  // sqrt(2) / 16, ..
        }
        atomicMax(&wexp, e);
        __syncthreads();
        e = wexp;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int w = tid + t * kOzThreads, i = w & 31, j = w >> 5;
            const unsigned long long re = oz_fixed(v[t].x, e, 51), im = oz_fixed(v[t].y, e, 51), ni = 2 * kOzBias - im;
#pragma unroll
            for (int d = 0; d < kOzSums; ++d) {  // real rows 2i (Mr, -Mi) and 2i + 1 (Mi, Mr)
                unsigned char* w0 = W + (i >> 4) * kOzWBytes;
                const int n = d * kOzHalf + 2 * (i & 15);
                *reinterpret_cast<uint32_t*>(w0 + b_off(n, 2 * j, kOzWRows)) = d < kOzDigits ? oz_digits(re, ni, d) : 0u;
                *reinterpret_cast<uint32_t*>(w0 + b_off(n + 1, 2 * j, kOzWRows)) = d < kOzDigits ? oz_digits(im, re, d) : 0u;
            }
        }
    }
    const int we = wexp;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc_smem_u32(&tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        for (int p = 0; p < 2; ++p)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem_u32(&done[p])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // the state is touched from here on; the operator was read before (see dense_tc_kernel)
    tc_grid_wait();
    tc_grid_next();

    const uint64_t ntiles = (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;
    const uint64_t t0 = a.reverse ? a.tiles - 1 - blockIdx.x : blockIdx.x;
    const uint64_t step = a.reverse ? 0 - uint64_t(gridDim.x) : uint64_t(gridDim.x);
    // copies: tile index tid + 512 m
    uint64_t cbase = 0, cm[3];
#pragma unroll
    for (int j = 0; j < 9; ++j) cbase |= uint64_t((tid >> j) & 1) << a.tile_bits[j];
#pragma unroll
    for (int j = 0; j < 3; ++j) cm[j] = uint64_t(1) << a.tile_bits[9 + j];
    auto coff = [&](int m) { return cbase | (m & 1 ? cm[0] : 0) | (m & 2 ? cm[1] : 0) | (m & 4 ? cm[2] : 0); };
    auto load = [&](uint64_t t) {
        const double2* s = sv + insert_zeros(t, a.tile_bits, kOzTileBits);
#pragma unroll
        for (int m = 0; m < 8; ++m) cp_async16(tc_smem_u32(tile + oz_swz(uint32_t(tid + 512 * m))), s + coff(m));
        cp_async_commit();
    };
    // this thread's components: row `rown`, memory-order components 8 h .. 8 h + 7
    uint32_t su = 0;
#pragma unroll
    for (int j = 0; j < 7; ++j) su |= uint32_t((rown >> j) & 1) << a.pos_g[j];
    su |= uint32_t(h & 1) << a.pos_t[3] | uint32_t(h >> 1) << a.pos_t[4];
    su = oz_swz(su);
    if (tid < kOzD) {
        uint32_t o = 0;
#pragma unroll
        for (int j = 0; j < kOzK; ++j) o |= uint32_t((tid >> j) & 1) << a.pos_t[j];
        toff[tid] = oz_swz(o);
    }
    const uint32_t t1 = oz_swz(1u << a.pos_t[0]), t2 = oz_swz(1u << a.pos_t[1]), t4 = oz_swz(1u << a.pos_t[2]);
    auto at = [&](int c) { return su ^ (c & 1 ? t1 : 0u) ^ (c & 2 ? t2 : 0u) ^ (c & 4 ? t4 : 0u); };
    uint64_t gr = 0;  // and their global offsets
#pragma unroll
    for (int j = 0; j < 7; ++j) gr |= uint64_t((rown >> j) & 1) << a.tile_bits[a.pos_g[j]];
    gr |= uint64_t(h & 1) << a.tile_bits[a.pos_t[3]] | uint64_t(h >> 1) << a.tile_bits[a.pos_t[4]];
    const uint64_t g1 = uint64_t(1) << a.tile_bits[a.pos_t[0]], g2 = uint64_t(1) << a.tile_bits[a.pos_t[1]],
                   g4 = uint64_t(1) << a.tile_bits[a.pos_t[2]];
    const uint32_t wd = tc_smem_u32(W), xd = tc_smem_u32(X);
    bool fail = false;
    load(t0);
    for (uint64_t k = 0; k < ntiles; ++k) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // the tile has landed; the previous tile's products have read the digits, and its results have left their space
        if (__syncthreads_or(fail)) break;
        double2 v[8];
        int e = 0;
        {
            int ec[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                v[c] = tile[at(c)];
                ec[c] = max((__double2hiint(v[c].x) >> 20) & 0x7ff, (__double2hiint(v[c].y) >> 20) & 0x7ff);
                e = max(e, ec[c]);
            }
            uint32_t code = uint32_t(e) << 16;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t d = uint32_t(min(e - ec[c], 3));
                code |= (d & 1u) << c | (d >> 1) << (8 + c);
                if (ec[c] > 0 && d == 3) code |= 1u << 31;
            }
            row_exp[h][rown] = code;
        }
        __syncthreads();
        uint32_t unsure = 0;  // bit c: this thread's output c is not certified
        {
            uint32_t code[4], near[3] = {0, 0, 0};  // bit j: component j of the row is at least 1/2, 1/4, 1/8 of the largest
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                code[p] = row_exp[p][rown];
                e = max(e, int((code[p] >> 16) & 0x7ffu));
            }
            bool rest = false;  // the row has other components
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int ep = int((code[p] >> 16) & 0x7ffu), left = kOzNear - (e - ep);  // binades below that still count
                const uint32_t d0 = code[p], d1 = code[p] >> 8, three = ~(d0 & d1);
                const uint32_t upto[3] = {~(d0 | d1), ~d1, three};  // components at most 0, 1, 2 binades below the thread's largest
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const int b = left - (2 - l);
                    near[l] |= ((b < 0 ? 0u : b == 0 ? upto[0] : b == 1 ? upto[1] : upto[2]) & 0xffu) << (8 * p);
                }
                rest |= ep > 0 && ((code[p] >> 31) != 0 || (three & ~(near[2] >> (8 * p)) & 0xffu) != 0);
            }
            // B >= M / 32: one product of 1/32, or kOzCount of 1/128 (sparse rows: see above)
            const int want = !rest && __popc(near[2]) <= kOzSparse ? 1 : kOzCount;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t h16 = heavy[0][8 * h + c], h8 = heavy[1][8 * h + c], h4 = heavy[2][8 * h + c];
                const uint32_t one = (h16 & near[0]) | (h8 & near[1]) | (h4 & near[2]);
                unsure |= uint32_t(one == 0 && __popc(near[2] & h16) < want) << c;
            }
            if (e == 0 || e == 0x7ff || we == 0x7ff) unsure = 0;  // zeros, and rows that become NaN
        }
#pragma unroll
        for (int c0 = 0; c0 < 8; c0 += 4) {  // 4 components: 8 fp16 of one core-matrix row
            uint32_t w[kOzDigits][4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const unsigned long long re = oz_fixed(v[c0 + c].x, e, 50), im = oz_fixed(v[c0 + c].y, e, 50);
#pragma unroll
                for (int d = 0; d < kOzDigits; ++d) w[d][c] = oz_digits(re, im, d);
            }
            const uint32_t o = b_off(rown, 16 * h + 2 * c0, 128);
#pragma unroll
            for (int d = 0; d < kOzDigits; ++d)
                *reinterpret_cast<uint4*>(X + d * kOzXBytes + o) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        const bool redo = __syncthreads_or(unsure);
        tc_fence_after();
        if (warp == 0) {
            if (lane == 0) {
                // X digit i times the W digits j = 0 .. 6 - i side by side: sums i .. 6 (digit 0 reaches the zero
                // rows, which clear the last sum)
                for (int p = 0; p < 2; ++p) {
#pragma unroll
                    for (int i = 0; i < kOzDigits; ++i)
#pragma unroll
                        for (int ks = 0; ks < kOzR / 16; ++ks)
                            oz_mma(tmem + uint32_t(p * kOzWRows + i * kOzHalf),
                                   b_desc(xd + uint32_t(i * kOzXBytes + ks * 128 * 32)),
                                   b_desc(wd + uint32_t(p * kOzWBytes + ks * kOzWRows * 32)),
                                   oz_idesc((kOzSums - i) * kOzHalf), i > 0 || ks > 0);
                    tc_commit(tc_smem_u32(&done[p]));
                }
            }
            __syncwarp();
        }
        if (redo) {  // (every thread has read its components: the tile is converted in place)
            const int bias = max(e - 127, 1);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                dfc y;
                df_split(v[c].x, y.rh, y.rl, bias);
                df_split(v[c].y, y.ih, y.il, bias);
                reinterpret_cast<dfc*>(tile)[at(c)] = y;
            }
            __syncthreads();
            double2 w[8];  // (the callee's argument lives in memory; v stays in registers)
            oz_redo(w, unsure, bias, op, reinterpret_cast<const dfc*>(tile), su ^ (h & 1 ? toff[8] : 0u) ^ (h & 2 ? toff[16] : 0u),
                    toff, urow, a, h, lane);
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = w[c];
            __syncthreads();
        }
        if (k + 1 < ntiles) load(t0 + (k + 1) * step);  // the tile's space is free
        if (!tc_wait_bounded(tc_smem_u32(&done[h >> 1]), uint32_t(k & 1))) {
            fail = true;
            if (lane == 0) atomicExch(&g_oz_status, 1);
        }
        tc_fence_after();
        // ---- results: 16 reals of this row, from the seven accumulators (the first half's while the second's
        // products run)
        // x = x_int 2^(e - 1072), w = w_int 2^(we - 1073) and the integer counts 2^45: a leading bit at 63
        // is worth 2^(e + we - 2037); rows or operators that are not finite give NaN
        const bool bad = e == 0x7ff || we == 0x7ff;
        const int ey = e + we - 1014;
#pragma unroll
        for (int c0 = 0; c0 < 8; c0 += 4) {
            float r[kOzSums][8];
#pragma unroll
            for (int s = 0; s < kOzSums; ++s)
                oz_ld8(tmem + (uint32_t(32 * q) << 16) + uint32_t((h >> 1) * kOzWRows + s * kOzHalf + 16 * (h & 1) + 2 * c0), r[s]);
            oz_ld_wait(r);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float x[kOzSums], y[kOzSums];
#pragma unroll
                for (int s = 0; s < kOzSums; ++s) {
                    x[s] = r[s][2 * c];
                    y[s] = r[s][2 * c + 1];
                }
                if (!((unsure >> (c0 + c)) & 1u)) v[c0 + c] = make_double2(oz_join(x, ey), oz_join(y, ey));
                if (bad)
                    v[c0 + c] = make_double2(__longlong_as_double(0x7ff8000000000000ll), __longlong_as_double(0x7ff8000000000000ll));
            }
        }
        tc_fence_before();
        double2* s = sv + insert_zeros(t0 + k * step, a.tile_bits, kOzTileBits);
        if (a.direct) {
            s += gr;
#pragma unroll
            for (int c = 0; c < 8; ++c) s[(c & 1 ? g1 : 0) | (c & 2 ? g2 : 0) | (c & 4 ? g4 : 0)] = v[c];
            continue;
        }
        __syncthreads();  // both halves' MMAs have read the digits
#pragma unroll
        for (int c = 0; c < 8; ++c) out[at(c)] = v[c];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 8; ++m) s[coff(m)] = out[oz_swz(uint32_t(tid + 512 * m))];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

}  // namespace qgb

using namespace qgb;

namespace qgb_host {

int oz_status_read_clear() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, qgb::g_oz_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) {
        const int z = 0;
        cudaMemcpyToSymbol(qgb::g_oz_status, &z, sizeof(int));
    }
    return v;
}

// Fixed-point tensor-core path for a complex128 block on five bits; QGB_EDECLINE (nothing touched) for any
// other op. Only blocks the caller knows to be unitary: their outputs are as large as their inputs, so
// errors relative to the row are errors relative to the result.
int try_dense_oz(void* sv, const void* op, int nbits, const int* sorted, const int* in_bits, const int* out_bits, int k,
                 int64_t batch, cudaStream_t st, const DensePass& pass) {
    if (k != kOzK || nbits < kOzTileBits || batch != 1 || !pass.fixed || pass.scale) return QGB_EDECLINE;
    if (qgb_get_dense_impl() == 0) return QGB_EDECLINE;
    OzArgs a{};
    int nt = 0, ng = 0, ti = 0;
    for (int b = 0; b < nbits && ti < kOzTileBits; ++b) {
        bool is_t = false;
        for (int j = 0; j < k; ++j) is_t |= sorted[j] == b;
        if (is_t) {
            a.pos_t[nt++] = ti;
            a.tile_bits[ti++] = b;
        } else if (ng < 7) {
            a.pos_g[ng++] = ti;
            a.tile_bits[ti++] = b;
        }
    }
    if (ti != kOzTileBits || nt != k || ng != 7) return QGB_EDECLINE;
    for (int i = 0; i < k; ++i) {
        int ci = 0, co = 0;
        for (int j = 0; j < k; ++j) {
            if (in_bits[j] == sorted[i]) ci = 1 << (k - 1 - j);
            if (out_bits[j] == sorted[i]) co = 1 << (k - 1 - j);
        }
        for (int j = 0; j < (1 << i); ++j) {
            a.perm_in[j | (1 << i)] = a.perm_in[j] | ci;
            a.perm_out[j | (1 << i)] = a.perm_out[j] | co;
        }
    }
    a.tiles = uint64_t(1) << (nbits - kOzTileBits);
    a.direct = a.pos_t[0] >= 3;
    a.reverse = pass.reverse && a.tiles <= 4096;  // states of up to 256 MB, as dense_tc_kernel
    static std::atomic<uint64_t> done{0};
    const int rc = allow_smem(dense_oz_kernel, kOzSmem, done, "dense_oz attribute");
    if (rc) return rc;
    const uint64_t cap = uint64_t(sm_count());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(a.tiles < cap ? a.tiles : cap));
    cfg.blockDim = dim3(kOzThreads);
    cfg.dynamicSmemBytes = kOzSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pass.early && a.tiles <= 1024 ? 1 : 0;  // while the state fits L2, as dense_tc_kernel
    cudaLaunchKernelEx(&cfg, dense_oz_kernel, (double2*)sv, (const double2*)op, a);
    if (pass.tensor) *pass.tensor = 1;
    return check_launch("dense_oz kernel");
}

}  // namespace qgb_host
