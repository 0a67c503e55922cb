// Tensor-core row engine (sm_100a: tcgen05 MMA, column FFTs in tensor memory).
//
// Same transform as the CUDA-core engine (fcwt_kernels.cu): the daughter
// product of the reference (src/fcwt/fcwt.cpp:197-311), the inverse FFT
// (fcwt.cpp:418-429), the normalisation (fcwt.cpp:431-445) and the crop to n
// (fcwt.cpp:396-416). Of a row of padded length N' (N, or N / D for a row
// decimated in time by D: keeping every D-th sample folds the spectrum to
// N' bins) with P2 = 16 R (R = 16, or 8 for N' <= 16384), M = N' / P2 columns,
//     t = c + M a        (c < M, a = a1 + R a2, a1 < R, a2 < 16)
//     q = L + k2 + P2 k1 (L a multiple of P2, k2 = kl + 16 kb, k1 < KC <= 64)
// the inverse transform is
//     G[c][k2]  = sum_{k1} w_M^{k1 c} Z[L + k2 + P2 k1]                  (GEMM)
//     X[kl][a1] = w_N'^{(L + kl) c} sum_{kb} G[c][kl + 16 kb] (w_N'^{16 c} w_R^{a1})^kb   (pass 1)
//     y[t]      = sum_{kl} X[kl][a1] (w_P2^{a1} w_16^{a2})^kl             (pass 2)
// (w_X = exp(+2 pi i / X), Z = spectrum x daughter weights x 1/N).
//
// The GEMM runs on the tensor cores with M = 128 columns c as its rows, so the
// accumulator lane of tensor memory is the column c and its 2 P2 accumulator
// columns are Re and Im of G[c][.]: a thread owns a column and runs the column's
// whole P2-point DFT on data of its own lane. The exchange between the two
// passes goes through tensor memory in place; a warp's stores are 32 consecutive
// samples (any n, any alignment of the row). No shared-memory transposes, output
// staging or CTA barriers inside a tile: only the two warps of a lane quadrant
// meet between the passes. With columns along the MMA's N (G and output tiles
// through shared memory, half-CTA barriers) the engine issued 61 instructions
// per point and took 1.12 ms for 3000 rows of 100,000 samples; this one issues
// 32 and takes 0.76 ms.
//
// A CTA has 8 column warps (two per quadrant: the DFTs and stores) and 8
// producer warps (the next row's Z, the MMA issue, the queue). What bounds it,
// 3000 x 100,000 complex64, cycles per row of a CTA: 72,000 in all, of which
// pass 1 23,000 (FP32 pipe, 15 clocks per point and warp), pass 2 31,000 (the
// SM's store path, 32 bytes per clock: 25,000 for the row's 800 KB), Z of rows
// with KC = 64 about 4,000 and the first MMAs of a tile 3,000.
//
// Precision: split FP16 (hi + lo, products hi hi + lo hi + hi lo, FP32
// accumulation, about 2^-21 relative per element); Z of a row is scaled by 2^e
// (max |Z| 2^e in [2^14, 2^15)); both DFT passes are FP32 for every output type.
//
// Operands. A = the DFT matrix w_M^{k1 c} of 128 columns (Re and Im parts, hi
// and lo), K-major in shared memory; it does not depend on the row. Tile T holds
// columns c = 128 T + lane of NT = M / 128 tiles. With T = b + (NT / 4) j,
// w_M^{k1 c} = w_M^{k1 (lane + 128 b)} i^{k1 j}: the quarter-turn factor of a
// residue class of k1 mod 4 is a choice of Re or Im part and sign, so one matrix
// A_b serves four tiles. The MMA's K step of 16 must share that factor:
//     KC = 64: step r holds k1 = r + 4 s;
//     KC = 32: step r holds k1 = r + 4 s and r + 2 + 4 s, and A has two versions
//              (j odd: the second half negated);
//     KC = 16: one step, and A has four versions (one per j).
// All three take 64 K columns of A. B = Z (Re, Im, hi, lo) as [k2][k1], K-major,
// rows in the order n = kl R + kb, so that a thread's kb values are consecutive
// accumulator columns.
#include <initializer_list>

#include "fcwt_dev.cuh"

namespace fcwt {
namespace dev {

constexpr int kTcColThreads = 256;                  // column warps: 2 per lane quadrant
constexpr int kTcProdThreads = 256;                 // producer warps: pre-pass, MMA issue, queue
constexpr int kTcThreads = kTcColThreads + kTcProdThreads;
// Registers: 128 per thread at launch (2 x 2 warpgroups), moved from the
// producers to the column warps: 2 x 168 + 2 x 88 = 4 x 128.
constexpr int kTcColRegs = 168, kTcProdRegs = 88;
constexpr int kTcSlots = 8;                         // unit descriptors in flight
constexpr int kTcTmemCols = 512;
constexpr int kTcTwhiSmem = 512;  // w_M table kept in SMEM when N / 1024 <= this

constexpr int kTcAArray = 128 * kTcMaxKc * 2;       // one of the four A arrays, 16 KB
constexpr int kTcZBytes = 4 * 256 * kTcMaxKc * 2;   // Z of the widest window, 128 KB
constexpr int kTcOffZ = 4 * kTcAArray;
constexpr int kTcColBytes = 4 * 128 * 4 * 8;        // pass-1 twiddles of four tiles, 16 KB
constexpr int kTcS2Bytes = 8 * 8 * 16;                // pass-2 twiddles: R / 2 pairs of a1 x 8
constexpr int kTcTabBytes = 4 * kTcAArray + kTcColBytes + kTcS2Bytes;  // one operand table in global memory
constexpr int kTcOffCol = kTcOffZ + kTcZBytes;
constexpr int kTcOffS2 = kTcOffCol + kTcColBytes;  // (right behind, as in the table)
constexpr int kTcOffTwlo = kTcOffS2 + kTcS2Bytes;
constexpr int kTcOffTwhi = kTcOffTwlo + (kP2 + kP2 / 16) * 8;
constexpr int kTcOffEnd = kTcOffTwhi + kTcTwhiSmem * 8;
constexpr size_t kTcSmemBytes = (size_t)kTcOffEnd + 1024;
static_assert(kTcSmemBytes <= 227 * 1024 - 3072, "tensor-core engine fits one CTA's shared memory");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major without swizzle: core matrices of
// 8 rows x 16 bytes; lbo = byte distance between core matrices along K, 128
// bytes between 8-row groups. The low word holds address and lbo, the high word
// is the same for all operands here.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr, uint32_t lbo) {
    return ((saddr >> 4) & 0x3FFFu) | (((lbo >> 4) & 0x3FFFu) << 16);
}
constexpr uint32_t kUmmaDescHi = (128u >> 4) | (1u << 14);
// Instruction descriptor: D f32, A/B f16, both K-major, M = 128, N = n; neg
// negates A.
__device__ __forceinline__ uint32_t umma_idesc(int n, uint32_t neg) {
    return (1u << 4) | (neg << 13) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint32_t adesc_lo, uint32_t bdesc_lo, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}\n" ::"r"(d),
        "r"(adesc_lo), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi));
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// tcgen05.wait::ld with registers of the loads it completes as operands, so
// that no read of them can be placed before the wait.
template <int C>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[C]) {
    static_assert(C % 16 == 0, "");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < C; i += 16)
        asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]),
                     "+r"(r[i + 6]), "+r"(r[i + 7]), "+r"(r[i + 8]), "+r"(r[i + 9]), "+r"(r[i + 10]),
                     "+r"(r[i + 11]), "+r"(r[i + 12]), "+r"(r[i + 13]), "+r"(r[i + 14]), "+r"(r[i + 15])
                     :
                     : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
            taddr),
        "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]),
        "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "f"(r[0]),
                 "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7])
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
// Bounded wait for phase `parity` of an mbarrier (gives up after
// kWaitLimitNs, recording kErrWaitTimeout). The tries run in a loop of four
// instructions, and the clock is read once per kTries of them, so that waiting
// warps take few issue slots from the working ones.
constexpr uint32_t kTries = 256;
__device__ __forceinline__ uint32_t mbar_try(uint32_t mbar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 c;\n\tmov.u32 c, 0;\n"
        "T%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra D%=;\n\t"
        "add.u32 c, c, 1;\n\tsetp.lt.u32 q, c, %3;\n\t@q bra T%=;\n"
        "D%=:\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity), "n"(kTries)
        : "memory");
    return done;
}
__device__ __forceinline__ void mbar_wait_slow(uint32_t mbar, uint32_t parity, int* err) {
    const unsigned long long t0 = global_ns();
    while (!mbar_try(mbar, parity)) {
        if (global_ns() - t0 > kWaitLimitNs) {
            *(volatile int*)err = *(volatile int*)err | kErrWaitTimeout;  // (may be host memory: no atomics)
            return;
        }
    }
}
__device__ __forceinline__ void mbar_wait(uint32_t mbar, uint32_t parity, int* err) {
    if (!mbar_try(mbar, parity)) mbar_wait_slow(mbar, parity, err);
}

__device__ __forceinline__ uint32_t h2bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// ---- packed pairs of floats (fma.rn.f32x2: two FMAs in one issue slot)
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float x, float y) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ f2 pku(uint32_t x, uint32_t y) { return pk(__uint_as_float(x), __uint_as_float(y)); }
__device__ __forceinline__ void unpk(f2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f2 neg2(f2 v) {
    float x, y;
    unpk(v, x, y);
    return pk(-x, -y);
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
struct Cx {
    f2 x, y;
};
__device__ __forceinline__ Cx dup(float2 w) { return {pk(w.x, w.x), pk(w.y, w.y)}; }
__device__ __forceinline__ Cx cmulx(const Cx& a, const Cx& w) {
    return {fma2(a.y, neg2(w.y), mul2(a.x, w.x)), fma2(a.y, w.x, mul2(a.x, w.y))};
}
// (a, b) <- (a + w b, -(a - w b)), w taken times i when ROT: six packed FMAs, the
// second output as (a + w b) - 2 a. Packed operands take no free sign, so the
// negated output is kept: after the stages up to length LEN element i carries
// the sign (-1)^popcount(i mod LEN), equal for both inputs of the next
// stage's butterflies, which is why w needs no sign of its own.
template <bool ROT>
__device__ __forceinline__ void bfly(Cx& a, Cx& b, const Cx& w) {
    f2 tx, ty;
    const f2 m2 = pk(-2.0f, -2.0f);
    if constexpr (!ROT) {
        tx = fma2(b.x, w.x, a.x);
        tx = fma2(b.y, neg2(w.y), tx);
        ty = fma2(b.y, w.x, a.y);
        ty = fma2(b.x, w.y, ty);
    } else {
        tx = fma2(b.x, neg2(w.y), a.x);
        tx = fma2(b.y, neg2(w.x), tx);
        ty = fma2(b.y, neg2(w.y), a.y);
        ty = fma2(b.x, w.x, ty);
    }
    b.x = fma2(a.x, m2, tx);
    b.y = fma2(a.y, m2, ty);
    a.x = tx;
    a.y = ty;
}
// popcount(i) mod 2 for i < 16 (a table in a constant, so that it folds)
__host__ __device__ constexpr int odd_bits(int i) { return (0x6996 >> i) & 1; }

// One stage of length LEN over x in bit-reversed order, for a DFT with base g:
// Y[a] = sum_j x[j] (g w_K^a)^j, as a decimation in time with the base folded
// into every butterfly: length 2 uses g^{K/2}, length 4 g^{K/4} {1, i}, length 8
// g^{K/8} w_8^{0,1} {1, i}, length 16 g w_16^{0..3} {1, i}.
template <int K, int LEN, int NW>
__device__ __forceinline__ void gstage(Cx (&x)[K], const Cx (&w)[NW]) {
    constexpr int H = LEN / 2;
#pragma unroll
    for (int j = 0; j < H; j++)
#pragma unroll
        for (int b = 0; b < K; b += LEN) {
            if (LEN >= 4 && j >= H / 2)
                bfly<true>(x[b + j], x[b + j + H], w[(j - H / 2) < NW ? (j - H / 2) : 0]);
            else
                bfly<false>(x[b + j], x[b + j + H], w[j < NW ? j : 0]);
        }
}

// w_N^e (e < N) from the two-level table. The low table is stored with one
// entry of padding per 16, so that the lanes' lookups, e = 16 c and multiples,
// do not meet in one bank (32-way conflicts on the plain table).
__device__ __forceinline__ int twlo_pos(int j) { return j + (j >> 4); }
__device__ __forceinline__ float2 tw_p(const float2* __restrict__ twlo, const float2* __restrict__ twhi, unsigned e) {
    return cmul(twlo[twlo_pos((int)(e & 1023u))], twhi[e >> 10]);
}

// The thread index as a value the compiler cannot move out of the unit loop:
// what is derived from it is recomputed where it is used instead of being kept
// in registers (and spilled) across the whole loop.
__device__ __forceinline__ int fresh_tid() {
    int t = threadIdx.x;
    asm volatile("" : "+r"(t));
    return t;
}

// ---- geometry of a row
struct ColGeo {
    int log2Np;   // decimated padded length N'
    int M;        // columns N' / P2
    int NT;       // 128-column tiles
    unsigned Nm;  // N - 1 (twiddle exponents are in units of 1/N)
    int D;        // time decimation
    int KC;       // blocks of P2 bins
};

// k1 of element j of 8-element chunk ch of the K dimension (see the file head).
__host__ __device__ constexpr int chunk_k1(int KC, int ch, int j) {
    if (KC == 64) return (ch >> 1) + 4 * (8 * (ch & 1) + j);
    if (KC == 32) return (ch >> 1) + 2 * (ch & 1) + 4 * j;
    return 2 * ch + (j >> 2) + 4 * (j & 3);
}

// One operand table: the 64 KB A_b: w_M^{k1 (lane + 128 b)}, M = 2^log2M, as four
// arrays (Re hi, Re lo, Im hi, Im lo) of the shared-memory layout: element (lane,
// chunk ch of 8 k1) at ch * 2048 + lane * 16. Built once per plan (block b per
// CTA, in float64) and copied to shared memory when a CTA needs it. Behind A_b
// the pass-1 twiddles of its tiles: column lane of tile jj at jj * 128 + lane,
// as float4 {beta, beta^2} and, 8 KB further, {beta^4, beta^8}, beta = w_N'^{16 c};
// then the pass-2 twiddles of pair p of a1 (sigma = w_{16 R}^{a1}, a1 = 2 p, 2 p + 1):
// sigma^8, sigma^4, sigma^2 w_8^{0,1}, sigma w_16^{0..3}, each as {Re, Re, Im, Im}.
__global__ void k_tc_tables(int log2M, int KC, int R, unsigned char* __restrict__ out) {
    const int b = blockIdx.x;
    const int M = 1 << log2M;
    unsigned char* o = out + (size_t)b * kTcTabBytes;
    for (int t = threadIdx.x; t < 512; t += blockDim.x) {
        const int nt = M >> 7, jj = t >> 7, lane = t & 127;
        const int c = 128 * (nt >= 4 ? b + (nt >> 2) * jj : jj) + lane;
        float v[8];
        for (int k = 0; k < 4; k++) {
            double sn, cs;
            sincospi(2.0 * (double)(((long long)c << k) & ((long long)R * M - 1)) / (double)((long long)R * M), &sn, &cs);
            v[2 * k] = (float)cs;
            v[2 * k + 1] = (float)sn;
        }
        float4* f = reinterpret_cast<float4*>(o + 4 * kTcAArray);
        f[t] = make_float4(v[0], v[1], v[2], v[3]);
        f[512 + t] = make_float4(v[4], v[5], v[6], v[7]);
    }
    for (int t = threadIdx.x; t < R / 2 * 8; t += blockDim.x) {
        const int p = t >> 3, k = t & 7;
        float v[4];
        for (int h = 0; h < 2; h++) {
            const int a1 = 2 * p + h;
            const int e = k == 0 ? 8 * a1 : k == 1 ? 4 * a1 : k < 4 ? 2 * a1 + 2 * R * (k - 2) : a1 + R * (k - 4);
            double sn, cs;
            sincospi(2.0 * (double)(e % (16 * R)) / (16.0 * R), &sn, &cs);
            v[h] = (float)cs;
            v[2 + h] = (float)sn;
        }
        reinterpret_cast<float4*>(o + 4 * kTcAArray + kTcColBytes)[t] = make_float4(v[0], v[1], v[2], v[3]);
    }
    for (int t = threadIdx.x; t < 128 * 64; t += blockDim.x) {
        const int j = t & 7, lane = (t >> 3) & 127, vch = t >> 10;  // element, row, version x chunk
        const int nch = KC / 8;
        const int v = vch / nch;  // version
        const int k1 = chunk_k1(KC, vch - v * nch, j);
        const int c = lane + 128 * b;
        double sn, cs;
        sincospi(2.0 * (double)(((long long)k1 * c) & (M - 1)) / (double)M, &sn, &cs);
        float2 w = make_float2((float)cs, (float)sn);
        if (c >= M) w = make_float2(0.0f, 0.0f);
        // versions: KC = 32, j odd negates k1 = 2, 3 mod 4; KC = 16: times i^{k1 v}
        const int m = KC == 32 ? (v == 1 && (k1 & 2) ? 2 : 0) : KC == 16 ? (k1 * v) & 3 : 0;
        if (m == 1) w = make_float2(-w.y, w.x);
        if (m == 2) w = make_float2(-w.x, -w.y);
        if (m == 3) w = make_float2(w.y, -w.x);
        const __half hr = __float2half_rn(w.x), hi = __float2half_rn(w.y);
        __half* p = reinterpret_cast<__half*>(o + vch * 2048 + lane * 16) + j;
        p[0] = hr;
        p[kTcAArray / 2] = __float2half_rn(w.x - __half2float(hr));
        p[2 * (kTcAArray / 2)] = hi;
        p[3 * (kTcAArray / 2)] = __float2half_rn(w.y - __half2float(hi));
    }
}

// Copies of one operand table into shared memory (one thread): A, and the
// twiddles once no column warp reads the previous ones.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, int bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void load_a(uint32_t sm, const unsigned char* src, int col_bytes, uint32_t mbar) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
                 "r"(4 * kTcAArray + col_bytes)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; i++) bulk_load(sm + i * kTcAArray, src + i * kTcAArray, kTcAArray, mbar);
}
__device__ __forceinline__ void load_col(uint32_t sm, const unsigned char* src, int col_bytes, uint32_t mbar) {
    bulk_load(sm + kTcOffCol, src + 4 * kTcAArray, col_bytes, mbar);
}

// Issues the MMAs of one accumulator block of a tile (quarter-turn index j):
// Re (part 0) or Im (part 1). Two warps issue the two parts. R = 16: two halves
// of the k2 rows, half 0 before half 1, so that pass 1 starts on half 0 while
// half 1 runs. R = 8: one block of N = 128 (a half would have N = 64, where
// reading A and B from shared memory takes 1.5 times as long as the MMA; the
// second accumulator buffer hides the latency anyway).
template <int R>
__device__ __forceinline__ void issue_block(int KC, int j, int part, int half, uint32_t tmem, uint32_t a0, uint32_t z0,
                                            uint32_t mbar) {
    constexpr int P2 = 16 * R;
    constexpr int W = R == 16 ? P2 / 2 : P2;  // accumulator columns of a block
    const uint32_t d = tmem + (uint32_t)(half * W + part * P2);
    const uint32_t zarr = (uint32_t)(KC * P2 * 2) >> 4;  // array strides in descriptor units of 16 bytes
    constexpr uint32_t aarr = kTcAArray >> 4;
    const uint32_t idp = umma_idesc(W, 0), idn = umma_idesc(W, 1);
    const int steps = KC / 16;
    const int rot = KC == 16 ? 0 : j;  // quarter turns per k1 mod 4 left to the issue
    const uint32_t ab = umma_desc_lo(a0 + (KC == 16 ? (uint32_t)(j * 2 * 2048) : KC == 32 ? (uint32_t)((j & 1) * 4 * 2048) : 0u),
                                     2048);
    const uint32_t zb = umma_desc_lo(z0 + (uint32_t)(half * W * 16), P2 * 16);
    uint32_t acc = 0;
    // lo hi and hi lo first: their sums are 2^-11 of the result, so only the hi hi
    // accumulations round at full magnitude
#pragma unroll 1
    for (int p = 0; p < 3; p++) {
        uint32_t as = ab + (p == 0 ? aarr : 0u), zs = zb + (p == 1 ? zarr : 0u);
        int m = 0;
#pragma unroll 1
        for (int s = 0; s < steps; s++) {
            // i^m (Wr + i Wi) = X + i Y; Re: X Zr - Y Zi, Im: Y Zr + X Zi
            const bool odd = (m & 1) != 0;
            const bool nx = m == 1 || m == 2, ny = m >= 2;
            const uint32_t ax = as + (odd ? 2 * aarr : 0u), ay = as + (odd ? 0u : 2 * aarr);
            mma_ss(d, part ? ay : ax, zs, (part ? ny : nx) ? idn : idp, acc);
            mma_ss(d, part ? ax : ay, zs + 2 * zarr, (part ? nx : !ny) ? idn : idp, 1);
            acc = 1;
            as += 4096 >> 4;
            zs += (2 * P2 * 16) >> 4;
            m = (m + rot) & 3;
        }
    }
    mma_commit(mbar + 8u * half);
    if (R == 8) mma_commit(mbar + 8u);
}

__device__ __forceinline__ void prod_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kTcProdThreads) : "memory"); }

// Pre-pass of a row (producer warps): Z on the window, scaled by 2^e (max |Z|
// 2^e in [2^14, 2^15)), split into FP16 hi + lo, as the MMA's B operand. A task
// is (row n of B, chunk of 8 k1). The spectrum copy Xp and the weight table hold
// each block of P2 bins in the order n = perm_bin, so that a warp reads 32
// consecutive entries and its 16-byte shared-memory accesses are conflict-free.
// The unscaled values wait for the row's maximum in shared memory, in the place
// of the results. Folded rows (decimated): the window is F x KC x P2 bins and
// N' = KC P2. Returns 2^-e (1 + 2^-23).
template <int R, int KC, bool FOLD>
__device__ __forceinline__ float tc_prepass(const TcParams& P, const RowDesc& Rw, const SigDesc& S, unsigned char* zb,
                                            float* s_red) {
    constexpr int P2 = 16 * R;
    constexpr int kLogR = ilog2c(R);
    constexpr int zarr = KC * P2 * 2;
    const int tid = fresh_tid() - kTcColThreads;
    // A pair task is (row n, two chunks): 16 bins whose offsets are immediates.
    // Thread: row n, the pair tasks q0, q0 + QS, ...
    constexpr int PR = KC / 16;                     // pair tasks per row
    constexpr int QS = kTcProdThreads / P2;         // threads per row: 1 or 2
    const int n = tid & (P2 - 1);
    const int q0 = tid / P2;
    const int k2 = (n >> kLogR) + 16 * (n & (R - 1));
    const unsigned len = (unsigned)(Rw.hi - Rw.lo);
    const float* __restrict__ wrow = P.wts + Rw.woff + n;
    const float2* xrow = S.Xp + Rw.L + n;  // (plain loads: read-only ones may be moved above grid_dep_wait)
    const int u0 = Rw.L + k2 - Rw.lo;  // a bin is in [lo, hi) when (unsigned)(u0 + its offset) < len
    struct Load {
        float2 v[16];
        float m[16];
    };
    auto fetch = [&](int q, int f, Load& d) {
        const int ob = P2 * (q + f * KC);
        const float* wp = wrow + ob;
        const float2* xp = xrow + ob;
        const int u = u0 + ob;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int o = P2 * chunk_k1(KC, j >> 3, j & 7);
            d.v[j] = make_float2(0.0f, 0.0f);
            d.m[j] = 0.0f;
            if ((unsigned)(u + o) < len) {
                d.m[j] = __ldg(wp + o);
                d.v[j] = xp[o];
            }
        }
    };
    float mx = 0.0f;
    auto park = [&](int q, Load& d) {
        unsigned char* p = zb + n * 16 + 2 * q * (P2 * 16);
#pragma unroll
        for (int j = 0; j < 16; j++) d.v[j] = cscale(d.v[j], d.m[j]);
        if (FOLD)
            for (int f = 1; f < Rw.folds; f++) {
                Load e;
                fetch(q, f, e);
#pragma unroll
                for (int j = 0; j < 16; j++) d.v[j] = cadd(d.v[j], cscale(e.v[j], e.m[j]));
            }
        if (Rw.imag)
#pragma unroll
            for (int j = 0; j < 16; j++) d.v[j] = make_float2(-d.v[j].y, d.v[j].x);
#pragma unroll
        for (int j = 0; j < 16; j++) mx = fmaxf(mx, fmaxf(fabsf(d.v[j].x), fabsf(d.v[j].y)));
#pragma unroll
        for (int k = 0; k < 8; k++)
            *reinterpret_cast<float4*>(p + (k >> 2) * (P2 * 16) + (k & 3) * zarr) =
                make_float4(d.v[2 * k].x, d.v[2 * k].y, d.v[2 * k + 1].x, d.v[2 * k + 1].y);
    };
#pragma unroll 1
    for (int q = q0; q < PR; q += QS) {
        Load d;
        fetch(q, 0, d);
        park(q, d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((tid & 31) == 0) s_red[tid >> 5] = mx;
    prod_bar();
    mx = s_red[tid & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int ex = 0;
    if (mx > 0.0f) frexpf(mx, &ex);
    const int e2 = max(-126, min(126, 15 - ex));
    const float scale = ldexpf(1.0f, e2);
    // (the same tasks again: a thread reads back what it parked)
#pragma unroll 1
    for (int q = q0; q < PR; q += QS) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            unsigned char* p = zb + n * 16 + (2 * q + h) * (P2 * 16);
            uint32_t rh[4], rl[4], ih[4], il[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 t = *reinterpret_cast<const float4*>(p + k * zarr);
                const float ax = t.x * scale, ay = t.y * scale, cx = t.z * scale, cy = t.w * scale;
                const __half2 hr = __floats2half2_rn(ax, cx);
                const __half2 hi = __floats2half2_rn(ay, cy);
                const float2 fr = __half22float2(hr), fi = __half22float2(hi);
                rh[k] = h2bits(hr);
                ih[k] = h2bits(hi);
                rl[k] = h2bits(__floats2half2_rn(ax - fr.x, cx - fr.y));
                il[k] = h2bits(__floats2half2_rn(ay - fi.x, cy - fi.y));
            }
            *reinterpret_cast<uint4*>(p) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
            *reinterpret_cast<uint4*>(p + zarr) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
            *reinterpret_cast<uint4*>(p + 2 * zarr) = make_uint4(ih[0], ih[1], ih[2], ih[3]);
            *reinterpret_cast<uint4*>(p + 3 * zarr) = make_uint4(il[0], il[1], il[2], il[3]);
        }
    }
    // The tensor cores' accumulation drops bits towards zero: rows came out too small by 1e-7
    // to 3e-7 of their size, the largest part of their error (10000 x 200: 2.8e-7 of
    // which 2.2e-7 is that factor). One unit in the last place takes half of it back:
    // 1.95e-7; 100000 x 300 3.3 -> 2.6e-7, every 16th sample of it 3.6 -> 2.7e-7. What is left
    // goes with the blocks that hold bins rather than with KC (zeros drop nothing): rows of 12
    // grids of N = 16384 to 2^19 are off by -2.0e-7 to -0.4e-7 with KC = 64, -1.4e-7 to
    // -0.3e-7 with 32, -1.2e-7 to +0.5e-7 with 16; without the factor the smallest of all
    // was -0.7e-7. The same rows of the CUDA-core engine are off by -3.3e-7 to -0.9e-7.
    return ldexpf(1.0f + 1.1920929e-7f, -e2);
}

// Scalar butterfly of negated (neg) inputs: s = e + w o, d = e - w o.
__device__ __forceinline__ void bfly_s(bool neg, float2 e, float2 o, float2 w, float2& s, float2& d) {
    if (neg) {
        e = make_float2(-e.x, -e.y);
        o = make_float2(-o.x, -o.y);
    }
    s.x = fmaf(-o.y, w.y, fmaf(o.x, w.x, e.x));
    s.y = fmaf(o.x, w.y, fmaf(o.y, w.x, e.y));
    d.x = fmaf(2.0f, e.x, -s.x);
    d.y = fmaf(2.0f, e.y, -s.y);
}

// Pass 1 of one kl: DFT_R over kb of the column's accumulators r = {Re[R],
// Im[R]} with base beta and factor kappa, even and odd kb as packed halves; the
// last stage writes the outputs of pair p = a1 / 2 as {Re, Re, Im, Im} in place.
template <int R>
__device__ __forceinline__ void pass1_load(uint32_t tre, uint32_t (&r)[2 * R]) {
    if constexpr (R == 16) {
        tmem_ld16(tre, r);
        tmem_ld16(tre + 16 * R, r + 16);
    } else {
        tmem_ld8(tre, r);
        tmem_ld8(tre + 16 * R, r + 8);
    }
}
template <int R>
__device__ __forceinline__ void pass1(uint32_t tre, const uint32_t (&r)[2 * R], float2 kappa, const Cx (&g)[4],
                                      const float2 (&bw)[4]) {
    constexpr int H = R / 2;
    constexpr int LH = ilog2c(H);
    Cx x[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
        const int s = brev(j, LH);
        x[j] = {pku(r[2 * s], r[2 * s + 1]), pku(r[R + 2 * s], r[R + 2 * s + 1])};
    }
    // first stage (length 2) with kappa: a' = kappa a, w' = kappa g^{H/2}
    const Cx kp = dup(kappa);
    const Cx w0 = cmulx(g[0], kp);
#pragma unroll
    for (int j = 0; j < H; j += 2) {
        x[j] = cmulx(x[j], kp);
        bfly<false>(x[j], x[j + 1], w0);
    }
    {
        const Cx w[1] = {g[1]};
        gstage<H, 4>(x, w);
    }
    if constexpr (H == 8) {
        const Cx w[2] = {g[2], g[3]};
        gstage<H, 8>(x, w);
    }
    // last stage: X[a] = E[a] + beta w_R^a O[a], a < H, and X[a + H] = E[a] - ...;
    // E and O carry the sign of a, which scalar FMAs take for free
    float o[2 * R];
#pragma unroll
    for (int a = 0; a < H; a++) {
        float ex, ey, ox, oy;
        unpk(x[a].x, ex, ox);
        unpk(x[a].y, ey, oy);
        const float2 b = bw[a < H / 2 ? a : a - H / 2];
        float2 sm, df;
        bfly_s(odd_bits(a) != 0, make_float2(ex, ey), make_float2(ox, oy), a < H / 2 ? b : make_float2(-b.y, b.x), sm, df);
        o[(a >> 1) * 4 + (a & 1)] = sm.x;
        o[(a >> 1) * 4 + (a & 1) + 2] = sm.y;
        o[((a + H) >> 1) * 4 + (a & 1)] = df.x;
        o[((a + H) >> 1) * 4 + (a & 1) + 2] = df.y;
    }
    if constexpr (R == 16) {
        tmem_st16(tre, o);
        tmem_st16(tre + 16 * R, o + 16);
    } else {
        tmem_st8(tre, o);
        tmem_st8(tre + 16 * R, o + 8);
    }
}

// Streaming store of sample a2 of `count`, predicated (no branch around it).
template <int OT>
__device__ __forceinline__ void store_point(int a2, int count, char* p, float re, float im) {
    if constexpr (OT == OUT_C64)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %0, %1;\n\t@p st.global.cs.v2.f32 [%2], {%3, %4};\n\t}\n" ::"r"(
                         count),
                     "r"(a2), "l"(p), "f"(re), "f"(im)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %0, %1;\n\t@p st.global.cs.b32 [%2], %3;\n\t}\n" ::"r"(count),
                     "r"(a2), "l"(p), "r"(pack16<OT>(make_float2(re, im)))
                     : "memory");
}
__device__ __forceinline__ float4 lds128(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// Last stage of pass 2 and the stores of one pair of a1: the outputs of the two
// a1 come as (Re, Im), and the sign of the inputs is free. LS: log2 of the
// samples between consecutive a2, so that the 32 addresses are two registers
// and immediates (0: taken from logS).
template <int OT, int LS>
__device__ __forceinline__ void finish_pair(const Cx (&x)[16], uint32_t tw, char* pa, char* pb, int la, int lb,
                                            int logS) {
    constexpr unsigned ES = OT == OUT_C64 ? 8 : 4;
    const size_t str = (size_t)ES << (LS ? LS : logS);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float4 w = lds128(tw + 16u * j);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int a2 = j + 4 * q;
            float e0x, e0y, o0x, o0y, e1x, e1y, o1x, o1y;
            unpk(x[a2].x, e0x, e1x);
            unpk(x[a2].y, e0y, e1y);
            unpk(x[a2 + 8].x, o0x, o1x);
            unpk(x[a2 + 8].y, o0y, o1y);
            const float2 w0 = q == 0 ? make_float2(w.x, w.z) : make_float2(-w.z, w.x);
            const float2 w1 = q == 0 ? make_float2(w.y, w.w) : make_float2(-w.w, w.y);
            const bool neg = odd_bits(a2) != 0;
            float2 s0, d0, s1, d1;
            bfly_s(neg, make_float2(e0x, e0y), make_float2(o0x, o0y), w0, s0, d0);
            bfly_s(neg, make_float2(e1x, e1y), make_float2(o1x, o1y), w1, s1, d1);
            store_point<OT>(a2, la, pa + a2 * str, s0.x, s0.y);
            store_point<OT>(a2, lb, pb + a2 * str, s1.x, s1.y);
            store_point<OT>(a2 + 8, la, pa + (a2 + 8) * str, d0.x, d0.y);
            store_point<OT>(a2 + 8, lb, pb + (a2 + 8) * str, d1.x, d1.y);
        }
    }
}

// finish_pair for the row's length: N' / 16 = 2^logS samples are between consecutive a2,
// logS = 9 or 10 for R = 8 and 10 to 19 for R = 16. Up to 16 the 15 steps of 8 bytes fit
// the 24-bit offset of a store (500000 x 300: 328 us, its power 295; with the steps added
// to the addresses 335 and 333). Longer rows add them.
template <int OT, int LO, int HI>
__device__ __forceinline__ void store_pair(const Cx (&x)[16], uint32_t tw, char* pa, char* pb, int la, int lb,
                                           int logS) {
    if constexpr (LO == HI) {
        finish_pair<OT, LO <= 16 ? LO : 0>(x, tw, pa, pb, la, lb, logS);
    } else {
        constexpr int MID = (LO + HI) / 2;
        if (logS <= MID)
            store_pair<OT, LO, MID>(x, tw, pa, pb, la, lb, logS);
        else
            store_pair<OT, MID + 1, HI>(x, tw, pa, pb, la, lb, logS);
    }
}

// One unit: a row's descriptors, its tiles and the scale of its Z.
struct UnitSlot {
    int idx;    // position in the queue; at or past the end: stop
    int unit;
    float inv;  // 2^-e
    int pad;
    RowDesc R;
    SigDesc S;
};
struct TcShared {
    unsigned long long mma[2][2];       // [accumulator buffer][half]: MMAs done (Re and Im commits)
    unsigned long long freeb[2];        // [accumulator buffer]: read by all column warps
    unsigned long long abar;            // operand table copied
    unsigned long long meta[kTcSlots];  // unit descriptor and scale published
    uint32_t tmem;
    float red[kTcProdThreads / 32];
    UnitSlot u[kTcSlots];
};

// Claims the CTA's next unit and pulls its weights and spectrum window into L2: first
// the unit of its block index, then the queue's.
__device__ __forceinline__ void tc_claim_next(const TcParams& P, UnitSlot& U, bool first) {
    const int i = first ? (int)blockIdx.x : (int)(gridDim.x + atomicAdd(P.counter, 1u));
    U.idx = i;
    if (i < P.n_list) {
        const int e = P.row_list[i];
        U.unit = e;
        U.R = P.rows[e & kUnitRowMask];
        U.S = P.sigs[U.R.sig];
        const int wlen = (16 << U.R.log2R) * U.R.kp * U.R.folds;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(P.wts + U.R.woff), "r"((unsigned)wlen * 4u)
                     : "memory");
        const int xe = min(wlen, (1 << (U.S.log2N - 1)) - U.R.L);
        if (xe > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(U.S.Xp + U.R.L), "r"((unsigned)xe * 8u)
                         : "memory");
    }
}

// Tiles of a unit run in the order s -> T = b + (NT / 4) j with b = s / 4,
// j = s % 4 (NT >= 4).
__device__ __forceinline__ ColGeo col_geo(const RowDesc& Rw, const SigDesc& S) {
    ColGeo G;
    G.D = Rw.dec;
    G.log2Np = S.log2N - (31 - __clz(Rw.dec));
    G.M = 1 << (G.log2Np - 4 - Rw.log2R);
    G.NT = max(1, G.M >> 7);
    G.Nm = (1u << S.log2N) - 1u;
    G.KC = Rw.kp;
    return G;
}
__device__ __forceinline__ int tile_b(const ColGeo& G, int s) { return G.NT >= 8 ? s >> 2 : 0; }
__device__ __forceinline__ int tile_j(const ColGeo& G, int s) { return G.NT >= 4 ? s & 3 : G.NT == 2 ? 2 * s : 0; }
__device__ __forceinline__ int tile_T(const ColGeo& G, int s) {
    return G.NT >= 4 ? (s >> 2) + (G.NT >> 2) * (s & 3) : s;
}

// Accumulator buffers: a tile takes 32 R of the 512 columns.
template <int R>
constexpr int kTcBufs = R == 16 ? 1 : 2;

// w_N^{1024 j}: in shared memory when it fits.
__device__ __forceinline__ const float2* high_table(const SigDesc& S, const float2* twhi_s) {
    return (1 << (S.log2N - kLog2P2)) <= kTcTwhiSmem ? twhi_s : S.tw + kP2;
}

// Producer warps: per unit the pre-pass into shared memory, then the MMAs of
// its tiles, each once the column warps have read the accumulators that it
// overwrites. Z of up to 64 KB alternates between two halves of its region, so
// that the next unit's pre-pass runs under the current unit; wider windows take
// the whole region and wait for the previous unit's last MMAs only.
template <int R>
__device__ __forceinline__ void produce(const TcParams& P, TcShared& sh, unsigned char* sm, uint32_t tmem) {
    constexpr int P2 = 16 * R;
    constexpr int NB = kTcBufs<R>;
    float2* twlo = reinterpret_cast<float2*>(sm + kTcOffTwlo);
    float2* twhi_s = reinterpret_cast<float2*>(sm + kTcOffTwhi);
    const int ptid = threadIdx.x - kTcColThreads;
    const int pw = ptid >> 5;
    const bool issuer = (ptid & 31) == 0 && pw < 2;
    const uint32_t a0 = smem_u32(sm);
    auto mma_done = [&](int t) {  // all MMAs up to tile t of this CTA
        const uint32_t m = smem_u32(&sh.mma[t % NB][0]);
        mbar_wait(m, (uint32_t)(t / NB) & 1u, P.err);
        mbar_wait(m + 8, (uint32_t)(t / NB) & 1u, P.err);
    };
    int t = 0;                // tiles issued
    auto free_all = [&]() {   // the accumulators of every issued tile are read
        for (int i = max(0, t - NB); i < t; i++)
            mbar_wait(smem_u32(&sh.freeb[i % NB]), (uint32_t)(i / NB) & 1u, P.err);
    };
    int zlast[2] = {-1, -1};  // last tile that reads each half of the Z region
    const unsigned char* acur = nullptr;  // operand table in shared memory
    uint32_t aphase = 0;
    int cur_log2N = -1;
    for (int k = 0;; k++) {
        UnitSlot& U = sh.u[k & (kTcSlots - 1)];
        prod_bar();  // the claim of this unit is visible; every producer is done with the previous unit
        if (U.idx >= P.n_list) {
            if (ptid == 0) mbar_arrive(smem_u32(&sh.meta[k & (kTcSlots - 1)]));
            break;
        }
        const ColGeo G = col_geo(U.R, U.S);
        int sb, se;
        tc_unit_tiles(U.unit, G.NT, &sb, &se);
        // where Z goes, once nothing reads it any more
        const bool half = G.KC * P2 * 8 <= kTcZBytes / 2;
        const int h0 = half ? k & 1 : 0, h1 = half ? h0 : 1;
        const int zl = max(h0 ? zlast[1] : zlast[0], h1 ? zlast[1] : zlast[0]);
        if (zl >= 0 && zl >= t - NB) mma_done(zl);  // (earlier tiles: done when their buffer was issued again)
        const uint32_t zoff = kTcOffZ + (half ? (uint32_t)h0 * (kTcZBytes / 2) : 0u);
        if (U.S.log2N != cur_log2N) {
            free_all();  // the column warps read the tables only before they free a tile
            const int M = 1 << (U.S.log2N - kLog2P2);
            for (int j = ptid; j < kP2; j += kTcProdThreads) twlo[twlo_pos(j)] = U.S.tw[j];
            if (M <= kTcTwhiSmem)
                for (int j = ptid; j < M; j += kTcProdThreads) twhi_s[j] = U.S.tw[kP2 + j];
            cur_log2N = U.S.log2N;
        }
        bool a_pending = false;
        if (k == 0) {
            // All that does not read the forward transform's results runs under its last
            // kernel: the tables above, the first operand table and the claim of the unit.
            acur = P.atab + U.R.aoff + (long long)tile_b(G, sb) * kTcTabBytes;
            if (ptid == 0) {
                // (the pass-2 twiddles behind the columns' are the same in every table: once)
                load_a(a0, acur, kTcColBytes + kTcS2Bytes, smem_u32(&sh.abar));
                load_col(a0, acur, kTcColBytes + kTcS2Bytes, smem_u32(&sh.abar));
            }
            a_pending = true;
            grid_dep_wait();
        }
        if (ptid == kTcProdThreads - 32) tc_claim_next(P, sh.u[(k + 1) & (kTcSlots - 1)], false);
        unsigned char* zb = sm + zoff;
        const float inv = U.R.folds > 1 ? tc_prepass<R, 64, true>(P, U.R, U.S, zb, sh.red)
                          : G.KC == 64  ? tc_prepass<R, 64, false>(P, U.R, U.S, zb, sh.red)
                          : G.KC == 32  ? tc_prepass<R, 32, false>(P, U.R, U.S, zb, sh.red)
                                        : tc_prepass<R, 16, false>(P, U.R, U.S, zb, sh.red);
        if (ptid == 0) U.inv = inv;
        for (int s = sb; s < se; s++) {
            const unsigned char* atab = P.atab + U.R.aoff + (long long)tile_b(G, s) * kTcTabBytes;
            if (s == sb) {
                fence_proxy_async_smem();
                prod_bar();
            }
            if (atab != acur) {
                // (the copying thread alone waits: another, held up until the issuers are through
                // with the unit, would find the barrier two phases on and wait for a third)
                if (ptid == 0) {
                    mma_done(t - 1);
                    load_a(a0, atab, kTcColBytes, smem_u32(&sh.abar));
                    free_all();
                    load_col(a0, atab, kTcColBytes, smem_u32(&sh.abar));
                }
                acur = atab;
                a_pending = true;
            }
            if (a_pending) {
                if (issuer) mbar_wait(smem_u32(&sh.abar), aphase, P.err);
                aphase ^= 1u;
                a_pending = false;
            }
            if (s == sb && ptid == 0) mbar_arrive(smem_u32(&sh.meta[k & (kTcSlots - 1)]));
            const int buf = t % NB;
            if (issuer) {
                if (t >= NB) mbar_wait(smem_u32(&sh.freeb[buf]), (uint32_t)(t / NB - 1) & 1u, P.err);
                tc_fence_after();
                for (int half = 0; half < (R == 16 ? 2 : 1); half++)
                    issue_block<R>(G.KC, tile_j(G, s), pw, half, tmem + (uint32_t)(buf * 2 * P2), a0, a0 + zoff,
                                   smem_u32(&sh.mma[buf][0]));
            }
            __syncwarp();
            t++;
        }
        if (h0 == 0) zlast[0] = t - 1;
        if (h1 == 1) zlast[1] = t - 1;
    }
}

// Column warps: the DFTs and stores of every tile, in the order of the issue.
template <int OT, int R>
__device__ __forceinline__ void consume(const TcParams& P, TcShared& sh, unsigned char* sm, uint32_t tmem) {
    constexpr int P2 = 16 * R;
    constexpr int NB = kTcBufs<R>;
    constexpr unsigned ES = OT == OUT_C64 ? 8 : 4;
    const float2* twlo = reinterpret_cast<const float2*>(sm + kTcOffTwlo);
    const float2* twhi_s = reinterpret_cast<const float2*>(sm + kTcOffTwhi);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int qd = warp & 3;   // lane quadrant
    const int w2 = warp >> 2;  // 0 or 1: every other kl, every other pair of a1
    const uint32_t tlane = tmem + ((uint32_t)(32 * qd) << 16);
    const uint32_t s2 = smem_u32(sm) + kTcOffS2;
    int t = 0;
    for (int k = 0;; k++) {
        const int slot = k & (kTcSlots - 1);
        mbar_wait(smem_u32(&sh.meta[slot]), (uint32_t)(k / kTcSlots) & 1u, P.err);
        const UnitSlot& U = sh.u[slot];
        if (U.idx >= P.n_list) break;
        const RowDesc& Rw = U.R;
        const ColGeo G = col_geo(Rw, U.S);
        const float2* twhi = high_table(U.S, twhi_s);
        const unsigned D = (unsigned)G.D, Nm = G.Nm;
        const float inv = U.inv;
        int sb, se;
        tc_unit_tiles(U.unit, G.NT, &sb, &se);
        char* outb = reinterpret_cast<char*>(P.outs[Rw.out_buf]) + Rw.out_off * ES;
        const int n = Rw.n_out;
        const int logS = G.log2Np - 4;  // samples between consecutive a2: 2^logS
        const bool active = 32 * qd < G.M;
#pragma unroll 1
        for (int s = sb; s < se; s++, t++) {
            const int buf = t % NB;
            const uint32_t par = (uint32_t)(t / NB) & 1u;
            const uint32_t mma = smem_u32(&sh.mma[buf][0]), fbar = smem_u32(&sh.freeb[buf]);
            const uint32_t tq = tlane + (uint32_t)(buf * 2 * P2);
            const int c = 128 * tile_T(G, s) + 32 * qd + lane;
            const unsigned cD = (unsigned)c * D;
            if (!active) {
                // no columns in this quadrant: only keep the order of the tiles
                mbar_wait(mma, par, P.err);
                mbar_wait(mma + 8, par, P.err);
                __syncwarp();
                if (lane == 0) mbar_arrive(fbar);
                continue;
            }
            {
                // kappa of kl = w2 + 2 i: 2^-e w_N'^{(L + kl) c}, looked up for i = 0 and 4
                auto kappa = [&](int kl) {
                    return cscale(tw_p(twlo, twhi, ((unsigned)(Rw.L + kl) * cD) & Nm), inv);
                };
                float2 kap = kappa(w2);
                const float2 kstep = tw_p(twlo, twhi, (2u * cD) & Nm);
                mbar_wait(mma, par, P.err);
                __syncwarp();
                tc_fence_after();
                // pass-1 twiddles, beta = w_N'^{16 c}
                float2 bw[4];
                Cx g[4];
                {
                    const uint32_t ca = smem_u32(sm) + kTcOffCol +
                                        16u * (uint32_t)((G.NT >= 4 ? s & 3 : s) * 128 + 32 * qd + lane);
                    const float4 b12 = lds128(ca), b48 = lds128(ca + 8192u);
                    constexpr float c1 = kCos64[4], s1 = kCos64[12], c2 = kCos64[8];
                    const float2 b1 = make_float2(b12.x, b12.y), b2 = make_float2(b12.z, b12.w);
                    bw[0] = b1;
                    if constexpr (R == 16) {
                        bw[1] = cmul(b1, make_float2(c1, s1));
                        bw[2] = cmul(b1, make_float2(c2, c2));
                        bw[3] = cmul(b1, make_float2(s1, c1));
                        g[0] = dup(make_float2(b48.z, b48.w));
                        g[1] = dup(make_float2(b48.x, b48.y));
                        g[2] = dup(b2);
                        g[3] = dup(cmul(b2, make_float2(c2, c2)));
                    } else {
                        bw[1] = cmul(b1, make_float2(c2, c2));
                        bw[2] = bw[3] = b1;
                        g[0] = dup(make_float2(b48.x, b48.y));
                        g[1] = dup(b2);
                        g[2] = g[3] = g[1];
                    }
                }
                // the next kl's accumulators are loaded under the current one's arithmetic
                const uint32_t t0 = tq + (uint32_t)(w2 * R);
                uint32_t ra[2 * R], rb[2 * R];
                pass1_load<R>(t0, ra);
#pragma unroll 1
                for (int i = 0; i < 8; i += 2) {
                    tmem_wait_ld(ra);
                    pass1_load<R>(t0 + (uint32_t)(2 * (i + 1) * R), rb);
                    pass1<R>(t0 + (uint32_t)(2 * i * R), ra, kap, g, bw);
                    kap = cmul(kap, kstep);
                    if (i == 2) {
                        mbar_wait(mma + 8, par, P.err);
                        __syncwarp();
                        tc_fence_after();
                    }
                    tmem_wait_ld(rb);
                    if (i < 6) pass1_load<R>(t0 + (uint32_t)(2 * (i + 2) * R), ra);
                    pass1<R>(t0 + (uint32_t)(2 * (i + 1) * R), rb, kap, g, bw);
                    kap = i == 2 ? kappa(w2 + 8) : cmul(kap, kstep);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            asm volatile("bar.sync %0, 64;" ::"r"(2 + qd) : "memory");  // the quadrant's two warps
            tc_fence_after();
            // pass 2: pairs p = w2 + 2 i of a1, the next pair loaded under the current one
            constexpr int NP = R / 4;
            uint32_t r[64];
            auto load_pair = [&](int i) {
                const int p = w2 + 2 * i;
                const uint32_t t0 = tq + (p < R / 4 ? (uint32_t)(4 * p) : (uint32_t)(P2 + 4 * p - R));
#pragma unroll
                for (int kl = 0; kl < 16; kl++) tmem_ld4(t0 + (uint32_t)(kl * R), r + 4 * kl);
            };
            load_pair(0);
            tmem_wait_ld(r);
            if (w2 == 1) asm volatile("bar.sync %0, 64;" ::"r"(6 + qd) : "memory");
#pragma unroll 1
            for (int i = 0; i < NP; i++) {
                const int p = w2 + 2 * i;
                Cx x[16];
#pragma unroll
                for (int kl = 0; kl < 16; kl++) {
                    const int kb = brev(kl, 4);
                    x[kl] = {pku(r[4 * kb], r[4 * kb + 1]), pku(r[4 * kb + 2], r[4 * kb + 3])};
                }
                const uint32_t tp = s2 + (uint32_t)p * 128u;
                auto ldtw = [&](int q) -> Cx {
                    const float4 v = lds128(tp + 16u * q);
                    return {pk(v.x, v.y), pk(v.z, v.w)};
                };
                {
                    const Cx w[1] = {ldtw(0)};
                    gstage<16, 2>(x, w);
                }
                if (i + 1 < NP) load_pair(i + 1);
                {
                    const Cx w[1] = {ldtw(1)};
                    gstage<16, 4>(x, w);
                }
                {
                    const Cx w[2] = {ldtw(2), ldtw(3)};
                    gstage<16, 8>(x, w);
                }
                // warp 1 of the quadrant starts when warp 0 begins to store: from there on one
                // warp of each scheduler computes while the other one stores
                if (i == 0 && w2 == 0) asm volatile("bar.arrive %0, 64;" ::"r"(6 + qd) : "memory");
                tmem_wait_ld(r);
                if (i == NP - 2) {
                    // this warp's last read of the tile's accumulators
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(fbar);
                }
                // y[t0 + S a2] for t0 = c + M a1, S = N' / 16
                const int ta = c + G.M * (2 * p), tb = ta + G.M;
                const int S1 = (1 << logS) - 1;
                int la = (n - ta + S1) >> logS, lb = (n - tb + S1) >> logS;  // stored a2 of each
                if (c >= G.M) la = lb = 0;
                char* pa = outb + (size_t)((unsigned)ta * ES);
                char* pb = outb + (size_t)((unsigned)tb * ES);
                store_pair<OT, R == 16 ? 10 : 9, R == 16 ? 17 : 10>(x, tp + 64u, pa, pb, la, lb, logS);
                __syncwarp();
            }
        }
    }
}

// One launch takes rows of one R (each R is register-allocated by itself).
template <int OT, int R>
__global__ void __launch_bounds__(kTcThreads, 1) k_row_tc(const __grid_constant__ TcParams P) {
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    unsigned char* sm = tc_smem_raw + ((1024u - (smem_u32(tc_smem_raw) & 1023u)) & 1023u);
    __shared__ __align__(8) TcShared sh;
    const int tid = threadIdx.x;
    const int warp = tid >> 5;

    if (tid == 0) {
        auto init = [](unsigned long long* b, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
        };
        for (int i = 0; i < 2; i++) {
            init(&sh.mma[i][0], 2);
            init(&sh.mma[i][1], 2);
            init(&sh.freeb[i], kTcColThreads / 32);
        }
        init(&sh.abar, 1);
        for (int i = 0; i < kTcSlots; i++) init(&sh.meta[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)),
                     "r"(kTcTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == kTcColThreads) tc_claim_next(P, sh.u[0], true);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    if (warp >= kTcColThreads / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcProdRegs));
        produce<R>(P, sh, sm, tmem);
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcColRegs));
        consume<OT, R>(P, sh, sm, tmem);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols));
}

// Plan-time weight table of the tensor-core rows: entry blk P2 + n of a row is
// the daughter weight of bin q = L + blk P2 + k2(n) times out_scale (0 outside
// [lo, hi)), the same float product the engines apply per bin, in the pre-pass's
// order n = kl R + kb of each block of P2 bins.
__global__ void k_tc_weights(const SigDesc* __restrict__ sigs, const RowDesc* __restrict__ rows,
                             const int* __restrict__ row_list, const float* __restrict__ pool,
                             float* __restrict__ wts) {
    const RowDesc R = rows[row_list[blockIdx.x]];
    const SigDesc S = sigs[R.sig];
    const float nm1 = (float)(1 << S.log2N) - 1.0f;
    const int P2 = 16 << R.log2R;
    const int len = P2 * R.kp * R.folds;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
        const int n = i & (P2 - 1);
        const int k2 = (n >> R.log2R) + 16 * (n & ((1 << R.log2R) - 1));
        const int q = R.L + (i - n) + k2;
        wts[R.woff + i] = (q >= R.lo && q < R.hi) ? bin_weight(R, S.mother, pool, nm1, q) * R.out_scale : 0.0f;
    }
}

}  // namespace dev

cudaError_t launch_tc_weights(const SigDesc* sigs, const RowDesc* rows, const int* row_list, int n_list,
                              const float* pool, float* wts, cudaStream_t st) {
    if (n_list <= 0) return cudaSuccess;
    dev::k_tc_weights<<<n_list, 256, 0, st>>>(sigs, rows, row_list, pool, wts);
    return cudaGetLastError();
}

// Operand tables of columns M = 2^log2M and KC blocks: tc_table_blocks(log2M)
// tables of tc_table_bytes() each.
size_t tc_table_bytes() { return (size_t)dev::kTcTabBytes; }
int tc_table_blocks(int log2M) { return log2M >= 10 ? 1 << (log2M - 9) : 1; }
cudaError_t launch_tc_tables(int log2M, int KC, int log2R, unsigned char* out, cudaStream_t st) {
    dev::k_tc_tables<<<tc_table_blocks(log2M), 512, 0, st>>>(log2M, KC, 1 << log2R, out);
    return cudaGetLastError();
}

template <int OT, int R>
cudaError_t tc_configure_one() {
    return cudaFuncSetAttribute(dev::k_row_tc<OT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)dev::kTcSmemBytes);
}

template <int R>
cudaError_t tc_configure_r() {
    cudaError_t e = cudaSuccess;
    for (cudaError_t r : {tc_configure_one<OUT_C64, R>(), tc_configure_one<OUT_BF16, R>(), tc_configure_one<OUT_F16, R>(),
                          tc_configure_one<OUT_POWER, R>(), tc_configure_one<OUT_DB, R>()})
        if (r != cudaSuccess && e == cudaSuccess) e = r;
    return e;
}

cudaError_t tc_configure() {
    const cudaError_t e = tc_configure_r<16>();
    return e != cudaSuccess ? e : tc_configure_r<8>();
}

template <int R>
cudaError_t launch_tc_r(const TcParams& p, int out_type, int grid, cudaStream_t st) {
    auto kernel = out_type == OUT_BF16    ? dev::k_row_tc<OUT_BF16, R>
                  : out_type == OUT_F16   ? dev::k_row_tc<OUT_F16, R>
                  : out_type == OUT_POWER ? dev::k_row_tc<OUT_POWER, R>
                  : out_type == OUT_DB    ? dev::k_row_tc<OUT_DB, R>
                                          : dev::k_row_tc<OUT_C64, R>;
    return launch_dependent(kernel, dim3((unsigned)grid), dim3(dev::kTcThreads), (size_t)dev::kTcSmemBytes, st, p);
}

cudaError_t launch_tc(const TcParams& p, int log2R, int out_type, int grid, cudaStream_t st) {
    return log2R == 4 ? launch_tc_r<16>(p, out_type, grid, st) : launch_tc_r<8>(p, out_type, grid, st);
}

}  // namespace fcwt
