// Rows of N <= 8192 samples: one CTA per row.
//
// The same products and inverse FFT as the other row engines (src/fcwt/fcwt.cpp:
// 197-311, 418-445 of the reference), for rows that are over in microseconds: the
// CTA weights the row's bins into shared memory, runs the whole inverse FFT there
// (Stockham stages of radix 16, 8, 4 or 2, FP32) and stores the samples in order.
// Time decimation by D folds the spectrum to N / D bins, whose inverse FFT is every
// D-th sample.
//
// Few rows are bound by serial latency (launch, descriptors, bins, three or four
// stages), so there is no work queue and no table is computed in the prologue; many
// rows of N = 8192 by one CTA per SM (512 threads of 128 registers). On the work queue of
// the persistent engine (claim, item, row, signal, 16 input chunks, one warp's column DFT
// in turn) a whole call took: 64 rows of 1000 samples 50 us, now 12; 2000 rows of 2048
// 121, now 44; 1000 of 4096 92, now 48; 1000 of 8192 130, now 97.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fcwt_dev.cuh"
#include "fcwt_fft.cuh"
#include "fcwt_internal.h"

namespace fcwt {
namespace dev {

constexpr int kSmallMaxLog2 = 13;
constexpr int kSmallTabLog2 = 10;

// One entry of padding per 16: the stages' strided writes (stride R) and their
// contiguous reads are then both free of bank conflicts.
__device__ __forceinline__ int small_pos(int i) { return i + (i >> 4); }

// One radix-R stage in place: every thread takes its inputs into registers (at most
// 16 values: blockDim >= L / 16), the CTA waits, and the results go to their places.
// In place a row of 8192 takes 70 KB instead of 139.
template <int R>
__device__ __forceinline__ void small_stage(float2* __restrict__ a, int log2L, int log2Ns, const float2* __restrict__ tw,
                                            int log2N, const float2* __restrict__ ts) {
    constexpr int LR = ilog2c(R);
    constexpr int T = 16 / R;  // butterflies per thread, at most
    const int Lr = 1 << (log2L - LR);
    // w_{Ns R} is a power of two of the root of the table in shared memory, or (the
    // last stage of L > 1024) of w_N
    const int log2T = min(log2L, kSmallTabLog2);
    const bool in_ts = log2Ns + LR <= log2T;
    const int shift = (in_ts ? log2T : log2N) - log2Ns - LR;
    auto root = [&](unsigned e) { return in_ts ? ts[small_pos((int)(e << shift))] : tw_lookup(tw, log2N, e << shift); };
    float2 v[T][R];
#pragma unroll
    for (int i = 0; i < T; i++) {
        const int j = threadIdx.x + i * blockDim.x;
        if (j < Lr) {
            const int k = j & ((1 << log2Ns) - 1);
#pragma unroll
            for (int r = 0; r < R; r++) v[i][r] = a[small_pos(j + r * Lr)];
            if (k > 0) {
                // w^1, 2, 3 and the multiples of w^4 from the table, the others as one product
                float2 w[4];
#pragma unroll
                for (int r = 1; r < (R < 4 ? R : 4); r++) {
                    w[r] = root((unsigned)(r * k));
                    v[i][r] = cmul(v[i][r], w[r]);
                }
#pragma unroll
                for (int r4 = 4; r4 < R; r4 += 4) {
                    const float2 w4 = root((unsigned)(r4 * k));
                    v[i][r4] = cmul(v[i][r4], w4);
#pragma unroll
                    for (int r = 1; r < 4; r++) v[i][r4 + r] = cmul(v[i][r4 + r], cmul(w4, w[r]));
                }
            }
            fft_reg<R, +1>(v[i]);
        }
        asm volatile("" ::: "memory");  // one butterfly after the other: together they spill
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T; i++) {
        const int j = threadIdx.x + i * blockDim.x;
        if (j < Lr) {
            const int k = j & ((1 << log2Ns) - 1);
            const int base = (j - k) * R + k;
#pragma unroll
            for (int m = 0; m < R; m++) a[small_pos(base + (m << log2Ns))] = v[i][m];
        }
    }
    __syncthreads();
}

template <int OT>
__global__ void __launch_bounds__(512) k_rows_small(const SigDesc* __restrict__ sigs, const RowDesc* __restrict__ rows,
                                                    const int* __restrict__ list, const float* __restrict__ pool,
                                                    const __grid_constant__ OutPtrs outs) {
    extern __shared__ float2 small_sm[];
    __shared__ RowDesc R;
    __shared__ SigDesc S;
    {
        const int r = list ? list[blockIdx.x] : (int)blockIdx.x;
        const int* src = reinterpret_cast<const int*>(rows + r);
        const int* ssrc = reinterpret_cast<const int*>(sigs + rows[r].sig);
        for (int i = threadIdx.x; i < (int)(sizeof(RowDesc) / 4); i += blockDim.x) reinterpret_cast<int*>(&R)[i] = src[i];
        for (int i = threadIdx.x; i < (int)(sizeof(SigDesc) / 4); i += blockDim.x) reinterpret_cast<int*>(&S)[i] = ssrc[i];
    }
    __syncthreads();
    const int log2N = S.log2N;
    const int N = 1 << log2N;
    const int log2D = 31 - __clz(R.dec);
    const int log2L = log2N > log2D ? log2N - log2D : 0;
    const int L = 1 << log2L;
    // Factors of the stages, in shared memory up to w_1024: read from global memory, the
    // strided entries of the middle stages are a line each (8000 x 2000: 223 us).
    __shared__ float2 ts[(1 << kSmallTabLog2) + (1 << kSmallTabLog2) / 16];
    const int log2T = min(log2L, kSmallTabLog2);
    for (int j = threadIdx.x; j < 1 << log2T; j += blockDim.x) ts[small_pos(j)] = tw_lookup(S.tw, log2N, (unsigned)j << (log2N - log2T));
    float2* a = small_sm;
    grid_dep_wait();  // (what follows reads the spectrum)
    const float nm1 = (float)N - 1.0f;
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        float2 z = make_float2(0.0f, 0.0f);
        for (int q = i; q < R.hi; q += L)
            if (q >= R.lo) z = cadd(z, bin_value(R, S, pool, nm1, q));
        a[small_pos(i)] = z;
    }
    __syncthreads();
    int log2Ns = 0;
    while (log2Ns < log2L) {
        const int rem = log2L - log2Ns;
        const int stages = (rem + 3) / 4;
        const int lr = (rem + stages - 1) / stages;  // 10 = 4 + 3 + 3: as few stages as possible, evenly
        switch (lr) {
            case 4: small_stage<16>(a, log2L, log2Ns, S.tw, log2N, ts); break;
            case 3: small_stage<8>(a, log2L, log2Ns, S.tw, log2N, ts); break;
            case 2: small_stage<4>(a, log2L, log2Ns, S.tw, log2N, ts); break;
            default: small_stage<2>(a, log2L, log2Ns, S.tw, log2N, ts); break;
        }
        log2Ns += lr;
    }
    void* outb = outs.p[R.out_buf];
    for (int t = threadIdx.x; t < R.n_out; t += blockDim.x) store_out<OT>(outb, R.out_off + t, a[small_pos(t)]);
}

}  // namespace dev

static size_t small_smem(int log2L) {
    const size_t L = (size_t)1 << log2L;
    return (L + L / 16 + 1) * sizeof(float2);
}

template <int OT>
static cudaError_t small_launch(const SigDesc* sigs, const RowDesc* rows, const int* list, int n_list, const float* pool,
                                const OutPtrs& outs, int log2L, cudaStream_t st) {
    // a stage's 16 values per thread, or 8 while that keeps the CTA small (shorter chains)
    const int threads = std::max(64, std::max(std::min(128, 1 << std::max(0, log2L - 3)), 1 << std::max(0, log2L - 4)));
    return launch_dependent(dev::k_rows_small<OT>, dim3((unsigned)n_list), dim3((unsigned)threads), small_smem(log2L),
                            st, sigs, rows, list, pool, outs);
}

// Rows of N <= 8192 in `list` (null: rows 0 .. n_list - 1); log2L: the largest
// transform length N / dec among them.
cudaError_t launch_rows_small(const SigDesc* sigs, const RowDesc* rows, const int* list, int n_list, const float* pool,
                              const OutPtrs& outs, int out_type, int log2L, cudaStream_t st) {
    if (n_list <= 0) return cudaSuccess;
    switch (out_type) {
        case OUT_BF16: return small_launch<OUT_BF16>(sigs, rows, list, n_list, pool, outs, log2L, st);
        case OUT_F16: return small_launch<OUT_F16>(sigs, rows, list, n_list, pool, outs, log2L, st);
        case OUT_POWER: return small_launch<OUT_POWER>(sigs, rows, list, n_list, pool, outs, log2L, st);
        case OUT_DB: return small_launch<OUT_DB>(sigs, rows, list, n_list, pool, outs, log2L, st);
        default: return small_launch<OUT_C64>(sigs, rows, list, n_list, pool, outs, log2L, st);
    }
}

cudaError_t small_configure() {
    cudaError_t e = cudaSuccess;
    const int b = (int)small_smem(dev::kSmallMaxLog2);
    for (cudaError_t r : {cudaFuncSetAttribute(dev::k_rows_small<OUT_C64>, cudaFuncAttributeMaxDynamicSharedMemorySize, b),
                          cudaFuncSetAttribute(dev::k_rows_small<OUT_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b),
                          cudaFuncSetAttribute(dev::k_rows_small<OUT_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, b),
                          cudaFuncSetAttribute(dev::k_rows_small<OUT_POWER>, cudaFuncAttributeMaxDynamicSharedMemorySize, b),
                          cudaFuncSetAttribute(dev::k_rows_small<OUT_DB>, cudaFuncAttributeMaxDynamicSharedMemorySize, b)})
        if (r != cudaSuccess && e == cudaSuccess) e = r;
    return e;
}

}  // namespace fcwt
