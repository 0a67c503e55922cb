// Forward (and unnormalised inverse) FFTs of whole signals: the spectrum
// Ihat = FFT_N(zero-padded signal) that every row of the transform reads
// (replaces fftwf r2c / c2c FORWARD, src/fcwt/fcwt.cpp:486-500, and the
// conjugate mirror of fcwt.cpp:507-510).
//
// A length-C complex FFT (C = 2^p) runs as one or two passes through global
// memory (L2-resident at these sizes); inside a pass each CTA transforms a
// tile of B columns x L points in shared memory with radix-16/8/4/2 Stockham
// stages:
//   p <= 12: one pass, the whole signal in one CTA;
//   p >= 13: C = C1 C2, j = j1 + C1 j2, k = k2 + C2 k1 (four-step):
//     pass A  for each j1, the C2-point DFT over j2, times w_C^{j1 k2}
//             -> T[j1 + C1 k2];
//     pass B  for each k2, the C1-point DFT over j1 -> Z[k2 + C2 k1].
// Columns are interleaved in shared memory (element i of column cc at
// i B + cc) so that the B columns of a tile are read and written as B
// consecutive elements of global memory.
//
// A real signal of N = 2C samples is transformed as the C-point FFT of its
// sample pairs z[j] = x[2j] + i x[2j+1], whose last pass splits it into the bins
// up to N / 2 of the real signal. Complex inputs and the inverse transforms run the C = N
// complex FFT.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fcwt_dev.cuh"
#include "fcwt_fft.cuh"
#include "fcwt_internal.h"

namespace fcwt {
namespace dev {

constexpr int kFftThreads = 128;
constexpr int kFftMaxLog2Tile = 12;  // B L <= 4096 complex values per CTA (2 x 32 KB)
constexpr int kFftSmemBytes = 2 * (1 << kFftMaxLog2Tile) * 8;
constexpr int kFftTargetCtas = 2 * 148;  // about two CTAs per SM of a B200

// Element idx of a signal with implicit zero padding: a complex sample, or
// (r2c) the real pair (x[2 idx], x[2 idx + 1]).
__device__ __forceinline__ float2 fwd_input(const float* __restrict__ in_r, const float2* __restrict__ in_c,
                                            const float* __restrict__ gain, int n_in, int idx, int r2c) {
    if (in_r && r2c) {
        const int i0 = 2 * idx;
        return make_float2(i0 < n_in ? __ldg(in_r + i0) : 0.0f, i0 + 1 < n_in ? __ldg(in_r + i0 + 1) : 0.0f);
    }
    if (idx >= n_in) return make_float2(0.0f, 0.0f);
    if (in_r) return make_float2(__ldg(in_r + idx), 0.0f);
    const float2 v = __ldg(in_c + idx);
    return gain ? cscale(v, 2.0f * __ldg(gain + idx)) : v;
}

// w_T^{SIGN e} from the two-level table of T = 2^log2T (which holds w_T^{+e}).
template <int SIGN>
__device__ __forceinline__ float2 fft_tw(const float2* __restrict__ tw, int log2T, unsigned e) {
    float2 w = tw_lookup(tw, log2T, e);
    if (SIGN < 0) w.y = -w.y;
    return w;
}

// Stage twiddles of a CTA: w_L^{SIGN j} for j < min(L, 1024); for longer L the factors
// w_L^{SIGN 1024 j} follow. Each is computed (2 j / L is exact), not looked up: the
// table of N gives most of them as products of two rounded factors, and the stages
// multiply them once more (smem_stage).
constexpr int kStageTw = 1024 + (1 << kFftMaxLog2Tile) / 1024;
template <int SIGN>
__device__ __forceinline__ void stage_tw_fill(float2* __restrict__ tl, int log2L) {
    const int n = log2L <= 10 ? 1 << log2L : 1024 + (1 << (log2L - 10));
    const float step = 2.0f / (float)(1 << log2L);
    for (int t = threadIdx.x; t < n; t += kFftThreads) {
        float sn, cs;
        sincospif((float)(t < 1024 ? t : (t - 1024) << 10) * step, &sn, &cs);
        tl[t] = make_float2(cs, SIGN < 0 ? -sn : sn);
    }
}
__device__ __forceinline__ float2 stage_tw(const float2* __restrict__ tl, unsigned e) {
    return e < 1024u ? tl[e] : cmul(tl[e & 1023u], tl[1024 + (e >> 10)]);
}

// One radix-R Stockham stage over L = 2^log2L points of B = 2^log2B
// interleaved columns: k = j mod Ns, v_r = in[j + r L/R] w_{Ns R}^{SIGN r k},
// V = DFT_R(v), out[(j - k) R + k + m Ns] = V_m.
template <int R, int SIGN>
__device__ __forceinline__ void smem_stage(const float2* __restrict__ in, float2* __restrict__ out, int log2L,
                                           int log2B, int log2Ns, const float2* __restrict__ tl) {
    constexpr int LR = ilog2c(R);
    const int B = 1 << log2B;
    const int Lr = 1 << (log2L - LR);
    const int tasks = Lr << log2B;
    const int shift = log2L - log2Ns - LR;  // w_{Ns R} = w_L^{2^shift}
    for (int t = threadIdx.x; t < tasks; t += kFftThreads) {
        const int cc = t & (B - 1);
        const int j = t >> log2B;
        const int k = j & ((1 << log2Ns) - 1);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = in[((j + r * Lr) << log2B) + cc];
        if (k > 0) {
            // w^1, 2, 3 and the multiples of w^4 from the table, the others as one product
            // (15 lookups of a radix-16 task kept the load unit busy)
            float2 w[4];
#pragma unroll
            for (int r = 1; r < (R < 4 ? R : 4); r++) {
                w[r] = stage_tw(tl, (unsigned)(r * k) << shift);
                v[r] = cmul(v[r], w[r]);
            }
#pragma unroll
            for (int r4 = 4; r4 < R; r4 += 4) {
                const float2 w4 = stage_tw(tl, (unsigned)(r4 * k) << shift);
                v[r4] = cmul(v[r4], w4);
#pragma unroll
                for (int r = 1; r < 4; r++) v[r4 + r] = cmul(v[r4 + r], cmul(w4, w[r]));
            }
        }
        fft_reg<R, SIGN>(v);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int m = 0; m < R; m++) out[((base + (m << log2Ns)) << log2B) + cc] = v[m];
    }
}

// All stages of an L-point FFT on the tile in `a` (natural order in and
// out); returns the buffer that holds the result.
template <int SIGN>
__device__ __forceinline__ float2* smem_fft(float2* a, float2* b, int log2L, int log2B, const float2* __restrict__ tl) {
    int log2Ns = 0;
    while (log2Ns < log2L) {
        const int lr = min(4, log2L - log2Ns);
        switch (lr) {
            case 4: smem_stage<16, SIGN>(a, b, log2L, log2B, log2Ns, tl); break;
            case 3: smem_stage<8, SIGN>(a, b, log2L, log2B, log2Ns, tl); break;
            case 2: smem_stage<4, SIGN>(a, b, log2L, log2B, log2Ns, tl); break;
            default: smem_stage<2, SIGN>(a, b, log2L, log2B, log2Ns, tl); break;
        }
        __syncthreads();
        float2* s = a;
        a = b;
        b = s;
        log2Ns += lr;
    }
    return a;
}

// One pass over a length-2^log2C array of the job blockIdx.y (or `one` when
// jobs is null). The CTA takes columns [B blockIdx.x, B blockIdx.x + B) of
// the S = C / L columns:
//   mode 0 (pass A): column col holds elements col + S i; its results are
//                    multiplied by w_C^{SIGN col k};
//   mode 1 (pass B): column col holds elements col L + i.
// Result k of column col goes to col + S k in both modes. src_sel: 0 = the
// job's input (zero padded; r2c: sample pairs), 2 = its tmp buffer; dst_sel:
// 1 = its spectrum X, 2 = its tmp buffer.
//
// SPLIT (the last pass of a real input's transform, mode 1): the results are
// Z = FFT_{N/2}(z) of the sample pairs, and the CTA writes the spectrum itself. With
// E = (Z[k] + conj Z[N/2-k]) / 2 and O = -i (Z[k] - conj Z[N/2-k]) / 2,
//   X[k] = E + w_N^{-k} O,   X[N/2 - k] = conj(E - w_N^{-k} O);
// bins above N / 2 are conjugates that no reader uses. Bin col + S k pairs with
// bin (S - col) + S (L - 1 - k), so the CTA takes B / 2 columns from
// B / 2 blockIdx.x on and their partners S - col (column 0, whose bins pair among
// themselves, comes with column S / 2, whose bins do too). A split kernel of
// its own cost a call one launch and one pass over the spectrum (with the memsets and
// the copy that went at the same time: 10000 samples x 200 rows 46 -> 40 us a call).
//
// zero: n_zero words to clear for the kernels after the transform.
template <int SIGN, bool SPLIT>
__global__ void __launch_bounds__(kFftThreads) k_fft_cols(const FwdJob* __restrict__ jobs, FwdJob one, int src_sel,
                                                          int dst_sel, int log2C, int log2L, int log2B, int mode,
                                                          int r2c, const float2* __restrict__ tw, int log2T,
                                                          unsigned* __restrict__ zero, int n_zero) {
    extern __shared__ float2 fft_sm[];
    __shared__ float2 tl[kStageTw];
    const FwdJob J = jobs ? jobs[blockIdx.y] : one;
    const int L = 1 << log2L;
    const int B = 1 << log2B;
    const int log2S = log2C - log2L;
    const int tot = L << log2B;
    const int log2H = SPLIT && log2S > 0 ? log2B - 1 : log2B;  // columns of the CTA's own, without the partners
    const int c0 = blockIdx.x << log2H;
    grid_dep_launch();
    if (zero && blockIdx.x == 0 && blockIdx.y == 0)
        for (int t = threadIdx.x; t < n_zero; t += kFftThreads) zero[t] = 0;
    float2* a = fft_sm;
    float2* b = fft_sm + tot;
    const float2* src = J.tmp;
    stage_tw_fill<SIGN>(tl, log2L);
    grid_dep_wait();  // (pass B: pass A's results)
    for (int t = threadIdx.x; t < tot; t += kFftThreads) {
        int i, cc;
        if (mode == 0) {
            cc = t & (B - 1);
            i = t >> log2B;
        } else {
            i = t & (L - 1);
            cc = t >> log2L;
        }
        int col = c0 + cc;
        if (SPLIT && (cc >> log2H)) {
            const int own = col - (1 << log2H);
            col = own == 0 ? 1 << (log2S - 1) : (1 << log2S) - own;
        }
        const int j = mode == 0 ? col + (i << log2S) : (col << log2L) + i;
        a[(i << log2B) + cc] = src_sel == 0 ? fwd_input(J.in_r, J.in_c, J.gain, J.n, j, r2c) : src[j];
    }
    __syncthreads();
    const float2* res = smem_fft<SIGN>(a, b, log2L, log2B, tl);
    if constexpr (SPLIT) {
        const int C = 1 << log2C;
        auto emit = [&](int q, float2 A, float2 Bz) {
            const float2 E = make_float2(0.5f * (A.x + Bz.x), 0.5f * (A.y - Bz.y));
            const float2 O = make_float2(0.5f * (A.y + Bz.y), -0.5f * (A.x - Bz.x));
            const float2 wo = cmul(fft_tw<SIGN>(tw, log2T, (unsigned)q), O);
            const float2 xk = make_float2(E.x + wo.x, E.y + wo.y);
            const float2 yk = make_float2(E.x - wo.x, wo.y - E.y);
            J.X[q] = xk;
            if (J.log2R) J.Xp[perm_bin(q, J.log2R)] = xk;
            if (2 * q == C) return;
            J.X[C - q] = yk;
            if (J.log2R && q > 0) J.Xp[perm_bin(C - q, J.log2R)] = yk;
        };
        if (log2S == 0) {
            for (int k = threadIdx.x; k <= L / 2; k += kFftThreads) emit(k, res[k], res[(L - k) & (L - 1)]);
            return;
        }
        for (int t = threadIdx.x; t < L << log2H; t += kFftThreads) {
            const int cc = t & ((1 << log2H) - 1);
            const int k = t >> log2H;
            const int col = c0 + cc;
            const float2* own = res + cc;
            const float2* par = own + (1 << log2H);
            if (col > 0) {
                emit(col + (k << log2S), own[k << log2B], par[(L - 1 - k) << log2B]);
            } else if (k < L / 2) {
                emit(k << log2S, own[k << log2B], own[((L - k) & (L - 1)) << log2B]);
            } else {
                const int k2 = k - L / 2;
                emit((1 << (log2S - 1)) + (k2 << log2S), par[k2 << log2B], par[(L - 1 - k2) << log2B]);
                if (k2 == 0) emit(C / 2, own[(L / 2) << log2B], own[(L / 2) << log2B]);
            }
        }
        return;
    }
    float2* dst = dst_sel == 1 ? J.X : J.tmp;
    // Inter-pass twiddle w_C^{SIGN col k}, looked up at each sample. (Stepped by a product
    // with lookups every four samples, the gradient of 8 x 40000 x 64 took 1.10 ms with its
    // forward instead of 1.14 but was off by 3.9e-7 of its size instead of 3.5e-7; a call of
    // 99991 x 300 takes 177 us either way.)
    for (int t = threadIdx.x; t < tot; t += kFftThreads) {
        const int cc = t & (B - 1);
        const int k = t >> log2B;
        const int col = c0 + cc;
        float2 v = res[t];
        if (mode == 0) v = cmul(v, fft_tw<SIGN>(tw, log2T, (unsigned)(col * k) << (log2T - log2C)));
        const int o = col + (k << log2S);
        dst[o] = v;
        if (dst_sel == 1 && J.log2R && o < (1 << (log2C - 1))) J.Xp[perm_bin(o, J.log2R)] = v;
    }
}

// ---- adjoint of the differentiable transform, N > 16384: pass B of the incoming
// gradient rows' FFTs and their use in one kernel. A CTA takes B columns k2 of
// the rows [r0, r0 + rows) of signal blockIdx.y: it transforms each row's columns
// in shared memory and adds, for its bins q = k2 + C2 k1 < N / 2, g_i(q) Ghat to H
// (in registers over its rows) and the sigma and frequency partial sums, so the
// rows' spectra are never written. (Writing them and reading them back took the
// second pass 43 us and the sums 11 us per 64 rows of N = 65536.)
// The CTAs of one bin tile, blockIdx.z, keep sums of their own: z = 0 in H, the others
// in part[z - 1], which the launches of one backward pass carry on (`first`: start at
// zero) and k_adjoint_hsum adds in the order of z. So the same call gives the same
// bits; with float atomics into H the order of the additions varied.
constexpr int kAdjColPos = (1 << kFftMaxLog2Tile) / 2 / kFftThreads;  // bins per thread, at most

__global__ void __launch_bounds__(kFftThreads)
    k_adjoint_cols(const float2* __restrict__ T, const float2* __restrict__ Xs, const float2* __restrict__ rowc,
                   int rows_total, int rows_per_cta, int log2C, int log2L, int log2B, const float2* __restrict__ tw,
                   float cb, float amp, float inv_sigma, float2* __restrict__ H, float2* __restrict__ part, int first,
                   double* __restrict__ acc_sigma, double* __restrict__ acc_f) {
    extern __shared__ float2 fft_sm[];
    __shared__ float2 tl[kStageTw];
    __shared__ float s_red[kFftThreads / 32][2];
    const int L = 1 << log2L, B = 1 << log2B;
    const int log2S = log2C - log2L;
    const int tot = L << log2B;
    const int pos = tot >> 1;  // bins below N / 2
    const int c0 = blockIdx.x << log2B;
    const int b = blockIdx.y;
    const int r0 = blockIdx.z * rows_per_cta;
    const int nr = min(rows_per_cta, rows_total - r0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2* hsum = blockIdx.z == 0 ? H + ((size_t)b << log2C)
                                   : part + (((size_t)(blockIdx.z - 1) * gridDim.y + b) << (log2C - 1));
    stage_tw_fill<-1>(tl, log2L);
    float2 h[kAdjColPos], xq[kAdjColPos];
#pragma unroll
    for (int i = 0; i < kAdjColPos; i++) {
        const int t = threadIdx.x + i * kFftThreads;
        h[i] = make_float2(0.0f, 0.0f);
        if (t < pos) {
            const int q = c0 + (t & (B - 1)) + ((t >> log2B) << log2S);
            xq[i] = __ldg(Xs + ((size_t)b << log2C) + q);
            if (!first) h[i] = hsum[q];
        }
    }
    double dsig = 0.0;
    for (int r = 0; r < nr; r++) {
        const float2* __restrict__ src = T + (((size_t)b * rows_total + r0 + r) << log2C) + ((size_t)c0 << log2L);
        float2* a = fft_sm;
        __syncthreads();
        for (int t = threadIdx.x; t < tot; t += kFftThreads) a[((t & (L - 1)) << log2B) + (t >> log2L)] = __ldcg(src + t);
        __syncthreads();
        const float2* res = smem_fft<-1>(a, fft_sm + tot, log2L, log2B, tl);
        const float2 rc = __ldg(rowc + r0 + r);  // (ca, dfdq)
        float ds = 0.0f, df = 0.0f;
#pragma unroll
        for (int i = 0; i < kAdjColPos; i++) {
            const int t = threadIdx.x + i * kFftThreads;
            if (t < pos) {
                const float qf = (float)(c0 + (t & (B - 1)) + ((t >> log2B) << log2S));
                const float u = rc.x * qf - cb;
                const float g = amp * expf(-0.5f * u * u);
                const float2 gh = res[t];
                h[i].x += g * gh.x;
                h[i].y += g * gh.y;
                const float re = xq[i].x * gh.x + xq[i].y * gh.y;  // Re(X conj(Gh))
                ds += -g * u * u * inv_sigma * re;
                df += g * u * rc.y * qf * re;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ds += __shfl_xor_sync(0xffffffffu, ds, o);
            df += __shfl_xor_sync(0xffffffffu, df, o);
        }
        if (lane == 0) {
            s_red[warp][0] = ds;
            s_red[warp][1] = df;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double d = 0.0;
            for (int w = 0; w < kFftThreads / 32; w++) {
                dsig += (double)s_red[w][0];
                d += (double)s_red[w][1];
            }
            atomicAdd(acc_f + r0 + r, d);
        }
    }
    if (threadIdx.x == 0) atomicAdd(acc_sigma, dsig);
#pragma unroll
    for (int i = 0; i < kAdjColPos; i++) {
        const int t = threadIdx.x + i * kFftThreads;
        if (t < pos) hsum[c0 + (t & (B - 1)) + ((t >> log2B) << log2S)] = h[i];
    }
}

// H += part[0] + part[1] + ... in this order, two bins per thread.
__global__ void k_adjoint_hsum(float2* __restrict__ H, const float2* __restrict__ part, int nparts, int log2N) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 1 << (log2N - 2)) return;
    const size_t stride = (size_t)gridDim.y << (log2N - 2);
    const float4* p = reinterpret_cast<const float4*>(part) + ((size_t)blockIdx.y << (log2N - 2)) + i;
    float4* hp = reinterpret_cast<float4*>(H) + ((size_t)blockIdx.y << (log2N - 1)) + i;
    float4 h = *hp;
#pragma unroll 4
    for (int z = 0; z < nparts; z++) {
        const float4 v = __ldcg(p + z * stride);
        h.x += v.x;
        h.y += v.y;
        h.z += v.z;
        h.w += v.w;
    }
    *hp = h;
}

}  // namespace dev

cudaError_t fft_configure() {
    cudaError_t e = cudaFuncSetAttribute(dev::k_fft_cols<-1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         dev::kFftSmemBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(dev::k_adjoint_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, dev::kFftSmemBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(dev::k_fft_cols<-1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dev::kFftSmemBytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(dev::k_fft_cols<+1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, dev::kFftSmemBytes);
}

// FFTs of njobs signals of length N = 2^log2N (jobs in device memory, or
// `one` for a single signal). SIGN -1: forward, real inputs (real) as r2c
// when N >= 4, result in each job's X (complex inputs: all N bins, real ones: the
// bins up to N / 2); SIGN +1: unnormalised inverse of complex inputs. zero: n_zero words
// that the first kernel clears. tw: the two-level table of N.
template <int SIGN>
static cudaError_t fft_signals(const FwdJob* jobs, const FwdJob& one, int njobs, int log2N, const float2* tw,
                               bool real, cudaStream_t st, int* n_kernels, unsigned* zero = nullptr, int n_zero = 0) {
    *n_kernels = 0;
    if (njobs <= 0) return cudaSuccess;
    if (log2N < 1) return cudaErrorInvalidValue;
    const int r2c = (SIGN < 0 && real && log2N >= 2) ? 1 : 0;
    const int log2C = log2N - r2c;
    auto pass = [&](int src, int dst, int log2L, int mode) -> cudaError_t {
        const int log2cols = log2C - log2L;
        // B = 2^log2B columns per CTA: at most 4096 / L, at most 8, and no more
        // than leaves about two CTAs per SM when there are enough columns (down to two:
        // one signal of 131072 is bound by latency; with four columns at least, a call of
        // 99991 x 300 took 183 us, with two 180)
        const bool split = r2c && dst == 1;
        int log2B = std::min(3, std::min(dev::kFftMaxLog2Tile - log2L, log2cols));
        while (log2B > 1 && ((long long)njobs << (log2cols - log2B)) < dev::kFftTargetCtas) log2B--;
        // (the split takes columns in pairs: log2B >= 1 unless there is one column)
        const int tile = 1 << (log2L + log2B);
        dim3 grid(1u << (log2cols - log2B), (unsigned)njobs);
        unsigned* z = *n_kernels == 0 ? zero : nullptr;
        auto kernel = dev::k_fft_cols<SIGN, false>;
        if constexpr (SIGN < 0) {
            if (split) kernel = dev::k_fft_cols<SIGN, true>;
        }
        (*n_kernels)++;
        if (src == 2)
            return launch_dependent(kernel, grid, dim3(dev::kFftThreads), (size_t)tile * 16, st, jobs, one, src, dst, log2C,
                                    log2L, log2B, mode, r2c, tw, log2N, z, n_zero);
        // (the first pass starts after all that is in the stream: later kernels count on it)
        kernel<<<grid, dev::kFftThreads, (size_t)tile * 16, st>>>(jobs, one, src, dst, log2C, log2L, log2B, mode, r2c, tw,
                                                                  log2N, z, n_zero);
        return cudaGetLastError();
    };
    cudaError_t e;
    if (log2C <= dev::kFftMaxLog2Tile) return pass(0, 1, log2C, 1);
    const int log2C2 = log2C / 2;  // pass A length (C2 <= C1)
    e = pass(0, 2, log2C2, 0);
    return e == cudaSuccess ? pass(2, 1, log2C - log2C2, 1) : e;
}

cudaError_t launch_forward(const float* in_r, const float2* in_c, int n, int log2N, const float2* tw,
                           float2* out, float2* tmp, cudaStream_t st, int* n_kernels, float2* Xp, int log2R,
                           unsigned* zero, int n_zero) {
    *n_kernels = 0;
    if (log2N == 0) {
        // N == 1: the DFT is the identity (one sample or none).
        cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float2), st);
        if (e == cudaSuccess && n_zero > 0) e = cudaMemsetAsync(zero, 0, (size_t)n_zero * sizeof(unsigned), st);
        if (e != cudaSuccess) return e;
        if (n >= 1) {
            if (in_r)
                e = cudaMemcpy2DAsync(out, sizeof(float2), in_r, sizeof(float), sizeof(float), 1,
                                      cudaMemcpyDeviceToDevice, st);
            else
                e = cudaMemcpyAsync(out, in_c, sizeof(float2), cudaMemcpyDeviceToDevice, st);
        }
        return e;
    }
    FwdJob one;
    one.in_r = in_r;
    one.in_c = in_r ? nullptr : in_c;
    one.n = n;
    one.log2R = Xp ? log2R : 0;
    one.X = out;
    one.tmp = tmp;
    one.Xp = Xp;
    one.gain = nullptr;
    return fft_signals<-1>(nullptr, one, 1, log2N, tw, in_r != nullptr, st, n_kernels, zero, n_zero);
}

cudaError_t launch_forward_batched(const FwdJob* jobs, int njobs, int log2N, const float2* tw, cudaStream_t st,
                                   int* n_kernels, bool real, unsigned* zero, int n_zero) {
    FwdJob none{};
    return fft_signals<-1>(jobs, none, njobs, log2N, tw, real, st, n_kernels, zero, n_zero);
}

// Rows a CTA of k_adjoint_cols takes when a launch has `rows` of them: enough CTAs for
// every SM, H read and written once per CTA.
int adjoint_long_rows_per_cta(int log2N, int batch, int rows) {
    const int log2C2 = log2N / 2, log2C1 = log2N - log2C2;
    const int groups = 1 << (log2C2 - std::min(3, dev::kFftMaxLog2Tile - log2C1));
    int per = 1;
    while (per < 16 && per < rows && (long long)groups * batch * ((rows + 2 * per - 1) / (2 * per)) >= 8 * 148) per *= 2;
    return per;
}

// The adjoint's row FFTs for N > 16384: pass A of `njobs` = batch x rows gradient
// rows into consecutive tmp buffers (N values each, from `tmp`), then the fused
// pass B. rowc: (ca, dfdq) of the rows; part: ceil(rows / per) - 1 sums of batch x N / 2
// bins (k_adjoint_cols).
cudaError_t launch_adjoint_long(const FwdJob* jobs, float2* tmp, int batch, int rows, int per, const float2* Xs,
                                const void* rowc, int log2N, const float2* tw, float cb, float amp, float inv_sigma,
                                float2* H, float2* part, bool first, double* acc_sigma, double* acc_f, cudaStream_t st) {
    const int log2C2 = log2N / 2, log2C1 = log2N - log2C2;
    FwdJob none{};
    int log2B = std::min(3, dev::kFftMaxLog2Tile - log2C2);
    dev::k_fft_cols<-1, false><<<dim3(1u << (log2C1 - log2B), (unsigned)(batch * rows)), dev::kFftThreads,
                          (size_t)16 << (log2C2 + log2B), st>>>(jobs, none, 0, 2, log2N, log2C2, log2B, 0, 0, tw, log2N,
                                                                          nullptr, 0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    log2B = std::min(3, dev::kFftMaxLog2Tile - log2C1);
    dev::k_adjoint_cols<<<dim3(1u << (log2C2 - log2B), batch, (rows + per - 1) / per), dev::kFftThreads,
                          (size_t)16 << (log2C1 + log2B), st>>>(tmp, Xs, static_cast<const float2*>(rowc), rows, per, log2N,
                                                                log2C1, log2B, tw, cb, amp, inv_sigma, H, part,
                                                                first ? 1 : 0, acc_sigma, acc_f);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_hsum(float2* H, const float2* part, int nparts, int log2N, int batch, cudaStream_t st) {
    if (nparts <= 0) return cudaSuccess;
    dev::k_adjoint_hsum<<<dim3((1u << (log2N - 2)) / 256, (unsigned)batch), 256, 0, st>>>(H, part, nparts, log2N);
    return cudaGetLastError();
}

cudaError_t launch_inverse_batched(const FwdJob* jobs, int njobs, int log2N, const float2* tw, cudaStream_t st,
                                   int* n_kernels) {
    FwdJob none{};
    return fft_signals<+1>(jobs, none, njobs, log2N, tw, false, st, n_kernels);
}

}  // namespace fcwt
