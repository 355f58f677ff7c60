// jci_fci_dense.cu -- the same-spin part of the one-group sigma as two dense
// matrix products, for short string lists.
//
//   S += H_alpha C + C H_beta + hd * C
// with H_spin[I][J] the same-spin singles (their part that does not depend on
// the other spin's string, hmatels_1x) and doubles (hmatels_2xaa) of the spin's
// strings, zero on the diagonal (mpi_source/action_util.c:210-245), and hd the
// diagonal of the whole Hamiltonian.  N strings make 2 N multiply-adds a
// determinant where the lists hold some s + d of them (350 of 504 at
// CAS(10,10), 522 of 1 848 at FCI(12,12)), but as a product they run on the
// FP64 tensor cores (mma.sync m8n8k4) with operands from shared memory, while
// the list kernels wait on a table load for every term.  FP32 operands are
// widened, so its sums are exact to FP64.  Measured, FP64, against the row
// kernel: 126 strings of each spin 10 us for 44, 252 16 for 66, 924 142 for 512
// (group kernel, transposes and stream of plan 7 there: 240); the tensor cores
// alone would take 85 of the 142.
#include <cuda_pipeline.h>

#include <algorithm>

#include "jci_internal.h"
#include "jci_kernels.cuh"

namespace jci {

namespace {

constexpr int kDPad = 32;         // rows of H are padded to this
constexpr int kDFlush = 128;      // k per partial sum

constexpr int kDKC = 32;          // k per staged chunk

// Chunks in flight: two leave room for three CTAs of the widest tile per SM
// (four of 16 measured the same: 142 to 150 us at FCI(12,12)).
__host__ __device__ constexpr int dense_stages(int bm) { return bm == 64 ? 2 : 3; }

template <typename T>
struct DenseArgs {
    int na, nb, lda, ldb;         // strings; leading dimensions of H
    const T *Ha, *Hb;             // [na][lda], [nb][ldb], zero-padded to lda / ldb
    const T *hd;
    int vec;                      // rows of C start on 16 bytes
    const int *skip;
};

__device__ __forceinline__ void dense_dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Row strides in shared memory: fragment loads (8 rows of A x 4 k; 4 k of B x
// 8 columns) fall in distinct banks.
constexpr int kDAS = kDKC + 4;
template <typename T, int BN>
constexpr int kDBS = BN + (sizeof(T) == 8 ? 4 : 8);

// The sum of one element over the nonzero elements of H alone.
template <typename T>
__device__ __noinline__ double dense_linked(const DenseArgs<T> &a, const T *C, int r, int c) {
    double sum = 0.0;
    for (int k = 0; k < a.na; k++) {
        const T h = a.Ha[(long long)r * a.lda + k];
        if (h != T(0)) sum = fma((double)h, (double)C[(long long)k * a.nb + c], sum);
    }
    for (int k = 0; k < a.nb; k++) {
        const T h = a.Hb[(long long)k * a.ldb + c];
        if (h != T(0)) sum = fma((double)C[(long long)r * a.nb + k], (double)h, sum);
    }
    return sum;
}

// Output tile 8 MT WM x 16 NT: each of the WM x 2 warps 8 MT x 8 NT; k runs over
// the alpha strings (A = H_alpha, B = C), then the beta strings (A = C,
// B = H_beta), chunks pipelined with cp.async.  32 x 32 tiles take eight warps
// (462 strings 36 us, 40 with four), 64 x 32 tiles four (924 strings 142 us, 146
// with eight).
template <typename T, int MT, int NT, int WM>
__global__ void __launch_bounds__(64 * WM)
    k_same_dense(DenseArgs<T> a, const T *__restrict__ C, T *__restrict__ S) {
    if (a.skip && *a.skip) return;
    constexpr int NTH = 64 * WM, BM = 8 * MT * WM, BN = 16 * NT, AS = kDAS, BS = kDBS<T, BN>;
    constexpr int KC = kDKC, ST = dense_stages(BM);
    constexpr int VE = 16 / sizeof(T);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *As = reinterpret_cast<T *>(smem_raw);   // [ST][BM][AS]
    T *Bs = As + ST * BM * AS;                 // [ST][KC][BS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wm = warp >> 1, wn = warp & 1;
    const int i0 = blockIdx.y * BM, j0 = blockIdx.x * BN;
    const int ka = (a.na + KC - 1) / KC, kb = (a.nb + KC - 1) / KC;
    // rows r0 .. + rows of src (row length len, nr rows in all), columns
    // c0 .. + cols, to dst; zeros outside
    auto load = [&](T *dst, int stride, int rows, int cols, const T *src, int r0, int nr, int c0,
                    int len, long long ld, bool vec) {
        if (vec) {
            const int per = cols / VE;
            for (int idx = tid; idx < rows * per; idx += NTH) {
                const int r = idx / per, c = VE * (idx - r * per);
                T *d = dst + r * stride + c;
                if (r0 + r < nr && c0 + c < len)  // len is a multiple of VE
                    __pipeline_memcpy_async(d, src + (long long)(r0 + r) * ld + c0 + c, 16);
                else
                    *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
            }
        } else {
            for (int idx = tid; idx < rows * cols; idx += NTH) {
                const int r = idx / cols, c = idx - r * cols;
                T *d = dst + r * stride + c;
                if (r0 + r < nr && c0 + c < len)
                    __pipeline_memcpy_async(d, src + (long long)(r0 + r) * ld + c0 + c, sizeof(T));
                else
                    *d = T(0);
            }
        }
    };
    auto stage = [&](int kc, int buf) {
        T *A = As + buf * BM * AS, *B = Bs + buf * KC * BS;
        if (kc < ka) {
            const int k0 = kc * KC;
            load(A, AS, BM, KC, a.Ha, i0, a.na, k0, a.lda, a.lda, true);
            load(B, BS, KC, BN, C, k0, a.na, j0, a.nb, a.nb, a.vec);
        } else {
            const int k0 = (kc - ka) * KC;
            load(A, AS, BM, KC, C, i0, a.na, k0, a.nb, a.nb, a.vec);
            load(B, BS, KC, BN, a.Hb, k0, a.nb, j0, a.ldb, a.ldb, true);
        }
    };
    // partial sums of kDFlush terms, added up apart: one chain over a row's
    // some hundred nonzero terms would round more often than the lists' sums,
    // which the list kernels cut in pieces
    double acc[MT][NT][2], total[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) acc[i][n][e] = total[i][n][e] = 0.0;
#pragma unroll
    for (int i = 0; i < ST - 1; i++) {
        if (i < ka + kb) stage(i, i);
        __pipeline_commit();
    }
    for (int kc = 0; kc < ka + kb; kc++) {
        if (kc % (kDFlush / KC) == 0) {
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        total[i][n][e] += acc[i][n][e];
                        acc[i][n][e] = 0.0;
                    }
        }
        // chunk kc has arrived, and all warps are done with chunk kc - 1, whose
        // buffer the next load goes to
        __pipeline_wait_prior(ST - 2);
        __syncthreads();
        const int next = kc + ST - 1, buf = kc % ST;
        if (next < ka + kb) stage(next, next % ST);
        __pipeline_commit();
        const T *ap = As + buf * BM * AS + (8 * MT * wm + g) * AS + t;
        const T *bp = Bs + buf * KC * BS + t * BS + 8 * NT * wn + g;
#pragma unroll
        for (int k = 0; k < KC; k += 4) {
            double av[MT], bv[NT];
#pragma unroll
            for (int i = 0; i < MT; i++) av[i] = (double)ap[8 * i * AS + k];
#pragma unroll
            for (int n = 0; n < NT; n++) bv[n] = (double)bp[k * BS + 8 * n];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int n = 0; n < NT; n++) dense_dmma(acc[i][n], av[i], bv[n]);
        }
    }
    // accumulator layout: lane holds row g, columns 2t and 2t+1 of a tile
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const int r = i0 + 8 * (MT * wm + i) + g;
        if (r >= a.na) continue;
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int c = j0 + 8 * (NT * wn + n) + 2 * t + e;
                if (c >= a.nb) continue;
                const long long o = (long long)r * a.nb + c;
                double sum = total[i][n][e] + acc[i][n][e];
                // An infinity or NaN of a determinant that H does not reach
                // must not come in through a product with zero.
                if (!isfinite(sum)) sum = dense_linked(a, C, r, c);
                S[o] = (T)((double)S[o] + fma((double)a.hd[o], (double)C[o], sum));
            }
    }
}

// H of one spin from the [e][string] tables (H zeroed before); one warp per
// string.
__global__ void __launch_bounds__(128)
    k_same_fill(int nstr, int ns, int nd, const uint32_t *__restrict__ fs,
                const double *__restrict__ a1T, const int *__restrict__ dblJ,
                const double *__restrict__ dblH, int ld, double *H, float *Hf) {
    const int s = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= nstr) return;
    const long long row = (long long)s * ld;
    for (int e = lane; e < ns; e += 32) {
        const long long o = (long long)e * nstr + s;
        const uint32_t x = fs[o];
        const double h = (x >> 31) ? -a1T[o] : a1T[o];
        H[row + (x & 0x3fffffffu)] = h;
        Hf[row + (x & 0x3fffffffu)] = (float)h;
    }
    for (int e = lane; e < nd; e += 32) {
        const long long o = (long long)e * nstr + s;
        H[row + dblJ[o]] = dblH[o];
        Hf[row + dblJ[o]] = (float)dblH[o];
    }
}

template <typename T, int MT, int NT, int WM>
jci_status dense_launch_t(const DenseArgs<T> &a, const T *x, T *y, cudaStream_t st) {
    constexpr int BM = 8 * MT * WM, BN = 16 * NT;
    const size_t smem = dense_stages(BM) *
                        (size_t)(BM * kDAS + kDKC * kDBS<T, BN>) * sizeof(T);
    JCI_CUDA(smem_optin(k_same_dense<T, MT, NT, WM>));
    dim3 g((a.nb + BN - 1) / BN, (a.na + BM - 1) / BM);
    k_same_dense<T, MT, NT, WM><<<g, 64 * WM, smem, st>>>(a, x, y);
    JCI_CUDA(cudaGetLastError());
    return JCI_OK;
}

}  // namespace

jci_status same_dense_build(SameDense *t, int spin, int nstr) {
    t->n[spin] = nstr;
    t->ld[spin] = (nstr + kDPad - 1) / kDPad * kDPad;
    const size_t n = (size_t)nstr * t->ld[spin];
    JCI_CUDA(cudaMalloc(&t->H64[spin], n * sizeof(double)));
    JCI_CUDA(cudaMalloc(&t->H32[spin], n * sizeof(float)));
    return JCI_OK;
}

void same_dense_free(SameDense *t) {
    for (int sp = 0; sp < 2; sp++) {
        cudaFree(t->H64[sp]);
        cudaFree(t->H32[sp]);
    }
    cudaFree(t->zero);
    *t = SameDense();
}

jci_status same_dense_fill(SameDense *t, int spin, int ns, int nd, const uint32_t *fs,
                           const double *a1T, const int *dblJ, const double *dblH,
                           cudaStream_t st) {
    const size_t n = (size_t)t->n[spin] * t->ld[spin];
    JCI_CUDA(cudaMemsetAsync(t->H64[spin], 0, n * sizeof(double), st));
    JCI_CUDA(cudaMemsetAsync(t->H32[spin], 0, n * sizeof(float), st));
    k_same_fill<<<(t->n[spin] + 3) / 4, 128, 0, st>>>(t->n[spin], ns, nd, fs, a1T, dblJ, dblH,
                                                     t->ld[spin], t->H64[spin], t->H32[spin]);
    JCI_CUDA(cudaGetLastError());
    return JCI_OK;
}

// y += the same-spin part of H x and the diagonal.
template <typename T>
jci_status same_dense_launch(const SameDense &t, const T *hd, const int *skip, int device,
                             const T *x, T *y, cudaStream_t st) {
    DenseArgs<T> a;
    a.na = t.n[0]; a.nb = t.n[1]; a.lda = t.ld[0]; a.ldb = t.ld[1];
    if constexpr (sizeof(T) == 8) {
        a.Ha = t.H64[0];
        a.Hb = t.H64[1];
    } else {
        a.Ha = t.H32[0];
        a.Hb = t.H32[1];
    }
    a.hd = hd;
    a.vec = (size_t)a.nb * sizeof(T) % 16 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
    a.skip = skip;
    int nsm = 0;
    JCI_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    // the widest tile that still gives every SM two CTAs (their k loops are
    // then bound by the tensor pipe, not by latency), or else the smallest
    auto ctas = [&](int bm, int bn) {
        return (long long)((a.na + bm - 1) / bm) * ((a.nb + bn - 1) / bn);
    };
    if (ctas(64, 32) >= 2 * nsm) return dense_launch_t<T, 4, 2, 2>(a, x, y, st);
    if (ctas(32, 32) >= nsm) return dense_launch_t<T, 1, 2, 4>(a, x, y, st);
    return dense_launch_t<T, 1, 2, 2>(a, x, y, st);
}

template jci_status same_dense_launch<double>(const SameDense &, const double *, const int *, int,
                                              const double *, double *, cudaStream_t);
template jci_status same_dense_launch<float>(const SameDense &, const float *, const int *, int,
                                             const float *, float *, cudaStream_t);

}  // namespace jci
