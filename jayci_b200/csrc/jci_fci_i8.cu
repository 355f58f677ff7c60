// jci_fci_i8.cu -- the alpha-single x beta-single part of sigma (one-group
// spaces) on the 5th-generation tensor cores, by exact integer products of
// operands split into 8-bit digits (the Ozaki scheme: K. Ozaki, T. Ogita,
// S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012) 95; on integer matrix
// units H. Ootomo, K. Ozaki, R. Yokota, IJHPCA 38 (2024) 297).
//
// For one alpha string Ia with alpha singles j -> (Ja_j, phase s_j, pair p_j)
// (hmatels_2xab, action_util.c:250),
//   T[m][Jb] = sum_j A[m][j] c(Ja_j, Jb),  A[m][j] = s_j (p_j | m)
// over the panel rows m, the orbital pairs that the beta singles move; then
// every beta string adds its singles' entries of T to sigma(Ia, .).  (The
// alpha singles of an unchanged beta string are a one-body pass elsewhere.)
//
// Why integers: the product is 2 x 120 x 64 operations a determinant at
// FCI(16,16) and the FP64 tensor pipe retires 64 multiply-adds a clock and
// SM, the int8 pipe 8192.  Every column of the rows that one string's singles
// reach is scaled by a power of two to |x| < 1 and written as NS balanced
// base-256 digits, the integrals likewise (one scale 2^f for the panel in FP64,
// one for each of its rows in FP32), and
//   T = 2^(e_col + f) sum_s 256^-s sum_{u+v=s} A_u B_v
// with each sum over j exact in 32-bit integers (tcgen05.mma kind::i8,
// tensor-memory accumulators, one per s: s < 8 of NS = 7 digits in FP64, s < 4
// of NS = 4 in FP32).
//
// What is left out of T lies some 2^-55 (FP64) or 2^-31 (FP32) below the largest
// integral times the largest element of that sum.  That is a bound for the sum,
// as a floating one has it, in c: an element of sigma feels no element of c that
// H does not connect to it.  In the integrals it is looser: products with an
// integral far below the largest one of the panel (FP32: of its row) are accurate
// to that integral's scale, not to their own.  Measured against 80-bit
// arithmetic, FCI(12,12), a random vector and one with weights over eight
// decades: sigma's relative error is 5.0e-16 and 4.5e-16 in FP64 (FP64
// tensor-core product: 5.1e-16, 4.5e-16), 6.3e-8 and 6.4e-8 in FP32 (3xTF32
// product: 1.3e-7, 1.3e-7); element by element, beside sum_j |H_ij| |c_j|, at
// most 2.1e-15 and 4.6e-7 where three elements stand 1e10 (FP32: 1e6) above the
// others (floating products: 1.1e-15, 4.6e-7; with one scale for a column of all
// strings it was 9.6e-9 and 4.6e-5).
// MMAs of 128 x 48 x 32 with A in tensor memory, issued from several warps,
// take 27 clocks each (one thread's issue alone takes 44; A from shared memory
// makes 48 of reading 6 KB of operands at 128 bytes a clock): 68 of them make
// 128 x 48 x 64 in FP64, 1 840 clocks where the FP64 tensor pipe needs 6 144
// at its peak.
//
// While the integer MMAs run the FP64 units stand nearly still (measured: 2.8
// clocks an operation, warp and SM instead of 0.5).  So T of a chunk of
// columns whose largest elements lie within 2^2 of each other -- then scaled
// by one exponent -- stays an integer (64 bits, the whole sum less 2^-56 of
// the largest product), is gathered by integer adds of 96 bits, and becomes a
// double once per string and chunk.  Other chunks (a few large elements among
// small ones) keep one exponent per column and take T in FP64.
//
// The digits of a row of c are cut once, by the scales of whole columns, for the
// plain strings, whose own largest elements lie near those scales; for the other
// ones, graded, the product cuts c again for each string (k_i8_grade, below).
// Random vectors have plain strings only, CI vectors with weights over decades
// mostly graded ones.
//
// Measured, one sigma of a random vector / of one with weights over decades
// (10^(-0.3 level) and energy denominators), whole call: FCI(16,16) FP64 127 /
// 163 ms, FP32 95 / 106; FCI(14,14) FP64 7.2 / 8.8, FP32 4.9 / 5.3.  (With the
// FP64 tensor-core product through a compact panel and 3xTF32, whatever the
// vector: 232 at FCI(16,16) in FP64, 12.4 and 8.6 at FCI(14,14).)  The plain
// product takes about 5 000 clocks a chunk of 48 columns: the tensor pipe is
// busy for 1 900 to 2 200 of them, the extraction and gather warps issue about
// one instruction in seven clocks each.
//
// An alpha string that reaches an infinity or NaN takes its products with that
// chunk of c in plain floating arithmetic from c itself, and with an infinity or
// NaN among the integrals every string does, so such values spread as they always
// did: to what H connects them to.
#include <cuda_pipeline.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "jci_internal.h"
#include "jci_kernels.cuh"

namespace jci {

namespace {

constexpr int kIC = 48;            // columns per chunk (the MMA's N)
constexpr int kIM = 128;           // panel rows (the MMA's M)
constexpr int kIP = kIC + 1;       // row stride of T in shared memory (odd: no bank conflicts)
constexpr int kIThreads = 1024;
// Warps of each role (32 in all): extract (a multiple of 4, the quarters of
// tensor memory), gather, issue MMAs, load digits (of graded strings: cut them,
// two warps for each 16 columns of a chunk).  Two warps load as fast as six and
// leave four to the gather: FCI(16,16) 126 ms a sigma, 138 with six.
template <typename T, bool GRADED>
struct I8Roles {
    static constexpr int ext = sizeof(T) == 8 ? 8 : 12, iss = sizeof(T) == 8 ? 4 : 2;
    static constexpr int load = GRADED ? 6 : 2, gat = 32 - ext - iss - load;
};
constexpr int kISeg = 8;           // list entries a lane adds at most
constexpr int kIRing = 3;          // buffers of B, of the chunk lists and scales
constexpr int kIZero = (kIM - 1) * kIP + kIC - 1;  // position of an always-zero T element
constexpr int kIEMin = -960;       // least exponent of the integrals' scale
constexpr int kIEBias = 60;        // bias of FP64's scales (8 in FP32)

template <typename T>
constexpr int kDigits = sizeof(T) == 8 ? 7 : 4;
// Sums kept: the digit products with u + v < kSums.  FP64 takes u + v = 7 too
// (34 products): without them they were the largest error by far.
template <int NS>
constexpr int kSums = NS == 7 ? 8 : NS;

constexpr int kISpread = 2;        // largest spread of column exponents of an integer chunk
// A chunk's columns: one exponent (T in integers), one each, or with an
// infinity or NaN.
constexpr int kIOne = 1, kIEach = 0, kIBad = 2;

// 16 bytes of a row of c.
template <typename T>
struct alignas(16) CutVec {
    T v[16 / sizeof(T)];
};

template <typename T>
struct I8Args {
    int na, nb, nchunk, K, KP, nrow;  // KP: K padded to 32 or 64; nrow: panel rows in use
    const uint32_t *fsA;       // [single][Ia] target | phase << 31
    const uint16_t *fpA;       // [single][Ia] pair index
    const T *m2;               // packed (pq|rs)
    const uint8_t *eri;        // [sign][pair][128][8 or 4] digits of +-(pair | row m)
    const T *rscale;           // [128] 2^(f + bias) of row m's integrals, see k_i8_eri
    const int *rowpair;        // [128] pair index of row m, -1 for padding
    int vec;                   // rows of c start on 16 bytes
    const uint8_t *sl;         // [chunk][string][3][NS][16] digits of c, cut by column
    const T *cscale;           // [chunk * 48]
    const uint8_t *flags;      // [string][chunk] kIGraded | kISame, see k_i8_grade
    const int *nstr, *strs;    // numbers of plain and graded strings, [2][na] the strings
    const uint32_t *lofs;      // [chunk + 1] first 16-byte unit of each chunk's lists
    const uint4 *lists;
    int lmax;                  // longest chunk list, in 16-byte units
    int npair;
    int expire;                // test hook: CTA 0 never hands over its first chunk
    const int *skip;
};

__device__ __forceinline__ uint32_t i8_smem(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: start address, leading-dimension byte
// offset (between blocks of 8 k), stride byte offset (between blocks of 16
// m or n), version 1, no swizzle.  Both operands are MN-major: 16 bytes hold
// 16 consecutive m (n) of one k, 8 consecutive k follow each other.
__device__ __forceinline__ uint64_t i8_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::i8: 32-bit integer accumulator, signed A
// (tensor memory, K-major) and B (MN-major), M = 128, N = 48.
constexpr uint32_t kI8Idesc = (2u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                              ((uint32_t)(kIC >> 3) << 17) | ((uint32_t)(kIM >> 4) << 24);

__device__ __forceinline__ void i8_mma(uint32_t d, uint32_t at, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(at), "l"(bd), "r"(kI8Idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ uint64_t i8_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Whether the phase with the given parity has completed.
__device__ __forceinline__ bool i8_test(uint32_t mbar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    return done != 0;
}

// Wait for the phase with the given parity; false after about one second of
// global time (or 2^26 attempts) without completion.  (The clock is read only
// when there is something to wait for.)
__device__ __forceinline__ bool i8_wait(uint32_t mbar, uint32_t parity) {
    if (i8_test(mbar, parity)) return true;
    const uint64_t t0 = i8_ns();
    for (int it = 0; it < (1 << 26); it++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 255) == 255 && i8_ns() - t0 > 1000000000ull) return false;
    }
    return false;
}

// True in one lane of a converged warp.
__device__ __forceinline__ bool i8_elect() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(r));
    return r != 0;
}

__device__ __forceinline__ void i8_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// Barrier of one role's W warps (id 1 or 2); true for all when any of them
// passes pred.
template <int W>
__device__ __forceinline__ bool i8_sync_or(int id, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n"
        " barrier.red.or.pred.aligned q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(id), "n"(32 * W)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void i8_tm_ld(uint32_t addr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void i8_tm_st(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}

// ---- digits -----------------------------------------------------------------

// Least e with max <= 2^e * 127/128 (so that the top digit stays within
// [-127, 127] after the carries of the balanced lower digits), clamped.  The
// integrals are cut on their own; c is cut by the product's warps (i8_cut).
__host__ __device__ inline int i8_exponent(double mx) {
    int e;
    const double f = frexp(mx, &e);  // mx = f 2^e, f in [0.5, 1)
    if (f > 127.0 / 128.0) e++;
    return e < kIEMin ? kIEMin : e;
}

// The NS digits of x 2^-e, most significant first, in the bytes NS-1 .. 0
// of the result: x 2^-e = 2^-7 sum_u digit_u 256^-u to 2^-(8 NS).
template <int NS>
__host__ __device__ inline uint64_t i8_split(double x, int e) {
    const long long v = llrint(ldexp(x, 8 * NS - 1 - e));
    uint64_t carry = 0;
    for (int i = 0; i < NS - 1; i++) carry |= 0x80ull << (8 * i);
    return ((uint64_t)v + carry) ^ carry;
}

// The digits with the most significant one in byte 0.
template <int NS>
__host__ __device__ inline uint64_t i8_bytes(uint64_t w) {
    uint64_t r = 0;
    for (int u = 0; u < NS; u++) r |= ((w >> (8 * (NS - 1 - u))) & 0xff) << (8 * u);
    return r;
}

__device__ __forceinline__ unsigned long long i8_abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ bool i8_finite(unsigned long long b) {
    return b < 0x7ff0000000000000ull;
}
__device__ __forceinline__ double i8_from_bits(unsigned long long b) {
    return __longlong_as_double((long long)b);
}

// Largest |(pair | row)| of every panel row and, behind them, of the panel, as
// bits, into mx (zeroed before); an infinity or NaN counts as larger than every
// number.
__global__ void __launch_bounds__(256)
    k_i8_erimax(int npair, const int *__restrict__ rowpair, const double *__restrict__ m2,
                unsigned long long *mx) {
    const int pm = rowpair[blockIdx.x];
    unsigned long long m = 0;
    if (pm >= 0)
        for (int p = threadIdx.x; p < npair; p += 256) {
            const unsigned long long b = i8_abs_bits(m2[eri_index(p, pm)]);
            m = b > m ? b : m;
        }
    if (m) {
        atomicMax(mx + blockIdx.x, m);
        atomicMax(mx + kIM, m);
    }
}

// Digits of the integral table, both signs, and their scales (NaN when one of
// them is an infinity or NaN): CTA = panel row m.  FP32, with 31 bits, has a
// scale for each row; FP64, whose integer chunks add elements of different rows
// of T, one for the panel.
template <typename T, int NS>
__global__ void __launch_bounds__(128)
    k_i8_eri(int npair, const int *__restrict__ rowpair, const double *__restrict__ m2,
             const unsigned long long *__restrict__ mx, uint8_t *__restrict__ eri,
             T *__restrict__ rscale) {
    const int m = blockIdx.x, tid = threadIdx.x, pm = rowpair[m];
    const bool fin = i8_finite(mx[kIM]);
    int e = fin ? i8_exponent(i8_from_bits(mx[sizeof(T) == 8 ? kIM : m])) : 0;
    if (sizeof(T) == 4) e = max(e, -80);  // the scale stays a normal number
    // T = (sum_s acc_s 256^-s) 2^-14 2^(e + e_col); the kernel's sums carry
    // 2^42 (FP64) or 2^40, and the columns' scales 2^-bias
    if (tid == 0)
        rscale[m] = fin ? (T)ldexp(1.0, e - 14 + (sizeof(T) == 8 ? kIEBias - 42 : 8 - 40))
                        : (T)__longlong_as_double(0x7ff8000000000000ll);
    for (int p = tid; p < npair; p += 128)
        for (int sg = 0; sg < 2; sg++) {
            const double x = pm >= 0 && fin ? m2[eri_index(p, pm)] : 0.0;
            // digit u (most significant first) in byte u
            const uint64_t w = i8_bytes<NS>(i8_split<NS>(sg ? -x : x, e));
            const size_t o = ((size_t)sg * npair + p) * kIM + m;
            if (NS > 4)
                reinterpret_cast<uint64_t *>(eri)[o] = w;
            else
                reinterpret_cast<uint32_t *>(eri)[o] = (uint32_t)w;
        }
}

// ---- the product ------------------------------------------------------------

struct I8Layout {
    uint32_t b, bstride, t, tstride, raw, rawstride, list, lstride, sc, jo, rows, ex, misc;
    size_t total;
};

template <typename T, bool GRADED>
__host__ __device__ inline I8Layout i8_layout(int KP, int lmax) {
    constexpr int NS = kDigits<T>;
    I8Layout L;
    L.b = 0;
    L.bstride = (uint32_t)(NS * kIC * KP);
    L.t = L.b + kIRing * L.bstride;
    L.tstride = (uint32_t)((kIM * kIP * sizeof(T) + 15) / 16 * 16);
    L.raw = L.t + 2 * L.tstride;
    // a cutting warp's 8 x 16 tiles
    L.rawstride = GRADED ? (uint32_t)(KP / 16 * 128 * sizeof(T)) : 0;
    L.list = L.raw + I8Roles<T, GRADED>::load * L.rawstride;
    L.lstride = (uint32_t)lmax * 16;
    L.sc = L.list + kIRing * L.lstride;
    L.jo = L.sc + kIRing * kIC * (uint32_t)sizeof(T);
    L.rows = L.jo + 64 * 4;
    L.ex = L.rows + I8Roles<T, GRADED>::load * 64 * 4;
    L.misc = L.ex + (GRADED ? 2 * 2 * kIC * 4 : 0);
    L.total = L.misc + 192;
    return L;
}

// FP64: 2^34 sum over s of acc_s 256^(1-s).  |acc_s| <= (s + 1) 64 2^14, so the
// pairs 256 acc_s + acc_(s+1) stay below 2^31 and the whole sum, rounded to 6
// bits of acc_6 (2^-56 of the largest product), below 2^63: an integer in
// fourteen operations on 32-bit words (32 x 32 + 64-bit multiply-adds would
// take 2.3 clocks each, warp and SM).
__device__ __forceinline__ long long i8_join(const int (&a)[8]) {
    const int t01 = (a[0] << 8) + a[1], t23 = (a[2] << 8) + a[3];
    const int t45 = (a[4] << 8) + a[5], t6 = ((a[6] << 8) + a[7] + 8192) >> 14;
    return ((long long)t01 << 34) + ((long long)t23 << 18) + ((long long)t45 << 2) + (long long)t6;
}
// (2^52 + 2^31 + high) 2^32 - (2^84 + 2^63 + 2^52) + (2^52 + low), the first
// difference exact
__device__ __forceinline__ double i8_value(const int (&a)[8]) {
    const long long y = i8_join(a);
    const double h = __hiloint2double(0x43300000, (int)(y >> 32) ^ (int)0x80000000);
    const double l = __hiloint2double(0x43300000, (int)y);
    return fma(h, 4294967296.0, -(19342813113834066795298816.0 + 9223372036854775808.0 +
                                  4503599627370496.0)) + l;
}
__device__ __forceinline__ float i8_value(const int (&a)[4]) {
    return fmaf((float)((a[0] << 8) + a[1]), 4294967296.f,
                (float)((a[2] << 8) + a[3]) * 65536.f);
}

// 96-bit sums of 64-bit integers.
struct I8Sum {
    uint32_t lo, mid, hi;
    // += neg ? -x : x (neg is 0 or ~0)
    __device__ __forceinline__ void add(unsigned long long x, uint32_t neg) {
        const uint32_t a = (uint32_t)x ^ neg, b = (uint32_t)(x >> 32) ^ neg;
        const uint32_t c = (uint32_t)((int)b >> 31);
        asm("{\n .reg .u32 t;\n add.cc.u32 t, %3, 1;\n addc.cc.u32 %0, %0, %4;\n"
            " addc.cc.u32 %1, %1, %5;\n addc.u32 %2, %2, %6;\n}\n"
            : "+r"(lo), "+r"(mid), "+r"(hi)
            : "r"(neg), "r"(a), "r"(b), "r"(c));
    }
    __device__ __forceinline__ void add(const I8Sum &x) {
        asm("add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %4;\n addc.u32 %2, %2, %5;\n"
            : "+r"(lo), "+r"(mid), "+r"(hi)
            : "r"(x.lo), "r"(x.mid), "r"(x.hi));
    }
    __device__ __forceinline__ I8Sum from_lane_xor(uint32_t o) const {
        return {__shfl_xor_sync(~0u, lo, o), __shfl_xor_sync(~0u, mid, o),
                __shfl_xor_sync(~0u, hi, o)};
    }
    // rounded once: |sum| < 2^70, so hi:mid is below 2^51 and 1.5 2^52 + hi:mid
    // has the bits 0x43380000 + hi, mid
    __device__ __forceinline__ double value() const {
        const double h = __hiloint2double((int)(0x43380000u + hi), (int)mid);
        const double l = __hiloint2double(0x43300000, (int)lo);
        return fma(h, 4294967296.0, -(29014219670751100192948224.0 + 4503599627370496.0)) + l;
    }
};

__device__ __forceinline__ double i8_flip(double x, uint32_t neg) {
    return __hiloint2double(__double2hiint(x) ^ (int)neg, __double2loint(x));
}
__device__ __forceinline__ float i8_flip(float x, uint32_t neg) {
    return __uint_as_float(__float_as_uint(x) ^ neg);
}

// 4 x 4 bytes transposed: out[u] holds byte u of in[0..3].
__device__ __forceinline__ void i8_transpose4(const uint32_t (&in)[4], uint32_t (&out)[4]) {
    const uint32_t a = __byte_perm(in[0], in[1], 0x5140), b = __byte_perm(in[2], in[3], 0x5140);
    const uint32_t c = __byte_perm(in[0], in[1], 0x7362), d = __byte_perm(in[2], in[3], 0x7362);
    out[0] = __byte_perm(a, b, 0x5410);
    out[1] = __byte_perm(a, b, 0x7632);
    out[2] = __byte_perm(c, d, 0x5410);
    out[3] = __byte_perm(c, d, 0x7632);
}

// ---- c in digits, inside the product -----------------------------------------
//
// The exponent of column Jb is that of the largest |c(Ja_j, Jb)| over the alpha
// singles j of the CTA's string, not over the whole column: everything that the
// digits of a small element are cut against is then an element of the same sum.
// High words of the values order like their magnitudes; the exponent, biased,
// is such that the top digit stays within 127 after the carries of the lower
// ones (2^14 and 2^17 carry when the mantissa is 127/64 or more).
constexpr int kIEb = 62, kIEbF = 8;   // least biased exponents: the scales stay normal

// 32 leading bits of |x|
__device__ __forceinline__ uint32_t i8_high(double x) {
    return (uint32_t)__double2hiint(x) & 0x7fffffffu;
}
__device__ __forceinline__ uint32_t i8_high(float x) { return __float_as_uint(x) & 0x7fffffffu; }
template <typename T>
__device__ __forceinline__ bool i8_high_finite(uint32_t h) {
    return h < (sizeof(T) == 8 ? 0x7ff00000u : 0x7f800000u);
}
template <typename T>
__device__ __forceinline__ int i8_biased(uint32_t h) {
    return sizeof(T) == 8 ? max((int)((h + (1u << 14)) >> 20), kIEb)
                          : max((int)((h + (1u << 17)) >> 23), kIEbF);
}
// 2^(e - bias) of the column exponent, in integer instructions
__device__ __forceinline__ double i8_scale(int eb, double) {
    return __hiloint2double((eb - 1022 - kIEBias + 1023) << 20, 0);
}
__device__ __forceinline__ float i8_scale(int eb, float) {
    return __uint_as_float((uint32_t)(eb - 126 - 8 + 127) << 23);
}

// The balanced base-256 digits of x 2^-e (e of the biased exponent eb), most
// significant in byte 6 (FP64) or 3 (FP32), rounded to 55 or 31 bits below 2^e.
// Integer instructions only: the FP64 units stand still under integer MMAs.
// (FP64 zeros and subnormal numbers get a leading bit, and lose it with all
// others in a shift by 62 or more; PTX shifts by more than 63 give 0.)
__device__ __forceinline__ uint64_t i8_cut(double x, int eb) {
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) |
                       (uint32_t)__double2loint(x);
    uint64_t v;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m << 3), "r"((uint32_t)eb - ((hi >> 20) & 0x7ffu)));
    v = (v + 1) >> 1;
    const uint64_t sg = (uint64_t)((int64_t)(int32_t)hi >> 63);
    constexpr uint64_t carry = 0x0080808080808080ull;
    return ((v ^ sg) - sg + carry) ^ carry;
}
__device__ __forceinline__ uint64_t i8_cut(float x, int eb) {
    const uint32_t w = __float_as_uint(x), b = (w >> 23) & 0xffu;
    const uint32_t m = (w & 0x7fffffu) | (b ? 0x800000u : 0u);
    const uint32_t v = (__funnelshift_rc(m << 8, 0u, (uint32_t)(eb - (int)max(b, 1u))) + 1) >> 1;
    const uint32_t sg = (uint32_t)((int32_t)w >> 31);
    return ((v ^ sg) - sg + 0x00808080u) ^ 0x00808080u;
}

// Four neighbouring columns of a lane's row, cut and written as one word a
// digit (dst: the word of digit 0; SLICE: bytes from one digit's block to the
// next).
template <typename T, int SLICE>
__device__ __forceinline__ void i8_cut4(const T (&x)[4], const int (&eb)[4], unsigned char *dst) {
    constexpr int NS = kDigits<T>, slice = SLICE;
    uint32_t lo[4], hi[4], t[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint64_t w = i8_cut(x[i], eb[i]);
        lo[i] = (uint32_t)w;
        hi[i] = (uint32_t)(w >> 32);
    }
    if constexpr (NS > 4) {
        i8_transpose4(hi, t);  // bytes 4, 5, 6: digits 2, 1, 0
#pragma unroll
        for (int u = 0; u < 3; u++) *reinterpret_cast<uint32_t *>(dst + u * slice) = t[2 - u];
    }
    i8_transpose4(lo, t);      // bytes 0 .. 3: the last four digits
#pragma unroll
    for (int u = 0; u < 4; u++)
        *reinterpret_cast<uint32_t *>(dst + (NS - 4 + u) * slice) = t[3 - u];
}

// ---- c in digits, once for all strings ---------------------------------------
//
// The same cut with the exponent of the whole column, which every string whose
// singles reach an element near it can use: within kINear bits of the scale, so
// that the largest element of a string's sum keeps 52 bits (FP64) or 25 (FP32).
// For a vector whose columns are not graded that is every string, and cutting
// the rows once instead of for each of K strings saves a quarter of sigma's
// time.  Strings that miss it in some chunk are graded: their product cuts the
// digits of such chunks itself.
template <typename T>
constexpr int kINear = sizeof(T) == 8 ? 3 : 6;
constexpr int kIGraded = 1, kISame = 2;   // flags of a string's chunk: cut there; one exponent
// Masks of a row's columns in a chunk: elements near the scale, and elements
// that are not zero; further bits: the chunk's columns have one exponent, the
// row holds an infinity or NaN.
struct alignas(16) I8Mask {
    unsigned long long near, some;
};
constexpr unsigned long long kISameBit = 1ull << 62, kINotFinite = 1ull << 63;

// High word of the largest finite |c| of every column: 128 columns x 64 rows per
// CTA, one atomicMax per column.  Bound by the one read of c.
template <typename T>
__global__ void __launch_bounds__(256)
    k_i8_colmax(int na, int nb, const T *__restrict__ V, uint32_t *__restrict__ mx,
                const int *skip) {
    if (skip && *skip) return;
    __shared__ uint32_t part[128];
    const int col = blockIdx.x * 128 + (threadIdx.x & 127), h = threadIdx.x >> 7;
    const int r0 = blockIdx.y * 64 + 32 * h, r1 = min(na, r0 + 32);
    uint32_t m = 0;
    if (col < nb)
#pragma unroll 8
        for (int r = r0; r < r1; r++) {
            const uint32_t b = i8_high(V[(long long)r * nb + col]);
            if (i8_high_finite<T>(b)) m = max(m, b);
        }
    if (h) part[threadIdx.x & 127] = m;
    __syncthreads();
    if (!h && col < nb) atomicMax(mx + col, max(m, part[threadIdx.x]));
}

// Digits of c: thread = 4 consecutive columns of one row of a chunk; 16 rows
// per CTA.  sl[chunk][row][16-column block][u][16], so that the copies of the
// product read whole 32-byte sectors.
template <typename T>
__global__ void __launch_bounds__(192)
    k_i8_slice(int na, int nb, const T *__restrict__ V, const uint32_t *__restrict__ mx,
               uint8_t *__restrict__ sl, T *__restrict__ cscale, I8Mask *__restrict__ masks,
               const int *skip) {
    if (skip && *skip) return;
    constexpr int NS = kDigits<T>;
    __shared__ int es[kIC];
    __shared__ int emax, emin;
    __shared__ uint32_t ms[16][2][2];  // [row][near, some][24 columns | not finite << 31]
    const int c = blockIdx.x, nchunk = gridDim.x, tid = threadIdx.x;
    if (tid == 0) {
        emax = sizeof(T) == 8 ? kIEb : kIEbF;
        emin = 1 << 20;
    }
    if (tid < 64) (&ms[0][0][0])[tid] = 0;
    __syncthreads();
    if (tid < kIC) {
        const int col = c * kIC + tid;
        const uint32_t b = col < nb ? mx[col] : 0;
        es[tid] = b ? i8_biased<T>(b) : 0;  // 0: a zero column
        if (b) {
            atomicMax(&emax, es[tid]);
            atomicMin(&emin, es[tid]);
        }
    }
    __syncthreads();
    const bool one = sizeof(T) == 8 && emax - emin <= kISpread;
    if (blockIdx.y == 0 && tid < kIC)
        cscale[c * kIC + tid] = i8_scale(one || !es[tid] ? emax : es[tid], T(0));
    const int q = tid % 12, rl = tid / 12, row = blockIdx.y * 16 + rl, c0 = c * kIC + 4 * q;
    if (row < na) {
        T x[4];
        int eb[4];
        uint32_t near = 0, some = 0;
        const int b0 = 4 * (q % 6);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = es[4 * q + i];
            eb[i] = one || !e ? emax : e;
            x[i] = c0 + i < nb ? V[(long long)row * nb + c0 + i] : T(0);
            const uint32_t h = i8_high(x[i]);
            if (x[i] != T(0)) some |= 1u << (b0 + i);  // (so is a NaN)
            if (!i8_high_finite<T>(h)) {
                x[i] = T(0);
                some |= 1u << 31;
            } else if ((int)(h >> (sizeof(T) == 8 ? 20 : 23)) >= eb[i] - kINear<T>) {
                near |= 1u << (b0 + i);
            }
        }
        i8_cut4<T, 16>(x, eb, sl + ((size_t)c * na + row) * NS * kIC + (q >> 2) * (NS * 16) +
                                  4 * (q & 3));
        if (near) atomicOr(&ms[rl][0][q / 6], near);
        if (some) atomicOr(&ms[rl][1][q / 6], some);
    }
    __syncthreads();
    if (tid < 16 && blockIdx.y * 16 + tid < na) {
        const auto mask = [&](int k) {
            return (unsigned long long)(ms[tid][k][0] & 0xffffffu) |
                   (unsigned long long)(ms[tid][k][1] & 0xffffffu) << 24;
        };
        I8Mask m = {mask(0), mask(1)};
        if (one) m.near |= kISameBit;
        if ((ms[tid][1][0] | ms[tid][1][1]) >> 31) m.some |= kINotFinite;
        masks[(size_t)(blockIdx.y * 16 + tid) * nchunk + c] = m;
    }
}

// The flags of a string's chunks from the masks of the rows that its singles
// reach; the CTA that ends last then lists the plain and the graded strings in
// their order (neighbours share most rows of c: FCI(16,16) 126.3 ms a sigma, 127.6
// listed as they came in).  Bound by reading K masks a chunk, from L2: 1 ms of 126
// at FCI(16,16).
__global__ void __launch_bounds__(128)
    k_i8_grade(int na, int nchunk, int K, const uint32_t *__restrict__ fsA,
               const I8Mask *__restrict__ masks, uint8_t *__restrict__ flags,
               uint8_t *__restrict__ kind, int *__restrict__ nstr, int *__restrict__ strs,
               const int *skip) {
    if (skip && *skip) return;
    __shared__ int rows[64];
    __shared__ I8Mask part[4][32];
    __shared__ int before[128], last;
    const int Ia = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < K) rows[tid] = (int)(fsA[(long long)tid * na + Ia] & 0x3fffffffu);
    __syncthreads();
    bool any = false;
    for (int c0 = 0; c0 < nchunk; c0 += 32) {  // a warp, every fourth row of 32 chunks
        const int c = c0 + lane;
        I8Mask m = {0, 0};
        if (c < nchunk)
#pragma unroll 4
            for (int j = w; j < K; j += 4) {
                const I8Mask x = masks[(size_t)rows[j] * nchunk + c];
                m.near |= x.near;
                m.some |= x.some;
            }
        part[w][lane] = m;
        __syncthreads();
        if (w == 0 && c < nchunk) {
#pragma unroll
            for (int k = 1; k < 4; k++) {
                m.near |= part[k][lane].near;
                m.some |= part[k][lane].some;
            }
            const bool graded = (m.some & ~m.near) != 0;
            flags[(size_t)Ia * nchunk + c] =
                (uint8_t)((graded ? kIGraded : 0) | (m.near & kISameBit ? kISame : 0));
            any = any || graded;
        }
        __syncthreads();
    }
    any = __syncthreads_or(any);
    if (tid == 0) {
        kind[Ia] = any;
        __threadfence();
        last = atomicAdd(nstr + 2, 1) == na - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // thread t: 16 n strings from 16 n t on
    const int n = ((na + 15) / 16 + 127) / 128, i0 = 16 * n * tid;
    const auto words = [&](int v) {
        uint4 x = make_uint4(0, 0, 0, 0);
        if (i0 + 16 * v < na) x = __ldcg(reinterpret_cast<const uint4 *>(kind + i0 + 16 * v));
        return x;
    };
    int count = 0;
    for (int v = 0; v < n; v++) {
        const uint4 x = words(v);  // (bytes behind the last string are zero)
        count += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    }
    before[tid] = count;
    __syncthreads();
    int g = 0;
    for (int t = 0; t < tid; t++) g += before[t];
    if (tid == 127) {
        nstr[1] = g + count;
        nstr[0] = na - g - count;
    }
    int p = min(i0, na) - g;
    for (int v = 0; v < n; v++) {
        const uint4 x = words(v);
        const uint32_t q[4] = {x.x, x.y, x.z, x.w};
        for (int k = 0; k < 16; k++) {
            const int i = i0 + 16 * v + k;
            if (i >= na) break;
            if ((q[k >> 2] >> (8 * (k & 3))) & 1)
                strs[na + g++] = i;
            else
                strs[p++] = i;
        }
    }
}

// The MMAs of one chunk that issuer I of NI takes: whole accumulators, so that
// each is written by one thread in order: {6, 0}, {7, 1}, {5, 2}, {4, 3} of
// FP64's eight (8 or 9 digit products each); {3, 0}, {2, 1} of FP32's four.
template <int NS, int I>
__device__ __forceinline__ void i8_issue(uint32_t d0, uint32_t a0, uint64_t bd0, int ksteps) {
    constexpr uint64_t bslice = (8 * kIC) >> 4;   // B: [8 rows][digit][16 columns][row][16]
    for (int kk = 0; kk < ksteps; kk++) {
        const uint32_t at = a0 + 8 * kk;
        const uint64_t bd = bd0 + (uint64_t)kk * ((4 * NS * 8 * kIC) >> 4);
#pragma unroll
        for (int u = 0; u < NS; u++)
#pragma unroll
            for (int s = kSums<NS> - 1; s >= 0; s--) {
                const int first = s < NS ? 0 : s - NS + 1;  // lowest u with s - u < NS
                const bool mine = NS == 7 ? (I == 0   ? s == 6 || s == 0
                                             : I == 1 ? s == 7 || s == 1
                                             : I == 2 ? s == 5 || s == 2
                                                      : s == 4 || s == 3)
                                          : ((s == 3 || s == 0) == (I == 0));
                if (mine && u >= first && u <= s)
                    i8_mma(d0 + s * kIC, at + u * 16, bd + (s - u) * bslice,
                           (u > first || kk > 0) ? 1u : 0u);
            }
    }
}

// One CTA per SM walks the plain or the graded alpha strings; its warps take four roles, which
// meet only at mbarriers, so that the cutting, products, extractions and
// gathers of neighbouring chunks (48 beta strings) overlap:
//   loaders (2 warps, 6 for graded strings): the digits of chunk after chunk of
//     c's rows Ja_j into one of a ring of kIRing buffers (cp.async); of a graded
//     chunk c itself into shared memory (cp.async, each lane the elements that
//     it cuts), the exponents of these rows' columns, and the digits from them;
//     with them the chunk's lists;
//   issuers (4 warps, 2 in FP32): the MMAs of a chunk once its digits are there
//     and the accumulators have been read;
//   extractors (8 warps, 12 in FP32): per string, the digits of A into tensor
//     memory; per chunk, the accumulators tensor memory -> registers, the
//     digits' sums joined to T in one of two buffers in shared memory;
//   gatherers (the other warps): the sigma elements that the chunk's lists name,
//     plus their entries of T.
// The extraction does its FP64 work while the tensor cores are idle (they
// wait for the accumulators), the gather runs under the next chunk's MMAs.
// A chunk's lists hold, per group of 32 lanes, the lanes' beta strings and
// then their entries, byte offset in T | phase, entry k of the 32 lanes side
// by side.  A string with more than kISeg entries takes 2, 4, .. lanes,
// added up by shuffles (the strings of the chunk itself have up to 50 entries,
// the others a few).  A string occurs once per chunk, so sums run in a fixed
// order.
// Every wait is bounded; on expiry a role stops, the others' waits for it
// expire in turn, the kernel records an error, waits (also bounded) for its
// committed MMAs, frees its tensor memory and returns.
template <typename T, bool GRADED>
__global__ void __launch_bounds__(kIThreads, 1)
    k_sigma_i8(I8Args<T> a, const T *__restrict__ V, T *__restrict__ S, int *status) {
    if (a.skip && *a.skip) return;
    const int nstr = a.nstr[GRADED];
    const int *strs = a.strs + (GRADED ? a.na : 0);
    if ((int)blockIdx.x >= nstr) return;
    constexpr int NS = kDigits<T>;
    using Roles = I8Roles<T, GRADED>;
    constexpr int kIExt = Roles::ext, kIGat = Roles::gat, kIIss = Roles::iss, kILoad = Roles::load;
    static_assert(32 * (kIExt + kIGat + kIIss + kILoad) == kIThreads && kIC % (kIExt / 4) == 0,
                  "roles");
    static_assert(kIIss == (NS == 7 ? 4 : 2), "issuers");
    constexpr int NU = kSums<NS>;           // accumulators
    constexpr int NACC = NS <= 4 ? 2 : 1;   // sets of them in tensor memory
    constexpr int kACol = NACC * NU * kIC;  // A's columns: 16 per digit (at most 112)
    static_assert(kACol + NS * 16 <= 512 && kIM * kIP * 8 <= 65536, "tensor memory, list entries");
    extern __shared__ __align__(1024) unsigned char smem[];
    const I8Layout L = i8_layout<T, GRADED>(a.KP, a.lmax);
    const uint32_t sb = i8_smem(smem);
    T *scs = reinterpret_cast<T *>(smem + L.sc);
    uint32_t *jo = reinterpret_cast<uint32_t *>(smem + L.jo);
    const uint32_t bar_full = sb + L.misc, bar_gone = bar_full + 8 * kIRing;
    const uint32_t bar_done = bar_gone + 8 * kIRing, bar_free = bar_done + 16;
    const uint32_t bar_t = bar_free + 16, bar_tfree = bar_t + 16, bar_a = bar_tfree + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L.misc + 160);
    int *tint = reinterpret_cast<int *>(smem + L.misc + 164);  // [2] T holds integers
    int *mode = reinterpret_cast<int *>(smem + L.misc + 172);  // [ring] what the chunk's columns are
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(~0u, tid >> 5, 0);  // known to be the same in a warp
    const int K = a.K, KP = a.KP, nchunk = a.nchunk;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         i8_smem(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid < 2)  // the null element of the lists, in both buffers
        *reinterpret_cast<T *>(smem + L.t + tid * L.tstride + kIZero * sizeof(T)) = T(0);
    if (tid == 0) {
        auto init = [&](uint32_t bar, uint32_t n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory");
        };
        for (int i = 0; i < kIRing; i++) {
            init(bar_full + 8 * i, 32 * kILoad);
            init(bar_gone + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            init(bar_done + 8 * i, kIIss);
            init(bar_free + 8 * i, kIExt);
            init(bar_t + 8 * i, kIExt);
            init(bar_tfree + 8 * i, 1);
        }
        init(bar_a, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool failed = false;

    if (warp >= kIExt + kIGat + kIIss) {
        // ---- loaders
        const int w = warp - kIExt - kIGat - kIIss;
        int *rows = reinterpret_cast<int *>(smem + L.rows) + 64 * w;  // [64] rows of c, -1: none
        // copies: warp w takes the 8-row blocks w, w + kILoad, ..; a lane, pieces
        // of one row
        const int r8 = lane & 7, p4 = lane >> 3;
        constexpr int NQ = (3 * NS + 3) / 4;     // this lane's pieces of a row: 4 i + p4
        int doff[NQ];
#pragma unroll
        for (int i = 0; i < NQ; i++) {
            const int q = 4 * i + p4, n16 = q / NS, u = q - n16 * NS;
            doff[i] = u * (8 * kIC) + n16 * 128 + r8 * 16;
        }
        // cuts: warp w takes the columns 16 (w % 3) .. + 15 and every other block of
        // 8 rows; a lane, four columns of one row each
        constexpr int NT = 4;                    // its blocks, at most
        const int n16 = w % 3, half = w / 3, j8 = lane >> 2, q4 = lane & 3;
        const int nt = KP / 16, cc = 16 * n16 + 4 * q4;
        constexpr int P = sizeof(T) == 8 ? 2 : 1;  // 16-byte pieces of four elements
        constexpr int VE = 16 / sizeof(T);
        unsigned char *raw = smem + L.raw + w * L.rawstride + 16 * lane;
        uint32_t *ex = reinterpret_cast<uint32_t *>(smem + L.ex);  // [2][half][column]
        // this lane's elements of chunk c on their way; zeros past the row's end
        // and (written once) in rows without a single
        auto fetch = [&](int c) {
            const int col = c * kIC + cc, left = a.nb - col;
#pragma unroll
            for (int i = 0; i < NT; i++) {
                const int J = i < nt ? rows[8 * (half + 2 * i) + j8] : -1;
                if (J < 0) continue;
                const T *src = V + (long long)J * a.nb + col;
                unsigned char *dst = raw + i * P * 512;
                if (a.vec && left >= 4) {
#pragma unroll
                    for (int h = 0; h < P; h++)
                        __pipeline_memcpy_async(dst + h * 512, src + VE * h, 16);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        T *d = reinterpret_cast<T *>(dst + k / VE * 512) + k % VE;
                        if (k < left)
                            __pipeline_memcpy_async(d, src + k, sizeof(T));
                        else
                            *d = T(0);
                    }
                }
            }
        };
        auto value = [&](int i, T (&x)[4]) {
#pragma unroll
            for (int h = 0; h < P; h++) {
                const CutVec<T> y = *reinterpret_cast<const CutVec<T> *>(raw + (i * P + h) * 512);
#pragma unroll
                for (int k = 0; k < VE; k++) x[VE * h + k] = y.v[k];
            }
        };
        if constexpr (GRADED)
            for (int i = 0; i < nt * P; i++)
                *reinterpret_cast<uint4 *>(raw + i * 512) = make_uint4(0, 0, 0, 0);
        uint32_t g = 0, r = 0, par = 0;          // chunk, its ring slot and phase
        // a chunk of copied digits is handed over when the one behind it has been
        // asked for, so that two are on their way
        bool pend = false;
        uint32_t prev = 0;
        bool lose = a.expire && blockIdx.x == 0;
        auto hand = [&](uint32_t slot) {
            if (lose) {
                lose = false;
                return;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            i8_arrive(bar_full + 8 * slot);
        };
        auto flush = [&]() {
            __pipeline_wait_prior(0);
            if (pend) hand(prev);
            pend = false;
        };
        for (int is = blockIdx.x; is < nstr && !failed; is += gridDim.x) {
            const int Ia = strs[is];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = lane + 32 * i;
                rows[j] = j < K ? (int)(a.fsA[(long long)j * a.na + Ia] & 0x3fffffffu) : -1;
            }
            __syncwarp();
            const uint8_t *fl = a.flags + (size_t)Ia * nchunk;
            uint32_t f = fl[0], f1 = nchunk > 1 ? fl[1] : 0;  // flags of this chunk and the next
            if (GRADED && (f & kIGraded)) {
                flush();
                fetch(0);
                __pipeline_commit();
            }
            uint32_t o = a.lofs[0], o1 = a.lofs[1];
            for (int c = 0; c < nchunk; c++, g++) {
                const bool cut = GRADED && (f & kIGraded), cutnext = GRADED && (f1 & kIGraded);
                const uint32_t n = o1 - o, o2 = c + 2 <= nchunk ? a.lofs[c + 2] : 0;
                const uint32_t f2 = c + 2 < nchunk ? fl[c + 2] : 0;
                uint32_t mx[4] = {0, 0, 0, 0};
                uint32_t *exc = ex + (g & 1) * 2 * kIC;
                if (cut) {
                    flush();  // this chunk's elements, too
#pragma unroll
                    for (int i = 0; i < NT; i++)
                        if (i < nt) {
                            T x[4];
                            value(i, x);
#pragma unroll
                            for (int k = 0; k < 4; k++) mx[k] = max(mx[k], i8_high(x[k]));
                        }
#pragma unroll
                    for (int k = 0; k < 4; k++)
#pragma unroll
                        for (int l = 4; l < 32; l <<= 1)
                            mx[k] = max(mx[k], __shfl_xor_sync(~0u, mx[k], l));
                    if (j8 == 0)
                        *reinterpret_cast<uint4 *>(exc + half * kIC + cc) =
                            make_uint4(mx[0], mx[1], mx[2], mx[3]);
                } else if (pend && !__all_sync(~0u, i8_test(bar_gone + 8 * r, par ^ 1))) {
                    flush();  // the slot is still in use: hand over the chunk before first
                }
                // the slot's previous chunk has been gathered
                bool ok = __all_sync(~0u, i8_wait(bar_gone + 8 * r, par ^ 1));
                if constexpr (GRADED) {  // the exponents are exchanged: all stop or none
                    if (i8_sync_or<kILoad>(3, !ok)) ok = false;
                }
                if (!ok) { failed = true; break; }
                uint4 *ld = reinterpret_cast<uint4 *>(smem + L.list + r * L.lstride);
                for (uint32_t i = 32 * w + lane; i < n; i += 32 * kILoad)
                    __pipeline_memcpy_async(ld + i, a.lists + o + i, 16);
                unsigned char *slot = smem + L.b + r * L.bstride;
                if (cut) {
                    __pipeline_commit();
                    // the columns' exponents: of this lane's four, and their range
                    const uint4 y = *reinterpret_cast<const uint4 *>(exc + (half ^ 1) * kIC + cc);
                    mx[0] = max(mx[0], y.x);
                    mx[1] = max(mx[1], y.y);
                    mx[2] = max(mx[2], y.z);
                    mx[3] = max(mx[3], y.w);
                    const uint32_t h0 = max(exc[lane], exc[kIC + lane]);
                    const uint32_t h1 =
                        lane < kIC - 32 ? max(exc[32 + lane], exc[kIC + 32 + lane]) : 0u;
                    const uint32_t top = __reduce_max_sync(~0u, max(h0, h1));
                    const int emax = i8_biased<T>(top);
                    // zero columns go with any exponent
                    const int emin = __reduce_min_sync(~0u, min(h0 ? i8_biased<T>(h0) : 1 << 20,
                                                                h1 ? i8_biased<T>(h1) : 1 << 20));
                    const bool bad = !i8_high_finite<T>(top);
                    const bool one = sizeof(T) == 8 && emax - emin <= kISpread;
                    int eb[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) eb[k] = one ? emax : i8_biased<T>(mx[k]);
                    if (half == 0 && j8 == 0)
#pragma unroll
                        for (int k = 0; k < 4; k++) scs[r * kIC + cc + k] = i8_scale(eb[k], T(0));
                    if (w == 0 && lane == 0) mode[r] = bad ? kIBad : one ? kIOne : kIEach;
                    unsigned char *dst = slot + n16 * 128 + j8 * 16 + 4 * q4;
#pragma unroll
                    for (int i = 0; i < NT; i++)
                        if (i < nt) {
                            T x[4];
                            value(i, x);
                            // (rows without a single: A's digits there are zero)
                            if (8 * (half + 2 * i) + j8 < K)
                                i8_cut4<T, 8 * kIC>(x, eb, dst + (half + 2 * i) * (NS * 8 * kIC));
                        }
                    // the next chunk's elements, in the place of this one's
                    if (cutnext) fetch(c + 1);
                    __pipeline_commit();
                    __pipeline_wait_prior(1);  // the lists have landed
                    hand(r);
                } else {
                    const uint8_t *src = a.sl + (size_t)c * a.na * (NS * kIC) + 16 * p4;
                    for (int jb = w; jb < KP / 8; jb += kILoad) {
                        const int J = rows[8 * jb + r8];
                        const uint8_t *sj = src + (size_t)J * (NS * kIC);
                        unsigned char *dj = slot + jb * (NS * 8 * kIC);
                        if (J >= 0)
#pragma unroll
                            for (int i = 0; i < NQ; i++)
                                if (4 * i + 3 < 3 * NS || 4 * i + p4 < 3 * NS)
                                    __pipeline_memcpy_async(dj + doff[i], sj + 64 * i, 16);
                    }
                    constexpr int sn = kIC * (int)sizeof(T) / 16;
                    if (w == 0 && lane < sn)
                        __pipeline_memcpy_async(
                            reinterpret_cast<unsigned char *>(scs + r * kIC) + 16 * lane,
                            reinterpret_cast<const unsigned char *>(a.cscale + (size_t)c * kIC) +
                                16 * lane,
                            16);
                    if (GRADED && w == 0 && lane == 0) mode[r] = f & kISame ? kIOne : kIEach;
                    if (cutnext) fetch(c + 1);
                    __pipeline_commit();
                    if (pend) {
                        __pipeline_wait_prior(1);
                        hand(prev);
                    }
                    pend = true;
                    prev = r;
                }
                o = o1;
                o1 = o2;
                f = f1;
                f1 = f2;
                if (++r == kIRing) { r = 0; par ^= 1; }
            }
        }
        if (failed) pend = false;
        flush();
    } else if (warp >= kIExt + kIGat) {
        // ---- issuers: whole warps walk the chunks, an elected lane issues
        // (descriptors then live in uniform registers)
        const int I = warp - kIExt - kIGat;
        uint32_t g = 0, r = 0, par = 0, row = 0;
        for (int i = blockIdx.x; i < nstr && !failed; i += gridDim.x, row++) {
            failed = !__all_sync(~0u, i8_wait(bar_a, row & 1));
            for (int c = 0; c < nchunk && !failed; c++, g++) {
                const uint32_t acc = NACC == 2 ? g & 1 : 0;
                bool ok = i8_wait(bar_full + 8 * r, par);
                ok = ok && (g < NACC || i8_wait(bar_free + 8 * acc, (g / NACC - 1) & 1));
                if (!__all_sync(~0u, ok)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t bd = i8_desc(sb + L.b + r * L.bstride, NS * 8 * kIC, 128);
                const uint32_t d0 = tmem + acc * (NU * kIC), a0 = tmem + kACol;
                if (i8_elect()) {
                    if (I == 0)
                        i8_issue<NS, 0>(d0, a0, bd, KP / 32);
                    else if (I == 1)
                        i8_issue<NS, 1>(d0, a0, bd, KP / 32);
                    else if constexpr (kIIss == 4) {
                        if (I == 2)
                            i8_issue<NS, 2>(d0, a0, bd, KP / 32);
                        else
                            i8_issue<NS, 3>(d0, a0, bd, KP / 32);
                    }
                    asm volatile(
                        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 "
                        "[%0];" ::"r"(bar_done + 8 * acc)
                        : "memory");
                }
                __syncwarp();
                if (++r == kIRing) { r = 0; par ^= 1; }
            }
        }
        // leave nothing in flight (returns at once when all was waited for)
        for (uint32_t k = g > NACC ? g - NACC : 0; failed && k < g; k++)
            i8_wait(bar_done + 8 * (NACC == 2 ? k & 1 : 0), (k / NACC) & 1);
        __syncwarp();
    } else if (warp >= kIExt) {
        // ---- gatherers
        const int gw = warp - kIExt;
        const T rs = a.rscale[0];  // of integer chunks: FP64's rows have one scale
        uint32_t g = 0, r = 0, par = 0;
        for (int is = blockIdx.x; is < nstr && !failed; is += gridDim.x) {
            const int Ia = strs[is];
            T *srow = S + (long long)Ia * a.nb;
            for (int c = 0; c < nchunk; c++, g++) {
                bool ok = i8_wait(bar_full + 8 * r, par);
                // the lists have landed: load the sigma elements they name
                const unsigned char *lp = smem + L.list + r * L.lstride;
                const int ng = ok ? *reinterpret_cast<const int *>(lp) : 0;
                const uint2 *head = reinterpret_cast<const uint2 *>(lp + 16);
                const uint16_t *tg = reinterpret_cast<const uint16_t *>(head + ng) + lane;
                constexpr int UG = 3;
                int t[UG];
                T x[UG];
#pragma unroll
                for (int i = 0; i < UG; i++) {
                    const int gr = gw + i * kIGat;
                    t[i] = 0xffff;
                    if (gr < ng) t[i] = tg[32 * gr];
                    if (t[i] != 0xffff) x[i] = srow[t[i]];
                }
                ok = ok && i8_wait(bar_t + 8 * (g & 1), (g >> 1) & 1);
                if (__all_sync(~0u, ok)) {
                    const unsigned char *Ts = smem + L.t + (g & 1) * L.tstride;
                    const bool ints = sizeof(T) == 8 && tint[g & 1];
                    // the lane's entries of one group added to y
                    auto gather = [&](int gr, T y) {
                        const uint2 h = head[gr];
                        const int n = h.y & 0xffff, l = h.y >> 16;
                        const uint16_t *pe = reinterpret_cast<const uint16_t *>(lp + h.x) + lane;
                        if (ints) {
                            I8Sum v = {0, 0, 0};
#pragma unroll 4
                            for (int k = 0; k < n; k++) {
                                const uint32_t e = pe[32 * k];
                                v.add(*reinterpret_cast<const unsigned long long *>(Ts + (e & ~1u)),
                                      0u - (e & 1u));
                            }
                            for (int o = 1; o < 1 << l; o <<= 1) v.add(v.from_lane_xor(o));
                            return fma((T)v.value() * rs, scs[r * kIC], y);
                        }
#pragma unroll 4
                        for (int k = 0; k < n; k++) {
                            const uint32_t e = pe[32 * k];
                            y += i8_flip(*reinterpret_cast<const T *>(Ts + ((e & ~1u) >> (sizeof(T) == 8 ? 0 : 1))), e << 31);
                        }
                        for (int o = 1; o < 1 << l; o <<= 1) y += __shfl_xor_sync(~0u, y, o);
                        return y;
                    };
#pragma unroll
                    for (int i = 0; i < UG; i++) {
                        const int gr = gw + i * kIGat;
                        if (gr >= ng) break;
                        // lanes without a string of their own start from nothing
                        const T y = gather(gr, t[i] != 0xffff ? x[i] : T(0));
                        if (t[i] != 0xffff) srow[t[i]] = y;
                    }
                    for (int gr = gw + UG * kIGat; gr < ng; gr += kIGat) {
                        const int tt = tg[32 * gr];
                        const T y = gather(gr, tt != 0xffff ? srow[tt] : T(0));
                        if (tt != 0xffff) srow[tt] = y;
                    }
                } else {
                    ok = false;
                }
                // T and the chunk's lists are free, the string's sums in order
                if (i8_sync_or<kIGat>(2, !ok)) {
                    failed = true;
                    break;
                }
                if (gw == 0 && lane == 0) {
                    i8_arrive(bar_tfree + 8 * (g & 1));
                    i8_arrive(bar_gone + 8 * r);
                }
                if (++r == kIRing) { r = 0; par ^= 1; }
            }
        }
    } else {
        // ---- extractors
        const int m = 32 * (warp & 3) + lane;  // this lane's panel row
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        const T rs = a.rscale[m];
        const bool hfin = rs == rs;  // no infinity or NaN among the integrals
        uint32_t g = 0, r = 0, par = 0;
        bool ok = true;
        for (int is = blockIdx.x; is < nstr; is += gridDim.x) {
            const int Ia = strs[is];
            // the string's singles: table rows
            if (warp == 0) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int j = lane + 32 * i;
                    uint32_t off = ~0u;
                    if (j < K) {
                        const long long o = (long long)j * a.na + Ia;
                        const uint32_t e = a.fsA[o];
                        off = ((e >> 31) * (uint32_t)a.npair + a.fpA[o]) * kIM;
                    }
                    jo[j] = off;
                }
            }
            if (i8_sync_or<kIExt>(1, !ok)) {
                failed = true;
                break;
            }
            // A digits of row m, 16 singles at a time (all MMAs of the string
            // before have been waited for)
            for (int j0 = 16 * (warp >> 2); j0 < KP; j0 += 16 * (kIExt / 4)) {
                uint32_t w[NS][4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    uint32_t lo[4], hi[4], t[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int j = j0 + 4 * q + i;
                        const uint32_t o = jo[j];
                        uint64_t x = 0;
                        if (o != ~0u)
                            x = NS > 4 ? reinterpret_cast<const uint64_t *>(a.eri)[o + m]
                                       : reinterpret_cast<const uint32_t *>(a.eri)[o + m];
                        lo[i] = (uint32_t)x;
                        hi[i] = (uint32_t)(x >> 32);
                    }
                    i8_transpose4(lo, t);
#pragma unroll
                    for (int u = 0; u < 4; u++) w[u][q] = t[u];
                    if constexpr (NS > 4) {
                        i8_transpose4(hi, t);
#pragma unroll
                        for (int u = 4; u < NS; u++) w[u][q] = t[u - 4];
                    }
                }
#pragma unroll
                for (int u = 0; u < NS; u++) i8_tm_st(tl + kACol + 16 * u + j0 / 4, w[u]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            i8_sync_or<kIExt>(1, false);
            if (tid == 0) i8_arrive(bar_a);
            const uint8_t *fl = a.flags + (size_t)Ia * nchunk;
            uint32_t f = GRADED ? 0 : fl[0];
            for (int c = 0; c < nchunk; c++, g++) {
                const uint32_t acc = NACC == 2 ? g & 1 : 0;
                T *Ts = reinterpret_cast<T *>(smem + L.t + (g & 1) * L.tstride);
                // the chunk's digits are there (which orders the loaders' scales and
                // mode before the reads here), the gather of two chunks back is done,
                // this chunk's MMAs are
                int md;
                if constexpr (GRADED) {
                    ok = ok && i8_wait(bar_full + 8 * r, par);
                    md = mode[r];
                } else {  // known from the string's flags; FP64's integers need no scales here
                    md = f & kISame ? kIOne : kIEach;
                    f = c + 1 < nchunk ? fl[c + 1] : 0;
                    if (md != kIOne) ok = ok && i8_wait(bar_full + 8 * r, par);
                }
                const bool bad = md == kIBad || !hfin, ints = NS == 7 && md == kIOne && hfin;
                ok = ok && (g < 2 || i8_wait(bar_tfree + 8 * (g & 1), ((g >> 1) - 1) & 1));
                ok = ok && i8_wait(bar_done + 8 * acc, (g / NACC) & 1);
                ok = __all_sync(~0u, ok);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                constexpr int CW = kIC / (kIExt / 4);  // columns per warp
                const int cw = CW * (warp >> 2);
                const uint32_t ta = tl + acc * (NU * kIC) + cw;
                bool freed = false;
                // (a quarter without panel rows has nothing to extract)
                if (ok && !bad && 32 * (warp & 3) >= a.nrow) {
                } else if (ok && ints) {
                    if constexpr (NS == 7) {
                        long long *Ti = reinterpret_cast<long long *>(Ts) + m * kIP + cw;
#pragma unroll
                        for (int h = 0; h < CW; h += 4) {
                            int w[NU][4];
#pragma unroll
                            for (int s = 0; s < NU; s++) i8_tm_ld(ta + s * kIC + h, w[s]);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            if (h + 4 == CW) {
                                // all read: the next chunk's MMAs may start
                                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                                __syncwarp();
                                if (lane == 0) i8_arrive(bar_free + 8 * acc);
                                freed = true;
                            }
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                int d[NU];
#pragma unroll
                                for (int s = 0; s < NU; s++) d[s] = w[s][i];
                                Ti[h + i] = i8_join(d);
                            }
                        }
                    }
                } else if (ok && !bad) {
                    const T *scc = scs + r * kIC + cw;
#pragma unroll 1
                    for (int h = 0; h < CW; h += 4) {
                        int w[NU][4];
#pragma unroll
                        for (int s = 0; s < NU; s++) i8_tm_ld(ta + s * kIC + h, w[s]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            int d[NU];
#pragma unroll
                            for (int s = 0; s < NU; s++) d[s] = w[s][i];
                            Ts[m * kIP + cw + h + i] = i8_value(d) * rs * scc[h + i];
                        }
                    }
                } else if (ok) {
                    // an infinity or NaN among the elements or the integrals: the
                    // products from c and the integrals themselves
                    for (int idx = tid; idx < kIM * kIC; idx += 32 * kIExt) {
                        const int mm = idx / kIC, cc = idx - mm * kIC, col = c * kIC + cc;
                        const int pm = a.rowpair[mm];
                        T y = T(0);
                        if (col < a.nb && pm >= 0)
                            for (int j = 0; j < K; j++) {
                                const long long o = (long long)j * a.na + Ia;
                                const uint32_t e = a.fsA[o];
                                T h = a.m2[eri_index(a.fpA[o], pm)];
                                if (e >> 31) h = -h;
                                y = fma(h, V[(long long)(e & 0x3fffffffu) * a.nb + col], y);
                            }
                        Ts[mm * kIP + cc] = y;
                    }
                }
                if (tid == 0) tint[g & 1] = ints;
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (ok && lane == 0) {
                    if (!freed) i8_arrive(bar_free + 8 * acc);
                    i8_arrive(bar_t + 8 * (g & 1));
                }
                if (++r == kIRing) { r = 0; par ^= 1; }
            }
        }
        failed = failed || !ok;
    }
    if (failed && status) *(volatile int *)status = 1;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem)
                     : "memory");
    }
}

template <typename T>
jci_status i8_fill_t(I8Tables *t, const double *m2, cudaStream_t st) {
    constexpr int p = sizeof(T) == 8 ? 0 : 1;
    k_i8_eri<T, kDigits<T>><<<kIM, 128, 0, st>>>(t->npair, t->rowpair, m2, t->mx, t->eri[p],
                                                 (T *)t->rscale[p]);
    JCI_CUDA(cudaGetLastError());
    return JCI_OK;
}

}  // namespace

// Panel rows, chunk lists and (empty) digit tables of a space.  JCI_ERR_SPACE
// outside the engine's limits: at most 64 alpha singles, 127 pairs moved by
// the beta singles (n <= 16 active orbitals), 65 534 beta strings.
jci_status i8_tables_build(const jci_space *s, int npair, I8Tables *t) {
    const SpinSpace &A = s->sp[0], &B = s->sp[1];
    const int nb = B.nstr;
    if (nb < 1 || nb > 65534 || A.max_sing < 1 || A.max_sing > 64) return JCI_ERR_SPACE;
    std::vector<int> row(npair, -1), rowpair(kIM, -1);
    int nr = 0;
    auto add = [&](int p) {
        if (row[p] < 0) {
            if (nr < kIM) rowpair[nr] = p;
            row[p] = nr++;
        }
    };
    for (const Exc &x : B.sing) add(pair_index(x.io0, x.fo0));
    if (nr > kIM - 1) return JCI_ERR_SPACE;
    const int nchunk = (nb + kIC - 1) / kIC;
    struct Tgt {
        int b, n;
        std::vector<uint16_t> e;
    };
    std::vector<std::vector<Tgt>> ch(nchunk);
    auto put = [&](int c, int b, int m, int col, bool neg) {
        auto &v = ch[c];
        if (v.empty() || v.back().b != b) v.push_back({b, 0, {}});
        v.back().e.push_back((uint16_t)((m * kIP + col) * 8) | (neg ? 1u : 0u));
    };
    for (int i = 0; i < nb; i++) {
        for (long long k = B.soff[i]; k < B.soff[i + 1]; k++) {
            const Exc &x = B.sing[k];
            put(x.target / kIC, i, row[pair_index(x.io0, x.fo0)], x.target % kIC, x.sign < 0);
        }
    }
    std::vector<uint32_t> lofs(nchunk + 1, 0);
    std::vector<uint16_t> blob;
    int lmax = 1;
    for (int c = 0; c < nchunk; c++) {
        auto &v = ch[c];
        // lanes per string (a power of two) and entries per lane
        auto lanes = [](const Tgt &x) {
            int l = 0;
            while ((int)x.e.size() > (kISeg << l)) l++;
            return l;
        };
        auto len = [&](const Tgt &x) { return ((int)x.e.size() + (1 << lanes(x)) - 1) >> lanes(x); };
        std::stable_sort(v.begin(), v.end(), [&](const Tgt &x, const Tgt &y) {
            return lanes(x) != lanes(y) ? lanes(x) > lanes(y) : len(x) > len(y);
        });
        struct Grp {
            int l;
            std::vector<int> tgt;
        };
        std::vector<Grp> gs;
        for (int i = 0; i < (int)v.size(); i++) {
            const int l = lanes(v[i]);
            if (l > 5) return JCI_ERR_SPACE;
            if (gs.empty() || gs.back().l != l || (int)(gs.back().tgt.size() << l) == 32)
                gs.push_back({l, {}});
            gs.back().tgt.push_back(i);
        }
        const int ng = (int)gs.size();
        const size_t o = blob.size();            // in 16-bit units, a multiple of 8
        const size_t tgo = 8 + 4 * (size_t)ng;   // strings behind the groups' heads
        blob.resize(o + tgo + 32 * (size_t)ng, 0xffff);
        blob[o] = (uint16_t)ng;
        blob[o + 1] = 0;
        for (int g = 0; g < ng; g++) {
            const int l = gs[g].l;
            size_t k1 = 0;
            for (int i : gs[g].tgt) k1 = std::max(k1, (size_t)len(v[i]));
            const size_t eo = blob.size(), off = 2 * (eo - o);
            uint16_t *h = &blob[o + 8 + 4 * g];
            h[0] = (uint16_t)off;
            h[1] = (uint16_t)(off >> 16);
            h[2] = (uint16_t)k1;
            h[3] = (uint16_t)l;
            blob.resize(eo + 32 * k1, (uint16_t)(kIZero * 8));
            for (int q = 0; q < (int)gs[g].tgt.size(); q++) {
                const Tgt &x = v[gs[g].tgt[q]];
                blob[o + tgo + 32 * g + (q << l)] = (uint16_t)x.b;
                const int n1 = len(x);
                for (int k = 0; k < (int)x.e.size(); k++)
                    blob[eo + 32 * (k % n1) + (q << l) + k / n1] = x.e[k];
            }
        }
        blob.resize((blob.size() + 7) / 8 * 8, 0);
        lofs[c + 1] = (uint32_t)(blob.size() / 8);
        lmax = std::max(lmax, (int)(lofs[c + 1] - lofs[c]));
        std::vector<Tgt>().swap(v);
    }
    t->na = A.nstr;
    t->nb = nb;
    t->npair = npair;
    t->nchunk = nchunk;
    t->nrow = nr;
    t->lmax = lmax;
    auto up = [&](auto **dst, const auto *src, size_t n) {
        return cudaMalloc((void **)dst, n * sizeof(**dst)) != cudaSuccess ||
               cudaMemcpy(*dst, src, n * sizeof(**dst), cudaMemcpyHostToDevice) != cudaSuccess;
    };
    bool bad = up(&t->rowpair, rowpair.data(), rowpair.size()) ||
               up(&t->lofs, lofs.data(), lofs.size()) ||
               up(&t->lists, blob.data(), blob.size());
    for (int p = 0; p < 2 && !bad; p++) {
        const int ns = p ? kDigits<float> : kDigits<double>;
        bad = cudaMalloc((void **)&t->eri[p], (size_t)2 * npair * kIM * (ns > 4 ? 8 : 4)) != cudaSuccess ||
              cudaMalloc(&t->rscale[p], kIM * sizeof(double)) != cudaSuccess;
    }
    bad = bad || cudaMalloc((void **)&t->mx, (kIM + 1) * sizeof(*t->mx)) != cudaSuccess;
    if (bad) {
        cudaGetLastError();
        i8_tables_free(t);
        return JCI_ERR_NOMEM;
    }
    return JCI_OK;
}

void i8_tables_free(I8Tables *t) {
    cudaFree(t->rowpair);
    cudaFree(t->mx);
    cudaFree(t->lofs);
    cudaFree(t->lists);
    for (int p = 0; p < 2; p++) {
        cudaFree(t->eri[p]);
        cudaFree(t->rscale[p]);
        cudaFree(t->scratch[p]);
    }
    *t = I8Tables();
}

// Digit tables of the current integrals (both precisions).
jci_status i8_fill(I8Tables *t, const double *m2, cudaStream_t st) {
    JCI_CUDA(cudaMemsetAsync(t->mx, 0, (kIM + 1) * sizeof(*t->mx), st));
    k_i8_erimax<<<kIM, 256, 0, st>>>(t->npair, t->rowpair, m2, t->mx);
    jci_status r = i8_fill_t<double>(t, m2, st);
    return r ? r : i8_fill_t<float>(t, m2, st);
}

template <typename T>
static size_t i8_smem_bytes(const I8Tables &t, int sa) {
    return i8_layout<T, true>(sa <= 32 ? 32 : 64, t.lmax).total;  // the larger one
}

size_t i8_smem(const I8Tables &t, int sa, size_t w) {
    return w == 8 ? i8_smem_bytes<double>(t, sa) : i8_smem_bytes<float>(t, sa);
}

// Scratch of one precision: column maxima, numbers of strings and their kinds
// (zeroed before each use), column scales, masks, flags, lists of strings, digits; the byte
// offset of each.
struct I8Scratch {
    size_t nstr, kind, scale, masks, flags, strs, sl, total;
};
static I8Scratch i8_scratch_layout(const I8Tables &t, size_t w, int ns) {
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t blocks = (size_t)t.nchunk * t.na;
    I8Scratch l;
    l.nstr = up((size_t)t.nb * 4);
    l.kind = l.nstr + up(3 * sizeof(int));
    l.scale = l.kind + up((size_t)t.na + 15);
    l.masks = l.scale + up((size_t)t.nchunk * kIC * w);
    l.flags = l.masks + up(blocks * sizeof(I8Mask));
    l.strs = l.flags + up(blocks);
    l.sl = l.strs + up(2 * (size_t)t.na * sizeof(int));
    l.total = l.sl + blocks * ns * kIC;
    return l;
}

jci_status i8_scratch(I8Tables *t, size_t w, size_t most) {
    const int p = w == 8 ? 0 : 1, ns = p ? kDigits<float> : kDigits<double>;
    if (t->scratch[p]) return JCI_OK;
    const size_t bytes = i8_scratch_layout(*t, w, ns).total;
    if (bytes <= most && cudaMalloc(&t->scratch[p], bytes) == cudaSuccess) return JCI_OK;
    cudaGetLastError();
    t->scratch[p] = nullptr;
    return JCI_ERR_NOMEM;
}

// o += the alpha-single x beta-single part of H v.
template <typename T>
jci_status i8_launch(const I8Tables &t, const I8Input<T> &in, int device, const T *v, T *o,
                     int *status, int expire, cudaStream_t st) {
    constexpr int p = sizeof(T) == 8 ? 0 : 1;
    unsigned char *base = (unsigned char *)t.scratch[p];
    if (!base || in.sa > 64) return JCI_ERR_STATE;
    const I8Scratch l = i8_scratch_layout(t, sizeof(T), kDigits<T>);
    uint32_t *mx = (uint32_t *)base;
    int *nstr = (int *)(base + l.nstr), *strs = (int *)(base + l.strs);
    T *cscale = (T *)(base + l.scale);
    I8Mask *masks = (I8Mask *)(base + l.masks);
    uint8_t *flags = base + l.flags, *sl = base + l.sl;
    JCI_CUDA(cudaMemsetAsync(base, 0, l.scale, st));
    dim3 g1((t.nb + 127) / 128, (t.na + 63) / 64);
    k_i8_colmax<T><<<g1, 256, 0, st>>>(t.na, t.nb, v, mx, in.skip);
    dim3 g2(t.nchunk, (t.na + 15) / 16);
    k_i8_slice<T><<<g2, 192, 0, st>>>(t.na, t.nb, v, mx, sl, cscale, masks, in.skip);
    k_i8_grade<<<t.na, 128, 0, st>>>(t.na, t.nchunk, in.sa, in.fsA, masks, flags, base + l.kind,
                                     nstr, strs, in.skip);
    I8Args<T> a;
    a.na = t.na; a.nb = t.nb; a.nchunk = t.nchunk; a.nrow = t.nrow; a.K = in.sa; a.KP = in.sa <= 32 ? 32 : 64;
    a.fsA = in.fsA; a.fpA = in.fpA; a.m2 = in.m2;
    a.eri = t.eri[p]; a.rscale = (const T *)t.rscale[p]; a.rowpair = t.rowpair;
    a.sl = sl; a.cscale = cscale; a.flags = flags; a.nstr = nstr; a.strs = strs;
    a.vec = (size_t)t.nb * sizeof(T) % 16 == 0 && reinterpret_cast<uintptr_t>(v) % 16 == 0;
    a.lofs = t.lofs; a.lists = (const uint4 *)t.lists; a.lmax = t.lmax;
    a.npair = t.npair;
    a.expire = expire;
    a.skip = in.skip;
    int nsm = 0;
    JCI_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    const int grid = std::min(t.na, nsm);
    JCI_CUDA(smem_optin(k_sigma_i8<T, false>));
    JCI_CUDA(smem_optin(k_sigma_i8<T, true>));
    k_sigma_i8<T, false>
        <<<grid, kIThreads, i8_layout<T, false>(a.KP, t.lmax).total, st>>>(a, v, o, status);
    k_sigma_i8<T, true>
        <<<grid, kIThreads, i8_layout<T, true>(a.KP, t.lmax).total, st>>>(a, v, o, status);
    JCI_CUDA(cudaGetLastError());
    return JCI_OK;
}

template jci_status i8_launch<double>(const I8Tables &, const I8Input<double> &, int,
                                      const double *, double *, int *, int, cudaStream_t);
template jci_status i8_launch<float>(const I8Tables &, const I8Input<float> &, int, const float *,
                                     float *, int *, int, cudaStream_t);

}  // namespace jci
