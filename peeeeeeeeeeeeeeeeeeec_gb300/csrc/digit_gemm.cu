// C -= A B in FP64 accuracy on the tensor cores.
//
// GB300 issues 2 FP64 FMA per clock and SM (1.25 TFLOP/s) and 4096 BF16 ones
// (2 PFLOP/s), so a contraction is far cheaper as many exact BF16 products.
// The method is the error-free splitting of Ozaki, Ogita, Oishi and Rump
// (Numerical Algorithms 59, 2012), with integer digits.  The rows of B are
// scaled to a common size by powers of two, the columns of A by their inverses
// (an LU of badly scaled rows has L's columns grow as U's rows shrink); then
// every row of A and every column of B is scaled by a power of two to a 2-norm
// of at most 1 and cut into kDigits balanced digits of seven bits, x = sum_i d_i
// 2^(1 - 7 i), |d_i| <= 64 -- integers that BF16 holds exactly.  The product of
// digits i and j has weight 2^(2 - 7 (i + j)): the pairs with the same sum i + j
// up to kDigits + 1 are added up in one TMEM accumulator each.  A sum of up to ten
// pairs is an integer below 2^24 (10 x 2 K x 2^12 at K = 192 complex, 10 x K x 2^12 at K
// = 256 real), so FP32 accumulation is exact; the last two complex sums, of eleven and
// twelve pairs, could pass 2^24 and then round by a unit, 2^-82 and 2^-89.
//
// The sums are combined in 90-bit integers of unit 2^-89 and leave them once,
// rounded to FP64, for the subtraction from C: the only FP64 operation of an
// update.  Its error is what is dropped, the pairs i + j >= 14: about 2^-78 |row of A|
// |column of B| for digits that look random, 2^-72 at worst (11 x 2 K x 2^12 x 2^-96, all
// of one sign).
// A chain of K FP64 FMAs rounds at 2^-53 of its running sum, so entries whose C
// and update are both below 2^-kExactBelow |row| |column| are left out and done
// in FP64 (matrices of weakly coupled parts, systems at kHz).  Complex entries are
// looked at by their real and imaginary parts, as a chain rounds each for itself
// (small resistances beside j omega L); parts that are exactly zero, because no
// product has both factors (lossless systems), are told by bit masks of the
// operands' nonzero parts and cost nothing.  Down to that line an entry or part is then
// no less accurate than on the FP64 pipe, for digits that look random.  (Eleven digits, 66 pairs, with the line
// at 2^-18: 5% faster on random matrices, but 341 against 294 ms for the solve of
// the 8402-unknown box, where more entries take the FP64 way.)
//
// Operands.  Two kernels write the digits in the layout that the MMA reads
// from shared memory (K-major rows of 16 BF16 = 32 bytes, 32-byte swizzle),
// one contiguous block per (128-row or 48 / 96-column tile, 16 of K, digit),
// so that an untiled bulk copy brings each block and no tensor map is built.
// Complex: A holds Ar, Ai; B holds -Bi, Br, Bi (48 columns each), so that the
// 96-column windows [Br; Bi] and [-Bi; Br] give Re and Im side by side:
//   [Re | Im] += Ar [Br; Bi]^T + Ai [-Bi; Br]^T.
#include "digit_gemm.cuh"

#include <cuda_bf16.h>

#include <limits.h>

#include <algorithm>
#include <type_traits>

#include "../../include/peec_gb300.h"
#include "common.cuh"
#include "tc_gemm.cuh"

namespace peec {
namespace dg {

using tc::fence_after_sync;
using tc::fence_before_sync;
using tc::mbar_arrive;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::mma_bf16;
using tc::mma_commit;
using tc::smem_u32;

static const int kDigits = 12;              // 78 digit pairs
static const int kLowBits = 7 * (kDigits - 9);  // of the digits kept apart while they are cut (63 bits hold nine)
static const int kUnit = 7 * (kDigits + 1) - 2;  // sums are in units of 2^-kUnit
static const int kBM = 128;  // rows of a tile
static const int kKC = 16;   // K of a block: one MMA
static const int kNotFinite = 1 << 28;  // exponent of a row or column with an infinity or NaN

static const int kEpiWarps = 12;  // three per 32 rows, a third of the columns each

template <bool CX>
struct Shape {
    typedef typename std::conditional<CX, double2, double>::type Scalar;
    static constexpr int BN = CX ? 48 : 96;               // columns of a tile: 96 accumulator columns
    static constexpr int kABytes = CX ? 8192 : 4096;      // digits of one (tile, K block, digit)
    static constexpr int kBPart = CX ? 1536 : 3072;       // 48 (96) rows of 32 bytes
    static constexpr int kBBytes = CX ? 3 * kBPart : kBPart;
    static constexpr int kBytes = kABytes + kBBytes;
    static constexpr int kBuffers = CX ? 13 : 22;         // shared-memory ring of digit blocks
    static constexpr int kCols = CX ? 4 : 8;              // columns of an epilogue chunk: 64 bytes
    static constexpr int kWarpCols = CX ? 16 : 32;        // columns of an epilogue warp: 32 sums a thread
    static constexpr int kChunks = kWarpCols / kCols;
    static constexpr int kRowStride = CX ? 80 : 72;       // padded bytes of a chunk's row (conflict-free)
    static constexpr int kChunkBytes = 32 * kRowStride;   // two chunks per warp
    static constexpr size_t kSmem = (size_t)kBuffers * kBytes + (size_t)kEpiWarps * 2 * kChunkBytes + 512 + 1024;
};

// ---- digits ----------------------------------------------------------
static const int kZero = -(1 << 20);  // exponent of a zero

// biased exponent of x 2^shift; kZero for a zero or subnormal x
__device__ __forceinline__ int exponent(double x, int shift) {
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return ex == 0 ? kZero : ex + shift;
}
__device__ __forceinline__ bool not_finite(double x) { return ((__double_as_longlong(x) >> 52) & 0x7ff) == 0x7ff; }

// The square of x 2^(shift + 1022 - emax) (below 1), rounded up by about 2^-19:
// a row's sum of squares bounds its 2-norm.
__device__ __forceinline__ float square_up(double x, int shift, int emax) {
    const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(x) >> 32);
    const int ex = (int)(hi >> 20 & 0x7ff) + shift - emax + 126;  // biased FP32 exponent
    if (ex < 64 || (hi & 0x7ff00000u) == 0) return 0.0f;          // below 2^-62: within the margin of norm_shift
    const float y = __uint_as_float(((unsigned)ex << 23 | (hi & 0xfffffu) << 3) + 8);
    return y * y;
}
// t with sum of squares <= 4^t (with a margin for its own rounding), 0 .. 5
__device__ __forceinline__ int norm_shift(float sq) {
    sq *= 1.0001f;
    return (sq > 1.0f) + (sq > 4.0f) + (sq > 16.0f) + (sq > 64.0f) + (sq > 256.0f);
}

// The scaled x 2^(shift + 1022 - emax) (emax: at least the biased exponent of x
// 2^shift, so that it is below 1) in units of 2^(1 - 7 kDigits), as hi 2^kLowBits + lo,
// 0 <= lo < 2^kLowBits: the lowest digits in lo, nine in hi.
struct Fixed {
    long long hi;
    unsigned lo;
};
__device__ __forceinline__ Fixed fixed_point(double x, int shift, int emax) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7ff);
    Fixed r = {0, 0u};
    if (ex == 0) return r;
    const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    constexpr unsigned mask = (1u << kLowBits) - 1u;
    const int sh = ex + shift - emax + 9 + kLowBits;  // at most 9 + kLowBits
    unsigned long long hi;
    if (sh >= kLowBits) {
        hi = m << (sh - kLowBits);
    } else if (sh >= 0) {
        hi = m >> (kLowBits - sh);
        r.lo = (unsigned)(m << sh) & mask;
    } else if (sh > -56) {
        const unsigned long long v = (m + (1ull << (-sh - 1))) >> -sh;
        hi = v >> kLowBits;
        r.lo = (unsigned)v & mask;
    } else {
        hi = 0;
    }
    r.hi = (long long)hi;
    if (b >> 63) {
        r.hi = (long long)(~hi + (r.lo == 0 ? 1u : 0u));
        r.lo = (0u - r.lo) & mask;
    }
    return r;
}

// ef[r]: exponent of the largest |entry| of row r of B (0 for a zero row): B's
// rows are divided by 2^ef, A's columns multiplied.  One block per row.
template <bool CX>
__global__ void __launch_bounds__(256) k_row_exponents(const double *B, size_t ldb, int n, int *ef, unsigned *exact,
                                                       const int *code) {
    if (*code != 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *exact = 0;
    __shared__ int s_max[8];
    const double *row = B + (size_t)blockIdx.x * ldb * (CX ? 2 : 1);
    int e = 0;
    for (int j = threadIdx.x; j < (CX ? 2 : 1) * n; j += 256)
        if (!not_finite(row[j])) e = max(e, (int)((__double_as_longlong(row[j]) >> 52) & 0x7ff));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, s));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) e = max(e, s_max[w]);
        ef[blockIdx.x] = e == 0 ? 0 : e - 1022;
    }
}

// Bit masks of a complex row of A or column of B: which of its (up to kMaskWords 32)
// real and imaginary parts are not zero.
static const int kMaskWords = 6;
struct Mask {
    unsigned re[8], im[8];
};
__device__ __forceinline__ void store_mask(Mask *masks, int i, int o, const double (*x)[2]) {
    unsigned re = 0, im = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        re |= (__double_as_longlong(x[t][0]) << 1) != 0 ? 1u << t : 0u;
        im |= (__double_as_longlong(x[t][1]) << 1) != 0 ? 1u << t : 0u;
    }
    reinterpret_cast<unsigned char *>(masks[i].re)[o] = (unsigned char)re;
    reinterpret_cast<unsigned char *>(masks[i].im)[o] = (unsigned char)im;
}

// The lowest balanced digit (-64 .. 63) of X; X <- (X - digit) / 128.  s: its
// number, counted from 0; the last one left is the leading digit (-64 .. 64).
__device__ __forceinline__ float next_digit(Fixed &X, int s) {
    int d;
    if (s >= 9) {  // the lowest, in lo, then a carry into hi
        d = (int)(X.lo << 25) >> 25;
        X.lo = (unsigned)((int)X.lo - d) >> 7;
        if (s == 9) X.hi += X.lo;
    } else if (s > 0) {
        d = (int)((unsigned)X.hi << 25) >> 25;
        X.hi = (X.hi - d) >> 7;
    } else {
        d = (int)X.hi;
    }
    return (float)d;
}
// two integers up to 256 in magnitude as packed BF16 (exact)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

// Eight fixed-point values (consecutive in K) as one 16-byte row piece of
// each digit: out + (digit - 1) * stride.  neg (optional): the negated digits.
__device__ __forceinline__ void store_digits(const Fixed *X0, unsigned char *out, size_t stride,
                                             unsigned char *neg) {
    Fixed X[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) X[t] = X0[t];
#pragma unroll
    for (int s = kDigits - 1; s >= 0; --s) {
        float f[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) f[t] = next_digit(X[t], s);
        uint4 w;
        w.x = pack_bf16(f[0], f[1]);
        w.y = pack_bf16(f[2], f[3]);
        w.z = pack_bf16(f[4], f[5]);
        w.w = pack_bf16(f[6], f[7]);
        *reinterpret_cast<uint4 *>(out + (size_t)s * stride) = w;
        if (neg) {
            // flip both signs; a zero keeps its sign bit irrelevant
            w.x ^= 0x80008000u;
            w.y ^= 0x80008000u;
            w.z ^= 0x80008000u;
            w.w ^= 0x80008000u;
            *reinterpret_cast<uint4 *>(neg + (size_t)s * stride) = w;
        }
    }
}

// byte offset of row r, K half o of a 16-column block (32-byte swizzle)
__device__ __forceinline__ int swizzled(int r, int o) { return r * 32 + ((o ^ ((r >> 2) & 1)) << 4); }

// Digits of A's rows: TPR threads per row (K <= 8 TPR), each eight consecutive
// entries.
template <bool CX, int TPR>
__global__ void __launch_bounds__(256) k_digits_rows(const double *A, size_t lda, int m, int k, int kc_count,
                                                     unsigned char *out, int *ea, Mask *masks, const int *ef,
                                                     const int *code) {
    if (*code != 0) return;
    constexpr int P = CX ? 2 : 1;
    const int row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, o = threadIdx.x % TPR;
    double x[8][P];
    int f[8];
    int emax = kZero;
    bool bad = false;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int c = 8 * o + t;
        f[t] = c < k ? ef[c] : 0;
#pragma unroll
        for (int p = 0; p < P; ++p) x[t][p] = 0.0;
        if (row < m && c < k) {
            if constexpr (CX) {
                const double2 z = reinterpret_cast<const double2 *>(A)[(size_t)row * lda + c];
                x[t][0] = z.x;
                x[t][P - 1] = z.y;
            } else {
                x[t][0] = A[(size_t)row * lda + c];
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            emax = max(emax, exponent(x[t][p], f[t]));
            bad |= not_finite(x[t][p]);
        }
    }
#pragma unroll
    for (int s = TPR / 2; s > 0; s >>= 1) {
        emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, s));
        bad |= (bool)__shfl_xor_sync(0xffffffffu, (int)bad, s);
    }
    float sq = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int p = 0; p < P; ++p) sq += square_up(x[t][p], f[t], emax);
#pragma unroll
    for (int s = TPR / 2; s > 0; s >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
    emax += norm_shift(sq);
    if (o == 0) ea[row] = bad ? kNotFinite : emax < kZero / 2 ? kZero : emax - 1022;
    if constexpr (CX) store_mask(masks, row, o, x);
    if (o >= 2 * kc_count) return;
    const int tile = row / kBM, r = row % kBM;
    unsigned char *base = out + (size_t)(tile * kc_count + (o >> 1)) * kDigits * Shape<CX>::kABytes + swizzled(r, o & 1);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        Fixed X[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) X[t] = bad ? Fixed{0, 0u} : fixed_point(x[t][p], f[t], emax);
        store_digits(X, base + p * 4096, Shape<CX>::kABytes, nullptr);
    }
}

// Digits of B's columns: 64 columns per block, eight threads per column, each
// eight consecutive rows at a time: once for the exponents, once for the digits
// (the second read is from the caches).
template <bool CX>
__device__ __forceinline__ void load_rows(const double *B, size_t ldb, int n, int k, int col, int r0, const int *ef,
                                          double (*x)[CX ? 2 : 1], int *f) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int r = r0 + t;
        f[t] = 0;
        x[t][0] = x[t][CX ? 1 : 0] = 0.0;
        if (col < n && r < k) {
            f[t] = -ef[r];
            if constexpr (CX) {
                const double2 z = reinterpret_cast<const double2 *>(B)[(size_t)r * ldb + col];
                x[t][0] = z.x;
                x[t][1] = z.y;
            } else {
                x[t][0] = B[(size_t)r * ldb + col];
            }
        }
    }
}

template <bool CX>
__global__ void __launch_bounds__(512) k_digits_cols(const double *B, size_t ldb, int n, int k, int kc_count,
                                                     unsigned char *out, int *eb, Mask *masks, const int *ef,
                                                     const int *code) {
    if (*code != 0) return;
    constexpr int P = CX ? 2 : 1;
    __shared__ int s_max[8][64];
    __shared__ float s_sq[8][64];
    __shared__ int s_bad[64];
    const int cx = threadIdx.x & 63, ty = threadIdx.x >> 6;
    const int col = blockIdx.x * 64 + cx;
    if (ty == 0) s_bad[cx] = 0;
    __syncthreads();
    double x[8][P];
    int f[8];
    int emax = kZero;
    float sq = 0.0f;  // sum of squares relative to emax
    bool bad = false;
    for (int o = ty; o < 2 * kc_count; o += 8) {
        load_rows<CX>(B, ldb, n, k, col, 8 * o, ef, x, f);
        int e = emax;
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int p = 0; p < P; ++p) {
                e = max(e, exponent(x[t][p], f[t]));
                bad |= not_finite(x[t][p]);
            }
        if (e > emax) {
            sq = e - emax < 60 ? sq * exp2f((float)(2 * (emax - e))) : 0.0f;
            emax = e;
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int p = 0; p < P; ++p) sq += square_up(x[t][p], f[t], emax);
    }
    s_max[ty][cx] = emax;
    s_sq[ty][cx] = sq;
    if (bad) s_bad[cx] = 1;
    __syncthreads();
    bad = s_bad[cx] != 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) emax = max(emax, s_max[t][cx]);
    sq = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int d = emax - s_max[t][cx];
        if (d < 60) sq += s_sq[t][cx] * exp2f((float)(-2 * d));
    }
    emax += norm_shift(sq);
    const int tile = col / Shape<CX>::BN, r = col % Shape<CX>::BN;
    if (tile >= (n + Shape<CX>::BN - 1) / Shape<CX>::BN) return;
    if (ty == 0) eb[col] = bad ? kNotFinite : emax < kZero / 2 ? kZero : emax - 1022;
    for (int o = ty; o < (2 * kc_count + 3) / 4 * 4; o += 8) {
        load_rows<CX>(B, ldb, n, k, col, 8 * o, ef, x, f);
        if constexpr (CX) store_mask(masks, col, o, x);
        if (o >= 2 * kc_count) break;
        unsigned char *base =
            out + (size_t)(tile * kc_count + (o >> 1)) * kDigits * Shape<CX>::kBBytes + swizzled(r, o & 1);
        Fixed X[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) X[t] = bad ? Fixed{0, 0u} : fixed_point(x[t][0], f[t], emax);
        store_digits(X, base + (CX ? Shape<CX>::kBPart : 0), Shape<CX>::kBBytes, nullptr);  // Br
        if constexpr (CX) {
#pragma unroll
            for (int t = 0; t < 8; ++t) X[t] = bad ? Fixed{0, 0u} : fixed_point(x[t][1], f[t], emax);
            store_digits(X, base + 2 * Shape<CX>::kBPart, Shape<CX>::kBBytes, base);  // Bi, -Bi
        }
    }
}

// ---- product ---------------------------------------------------------
__device__ __forceinline__ void bulk_load(void *smem_dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Shared-memory matrix descriptor, K-major, 32-byte swizzle: rows of 32
// bytes, groups of 8 rows 256 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)6 << 61;
}

// The integer that a sum's FP32 value is (|x| <= 2^24), with fixed-latency
// operations: F2I issues at an eighth of their rate.
__device__ __forceinline__ int integer(float x) {
    const float M = 12582912.0f;  // 1.5 2^23: x + M holds x in its low bits for |x| <= 2^22
    const float t = fmaf(x, 0x1p-11f, M);
    const float r = fmaf(t - M, -2048.0f, x);  // |r| <= 1024, exact
    return (__float_as_int(t) - 0x4B400000) * 2048 + (__float_as_int(r + M) - 0x4B400000);
}

// v 2^E and `low` (kUnit - 61 bits) below it, as FP64 bits: rounded once
// to 53 bits by integer operations (an FP64 conversion takes one of GB300's two
// FP64 slots per clock and SM).  No branches: eight of these run interleaved.
// Results below 2^-1022 are zero.
__device__ __forceinline__ long long compose(long long v, unsigned low, int E) {
    const unsigned sign = (unsigned)((int)(v >> 32) >> 31);
    constexpr int bits = kUnit - 61;
    low = ((low ^ sign) & ((1u << bits) - 1u)) - sign;  // negated: ~x + 1 over both words
    const unsigned long long a = ((unsigned long long)v ^ ((unsigned long long)sign << 32 | sign)) + (low >> bits);
    unsigned hi = (unsigned)(a >> 32), lo = (unsigned)a;
    low <<= 32 - bits;
#pragma unroll
    for (int t = 0; t < 2; ++t) {  // leading zero words
        const bool z = hi == 0;
        hi = z ? lo : hi;
        lo = z ? low : lo;
        low = z ? 0u : low;
        E -= z ? 32 : 0;
    }
    const int c = __clz((int)hi);
    const unsigned h = __funnelshift_l(lo, hi, c), l = __funnelshift_l(low, lo, c);  // top bit 63
    const int be = 1086 - c + E;
    const unsigned ml = __funnelshift_r(l, h, 11), up = l >> 10 & 1u;
    const unsigned long long m = ((unsigned long long)(((unsigned)(be - 1) << 20) + (h >> 11)) << 32 | ml) + up;
    const bool tiny = be < 1 || h == 0, huge = be > 2046;
    const unsigned rh = tiny ? 0u : huge ? 0x7ff00000u : (unsigned)(m >> 32), rl = tiny || huge ? 0u : (unsigned)m;
    return (long long)((unsigned long long)(rh | (sign & 0x80000000u)) << 32 | rl);
}

// 8 consecutive FP32 columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "r"(taddr)
        : "memory");
}
// 8 words of this warp's 32 TMEM lanes out; 4 back below
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const int *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, int *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// the loads' results are complete (and not used earlier)
__device__ __forceinline__ void tmem_wait_ld(int *v, int *w) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3])::"memory");
}

struct Args {
    const unsigned char *a, *b;
    const int *ea, *eb;
    const Mask *ma, *mb;
    double *c;
    size_t ldc;
    const double *a64, *b64;  // the operands, for entries done in FP64
    size_t lda, ldb;
    int m, n, k, kc_count;
    unsigned *exact;       // entries done in FP64 so far
    unsigned exact_limit;  // beyond it *code becomes 7
    int *code;
};

static const int kExactBelow = 25;  // entries below 2^-25 of |row| |column| take the FP64 way
// |v| 2^-61 below 2^-kExactBelow
__device__ __forceinline__ bool below(long long v) {
    return (unsigned)((int)(v >> 32) + (1 << (29 - kExactBelow))) < (2u << (29 - kExactBelow));
}
// |z| below 2^(E - kExactBelow)
__device__ __forceinline__ bool below(double z, int E) {
    return (int)((__double_as_longlong(z) >> 52) & 0x7ff) < E + 1023 - kExactBelow;
}

// Parts of this lane's row (i) in columns j0 .. + 15 that are sums of zeros: bit c
// for the real part of column j0 + c, bit 16 + c for the imaginary one.  (An
// infinity or NaN times zero is none.)
__device__ __forceinline__ unsigned zero_parts(const Args &A, int i, int j0) {
    const int lane = threadIdx.x & 31, words = (2 * A.kc_count + 3) / 4;
    const bool bad = A.ea[i] >= kNotFinite;
    const unsigned bad_columns = __ballot_sync(0xffffffffu, A.eb[j0 + (lane & 15)] >= kNotFinite);
    unsigned re[kMaskWords], im[kMaskWords], zero = 0;
#pragma unroll
    for (int w = 0; w < kMaskWords; ++w) {
        re[w] = w < words ? A.ma[i].re[w] : 0u;
        im[w] = w < words ? A.ma[i].im[w] : 0u;
    }
#pragma unroll 2
    for (int c = 0; c < 16; ++c) {
        unsigned r = 0, s = 0;
#pragma unroll
        for (int w = 0; w < kMaskWords; ++w)
            if (w < words) {
                const unsigned br = A.mb[j0 + c].re[w], bi = A.mb[j0 + c].im[w];
                r |= (re[w] & br) | (im[w] & bi);
                s |= (re[w] & bi) | (im[w] & br);
            }
        zero |= (r == 0 ? 1u : 0u) << c | (s == 0 ? 0x10000u : 0u) << c;
    }
    return bad ? 0u : zero & ~bad_columns;
}

// One entry of C -= A B in FP64: K products from k0 on, `step` apart.
template <bool CX>
__device__ __forceinline__ double2 exact_sum(const Args &A, int i, int j, int k0, int step) {
    double2 z = make_double2(0.0, 0.0);
    if constexpr (CX) {
        const double2 *a = reinterpret_cast<const double2 *>(A.a64) + (size_t)i * A.lda;
        const double2 *b = reinterpret_cast<const double2 *>(A.b64) + j;
#pragma unroll 2
        for (int k = k0; k < A.k; k += step) {
            const double2 x = a[k], y = b[(size_t)k * A.ldb];
            z.x = fma(-x.y, y.y, fma(x.x, y.x, z.x));
            z.y = fma(x.y, y.x, fma(x.x, y.y, z.y));
        }
    } else {
        const double *a = A.a64 + (size_t)i * A.lda, *b = A.b64 + j;
#pragma unroll 4
        for (int k = k0; k < A.k; k += step) z.x = fma(a[k], b[(size_t)k * A.ldb], z.x);
    }
    return z;
}
template <bool CX>
__device__ __forceinline__ void exact_update(const Args &A, int i, int j, double2 z) {
    if constexpr (CX) {
        double2 *c = reinterpret_cast<double2 *>(A.c) + (size_t)i * A.ldc + j;
        const double2 y = *c;
        *c = make_double2(y.x - z.x, y.y - z.y);
    } else {
        A.c[(size_t)i * A.ldc + j] -= z.x;
    }
}
// The entries of rows row0 + lane whose column (from col0) has a bit in the lane's
// mask.  An FP64 instruction of a warp takes 64 cycles whatever its lanes do:
// with many lanes at work each takes an entry of its own, else the lanes share
// the products of one entry at a time (K = 192 complex: 768 instructions a round
// against 34 an entry).
template <bool CX>
__device__ __noinline__ void exact_entries(const Args &A, int row0, int col0, unsigned mask) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        const unsigned busy = __ballot_sync(0xffffffffu, mask != 0);
        if (busy == 0) return;
        if (__popc(busy) >= 20) {
            if (mask != 0) {
                const int j = col0 + __ffs((int)mask) - 1;
                mask &= mask - 1;
                exact_update<CX>(A, row0 + lane, j, exact_sum<CX>(A, row0 + lane, j, 0, 1));
            }
            __syncwarp();
            continue;
        }
        const int from = __ffs((int)busy) - 1;
        const int i = row0 + from, j = col0 + __ffs(__shfl_sync(0xffffffffu, (int)mask, from)) - 1;
        if (lane == from) mask &= mask - 1;
        double2 z = exact_sum<CX>(A, i, j, lane, 32);
        z.x = warp_sum(z.x);
        if constexpr (CX) z.y = warp_sum(z.y);
        if (lane == from) exact_update<CX>(A, i, j, z);
    }
}

__device__ __forceinline__ void copy_async(void *smem, const double2 *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_async(void *smem, const double *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }


// Passes of a tile over K: i + j = 13 .. 10, 9 .. 6, 5 .. 2, within a pass from the
// highest i + j down; the s-th sum of a pass is in accumulator s, 96 TMEM columns.
// The longest pass (42 pairs) comes first: it runs while the warps of the
// epilogue are busy with C of the tile before (with the leading sums first,
// 10 pairs, the MMAs then waited: 189k instead of 150k cycles a tile at K = 192).
// The 96 columns after the accumulators hold the epilogue's low words.
static const int kSlots = 4;
static const int kSlotCols = 96;
static const int kPasses = kDigits / kSlots;
static_assert(kDigits == kSlots * kPasses, "sums");
__host__ __device__ constexpr int pass_top(int pass) { return kDigits + 1 - kSlots * pass; }
__host__ __device__ constexpr int pass_digits(int pass) { return pass_top(pass) - 1; }
// A pass's digits (1-based) in the order in which a block's products are done
// with them, which is the order of their loads: top - 1, top - 2, ... (one for each
// sum but the last), then 1, n, 2, n - 1, ... of the rest.
__host__ __device__ constexpr int digit_order(int pass, int digit) {
    const int first = kSlots - 1, d = pass_digits(pass), rest = d - first;
    return digit > rest ? d - digit : first + (digit <= rest + 1 - digit ? 2 * (digit - 1) : 2 * (rest - digit) + 1);
}
__host__ __device__ constexpr int digit_at(int pass, int order) {
    for (int d = 1; d <= pass_digits(pass); ++d)
        if (digit_order(pass, d) == order) return d;
    return 0;
}

// MMAs and commits of a converged warp, issued by one elected lane: the warp's
// descriptors stay in uniform registers, where the instruction wants them (one
// lane's own branch around all of it cost about 90 cycles a pair).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void warp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    if (elect_one()) mma_bf16(d, a, b, idesc, more);
}
// the whole warp's answer: no lane goes on alone when the wait runs out
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void warp_commit(uint64_t *bar) {
    if (elect_one()) mma_commit(bar);
}

// The products of one K block in one pass, by one warp, every pair known at
// compile time (an MMA takes 48 cycles; with the pairs found at run time by one
// thread the issue took 340).
// ring: the ring slot of the block's first digit, phase: its use's parity.
template <bool CX, int PASS>
__device__ __forceinline__ bool issue_block(uint32_t base_addr, uint32_t tmem, int kc, int KC, int tile, int ring,
                                            uint32_t phase, uint64_t *full, uint64_t *empty, uint64_t *sum_full,
                                            uint64_t *sum_empty, volatile int *abort_flag) {
    typedef Shape<CX> S;
    constexpr uint32_t idesc = tc::idesc_bf16_f32(kBM, kSlotCols);
    constexpr int top = pass_top(PASS), bottom = top - kSlots + 1;
    const uint64_t desc0 = smem_desc_sw32(base_addr);
    uint32_t at[pass_digits(PASS)];  // ring slot of each digit of the block
    uint32_t wrapped = 0;
#pragma unroll
    for (int d = 0; d < pass_digits(PASS); ++d) {
        int r = ring + digit_order(PASS, d + 1);
        if (r >= S::kBuffers) {
            r -= S::kBuffers;
            wrapped |= 1u << d;
        }
        at[d] = (uint32_t)r;
    }
    auto desc = [&](int d) { return desc0 + (uint64_t)(at[d] * (uint32_t)(S::kBytes >> 4)); };
    auto ready = [&](int d) { return warp_wait(&full[at[d]], (phase ^ (wrapped >> d)) & 1u, abort_flag); };
    // release digit d (1-based) if this pair of sum g was its last in this block
    auto release = [&](int d, int g) {
        if (g == (d + 1 > bottom ? d + 1 : bottom)) warp_commit(&empty[at[d - 1]]);
    };
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        const int g = top - s;
        const uint32_t use = (uint32_t)(kPasses * tile + PASS);  // of this accumulator so far
        if (kc == 0) {
            if (use > 0 && !warp_wait(&sum_empty[s], (use - 1) & 1, abort_flag)) return false;
            fence_after_sync();
        }
        const uint32_t acc = tmem + (uint32_t)(s * kSlotCols);
#pragma unroll
        for (int v = 0; v < kDigits; ++v) {  // pairs (g - 1, 1), (1, g - 1), (g - 2, 2), ...
            if (v >= g - 1) continue;
            const int lo = (v >> 1) + 1, i = (v & 1) ? lo : g - lo, j = g - i;
            if (s == 0 && (v & 1) == 0) {  // every digit of the block is met here first
                if (!ready(i - 1) || (j != i && !ready(j - 1))) return false;
                fence_after_sync();
            }
            const uint64_t ad = desc(i - 1), bd = desc(j - 1) + (uint64_t)(S::kABytes >> 4);
            const uint32_t more = v > 0 || kc > 0 ? 1u : 0u;
            if constexpr (CX) {
                warp_mma(acc, ad, bd + (S::kBPart >> 4), idesc, more);  // Ar [Br; Bi]
                warp_mma(acc, ad + (4096 >> 4), bd, idesc, 1u);    // Ai [-Bi; Br]
            } else {
                warp_mma(acc, ad, bd, idesc, more);
            }
            if ((v & 1) || g == 2 * lo) {
                release(lo, g);
                if (g != 2 * lo) release(g - lo, g);
            }
        }
        if (kc == KC - 1) warp_commit(&sum_full[s]);
    }
    return true;
}

// A whole pass of one tile; advances the ring.
template <bool CX, int PASS>
__device__ __forceinline__ bool issue_pass(uint32_t base_addr, uint32_t tmem, int KC, int tile, int &ring,
                                           uint32_t &phase, uint64_t *full, uint64_t *empty, uint64_t *sum_full,
                                           uint64_t *sum_empty, volatile int *abort_flag) {
    for (int kc = 0; kc < KC; ++kc) {
        if (!issue_block<CX, PASS>(base_addr, tmem, kc, KC, tile, ring, phase, full, empty, sum_full, sum_empty,
                                   abort_flag))
            return false;
        ring += pass_digits(PASS);
        if (ring >= Shape<CX>::kBuffers) {
            ring -= Shape<CX>::kBuffers;
            phase ^= 1u;
        }
    }
    return true;
}

// Fourteen warps: lane 0 of warp 0 brings the digits, warp 1 issues the MMAs (the
// whole warp, an elected lane each), warps 2..13 take the sums from TMEM (32 rows and
// a third of the columns each: 32 sums a thread in registers; with eight warps of 64
// sums the registers spilled and a sum took 64 cycles) and update C, which comes
// into shared memory ahead of time (asynchronous copies of 64-byte row pieces, two
// in flight).
// A tile's digit pairs run in three passes over K, four accumulators (sums) each; each
// accumulator goes back as soon as its warps have read it, so the MMAs of one
// pass overlap the reads of the one before, and the update of C overlaps the
// next tile.
template <bool CX>
__global__ void __launch_bounds__(32 * (2 + kEpiWarps), 1) k_digit_gemm(Args A) {
    typedef Shape<CX> S;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    if (*A.code != 0) return;
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *stage = base + (size_t)S::kBuffers * S::kBytes;  // two chunks of C for each epilogue warp
    uint64_t *full = reinterpret_cast<uint64_t *>(stage + (size_t)kEpiWarps * 2 * S::kChunkBytes);  // [kBuffers]
    uint64_t *empty = full + S::kBuffers;                                                 // [kBuffers]
    uint64_t *sum_full = empty + S::kBuffers, *sum_empty = sum_full + kSlots;             // [kSlots]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sum_empty + kSlots);
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = (A.m + kBM - 1) / kBM, tiles_n = (A.n + S::BN - 1) / S::BN, ntiles = tiles_m * tiles_n;
    const int KC = A.kc_count;
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int i = 0; i < S::kBuffers; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(&sum_full[i], 1);
            mbar_init(&sum_empty[i], kEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    volatile int *abort_flag = &s_abort;
    if (warp == 0) {
        if (lane == 0) {
            int ring = 0;
            uint32_t phase = 1;  // of the use before: the first round finds every buffer empty
            for (int t = blockIdx.x; t < ntiles && !s_abort; t += gridDim.x) {
                int tm, tn;
                tc::tile_of(t, tiles_m, tiles_n, tm, tn);
                const unsigned char *ga = A.a + (size_t)tm * KC * kDigits * S::kABytes;
                const unsigned char *gb = A.b + (size_t)tn * KC * kDigits * S::kBBytes;
#pragma unroll
                for (int pass = 0; pass < kPasses; ++pass)
                    for (int kc = 0; kc < KC && !s_abort; ++kc) {
#pragma unroll
                        for (int o = 0; o < pass_digits(pass); ++o) {
                            const int d = digit_at(pass, o) - 1;
                            if (!mbar_wait(&empty[ring], phase, abort_flag)) {
                                s_abort = 1;
                                break;
                            }
                            unsigned char *dst = base + (size_t)ring * S::kBytes;
                            mbar_expect_tx(&full[ring], S::kBytes);
                            bulk_load(dst, ga + (size_t)(kc * kDigits + d) * S::kABytes, S::kABytes, &full[ring]);
                            bulk_load(dst + S::kABytes, gb + (size_t)(kc * kDigits + d) * S::kBBytes, S::kBBytes,
                                      &full[ring]);
                            if (++ring == S::kBuffers) {
                                ring = 0;
                                phase ^= 1u;
                            }
                        }
                    }
            }
        }
    } else if (warp == 1) {
        static_assert(kPasses == 3, "passes");
        const uint32_t base_addr = smem_u32(base);
        int ring = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = blockIdx.x, tile = 0; t < ntiles && ok; t += gridDim.x, ++tile)
            ok = issue_pass<CX, 0>(base_addr, tmem, KC, tile, ring, phase, full, empty, sum_full, sum_empty, abort_flag) &&
                 issue_pass<CX, 1>(base_addr, tmem, KC, tile, ring, phase, full, empty, sum_full, sum_empty, abort_flag) &&
                 issue_pass<CX, 2>(base_addr, tmem, KC, tile, ring, phase, full, empty, sum_full, sum_empty, abort_flag);
        if (!ok) s_abort = 1;
    } else {
        const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lanes 32 q .. + 31; third of the columns
        // two runs of 16 accumulator columns: Re and Im, or consecutive ones
        constexpr int o1 = CX ? 48 : 16;
        const uint32_t tb = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(h * (CX ? 16 : 32));
        const uint32_t ts = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(kSlots * kSlotCols + h * 32);  // low words
        unsigned char *mine = stage + (size_t)(warp - 2) * 2 * S::kChunkBytes;
        typedef typename S::Scalar Scalar;
        constexpr int RPI = 32 / S::kCols, kSteps = S::kCols;  // rows per warp access, accesses per chunk
        const int rr = lane / S::kCols, cc = lane % S::kCols;
        int tile = 0;
        unsigned fp64 = 0;  // this lane's entries done in FP64
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++tile) {
            int tm, tn;
            tc::tile_of(t, tiles_m, tiles_n, tm, tn);
            const int row0 = tm * kBM + 32 * q;
            const int col0 = tn * S::BN + h * S::kWarpCols;
            // this lane's piece of row rr and column cc of each chunk
            Scalar *cp = reinterpret_cast<Scalar *>(A.c) + (size_t)(row0 + rr) * A.ldc + col0 + cc;
            const int rows = A.m - row0 - rr, cols = A.n - col0 - cc;
            auto fetch = [&](int ch) {
                unsigned char *dst = mine + (ch & 1) * S::kChunkBytes + rr * S::kRowStride + cc * (int)sizeof(Scalar);
                if (ch * S::kCols < cols) {
                    const Scalar *src = cp + ch * S::kCols;
#pragma unroll
                    for (int it = 0; it < kSteps; ++it, src += RPI * A.ldc)
                        if (it * RPI < rows) copy_async(dst + it * RPI * S::kRowStride, src);
                }
                copy_commit();
            };
            fetch(0);
            fetch(1);
            unsigned zero = 0;  // (while the first sums are formed)
            if constexpr (CX) zero = zero_parts(A, row0 + lane, col0);
            // Sums of i + j >= 10 in units of 2^-kUnit; their bits below 2^-61 go to
            // TMEM, the rest is summed in units of 2^-61 with the others.
            long long run[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) run[c] = 0;
#pragma unroll 1
            for (int g = kDigits + 1; g >= 2; --g) {
                const int pass = (kDigits + 1 - g) / kSlots, s = (kDigits + 1 - g) % kSlots;
                ok = warp_wait(&sum_full[s], (uint32_t)(kPasses * tile + pass) & 1, abort_flag);
                if (!ok) goto leave;
                fence_after_sync();
                const int shift = 7 * ((g <= 9 ? 9 : kDigits + 1) - g);  // 0 .. 49, never 31
                const int m_lo = shift < 32 ? 1 << shift : 0, m_hi = shift < 32 ? 0 : 1 << (shift - 32);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    float v[8];
                    tmem_ld8(tb + (uint32_t)(s * kSlotCols + (p >> 1) * o1 + (p & 1) * 8), v);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const int x = integer(v[c]);
                        run[8 * p + c] += (long long)x * m_lo + (long long)((unsigned long long)((unsigned)x * (unsigned)m_hi) << 32);
                    }
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sum_empty[s]);
                if (g == 10) {
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        int low[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            low[c] = (int)((unsigned)run[8 * p + c] & ((1u << (kUnit - 61)) - 1u));
                            run[8 * p + c] >>= kUnit - 61;
                        }
                        tmem_st8(ts + 8 * p, low);
                    }
                }
            }
            tmem_wait_st();
            const int er = A.ea[row0 + lane];
            const int ec = A.eb[col0 + lane % S::kWarpCols];
            // C -= sums 2^(row exponent + column exponent), a chunk at a time
            unsigned exact = 0;  // columns of this lane's row left to FP64
#pragma unroll
            for (int ch = 0; ch < S::kChunks; ++ch) {
                unsigned char *buf = mine + (ch & 1) * S::kChunkBytes;
                copy_wait1();
                __syncwarp();
                int low[8];
                tmem_ld4(ts + (CX ? ch * 4 : ch * 8), low);
                tmem_ld4(ts + (CX ? 16 + ch * 4 : ch * 8 + 4), low + 4);
                tmem_wait_ld(low, low + 4);
                Scalar *p = reinterpret_cast<Scalar *>(buf + lane * S::kRowStride);
                double w[8];            // re, im of four columns, or eight columns
                unsigned small = 0u;    // columns whose update (complex: bits 0.. real, 16.. imaginary part) is below the limit
#pragma unroll
                for (int c = 0; c < S::kCols; ++c) {
                    const int col = ch * S::kCols + c;  // 0..15 (complex), 0..31 (real)
                    const int E = er + __shfl_sync(0xffffffffu, ec, col) - 61;
                    small |= below(run[col]) ? 1u << c : 0u;
                    w[c] = __longlong_as_double(compose(run[col], (unsigned)low[c], E));
                    if constexpr (CX) {
                        small |= below(run[16 + col]) ? 0x10000u << c : 0u;
                        w[4 + c] = __longlong_as_double(compose(run[16 + col], (unsigned)low[4 + c], E));
                    }
                }
#pragma unroll
                for (int c = 0; c < S::kCols; ++c) {
                    const int col = ch * S::kCols + c;
                    const Scalar z = p[c];
                    const int E = er + __shfl_sync(0xffffffffu, ec, col);
                    if constexpr (CX) {
                        const unsigned part = small >> c & ~(zero >> col);
                        const bool left = ((part & 1u) && below(z.x, E)) || ((part >> 16 & 1u) && below(z.y, E));
                        p[c] = make_double2(z.x - (left ? 0.0 : w[c]), z.y - (left ? 0.0 : w[4 + c]));
                        exact |= left ? 1u << col : 0u;
                    } else {
                        const bool left = (small >> c & 1u) && below(z, E);
                        p[c] = z - (left ? 0.0 : w[c]);
                        exact |= left ? 1u << col : 0u;
                    }
                }
                __syncwarp();
                if (ch * S::kCols < cols) {
                    const unsigned char *src = buf + rr * S::kRowStride + cc * (int)sizeof(Scalar);
                    Scalar *dst = cp + ch * S::kCols;
#pragma unroll
                    for (int it = 0; it < kSteps; ++it, dst += RPI * A.ldc)
                        if (it * RPI < rows) *dst = *reinterpret_cast<const Scalar *>(src + it * RPI * S::kRowStride);
                }
                __syncwarp();
                if (ch + 2 < S::kChunks)
                    fetch(ch + 2);
                else
                    copy_commit();
            }
            if (row0 + lane >= A.m) exact = 0;
            exact &= col0 + S::kWarpCols <= A.n ? 0xffffffffu : A.n > col0 ? (1u << (A.n - col0)) - 1u : 0u;
            if (__any_sync(0xffffffffu, exact != 0)) {
                fp64 += __popc(exact);
                exact_entries<CX>(A, row0, col0, exact);
            }
        }
        if constexpr (CX) {
            fp64 = __reduce_add_sync(0xffffffffu, fp64);
            if (lane == 0 && fp64 != 0 && atomicAdd(A.exact, fp64) + fp64 > A.exact_limit) atomicCAS(A.code, 0, 7);
        }
    leave:
        if (!ok) s_abort = 1;
    }
    __syncwarp();
    __syncthreads();
    if (s_abort) {
        if (threadIdx.x == 0) atomicCAS(A.code, 0, 6);
        // copies and MMAs already issued finish before shared memory and TMEM go
        for (int i = 0; i < 20000; ++i) __nanosleep(1000);
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

static size_t round_up(size_t v, size_t to) { return (v + to - 1) / to * to; }

template <bool CX>
static bool run(const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc, int m, int n, int k,
                DigitScratch &s, int *code, size_t exact_limit) {
    typedef Shape<CX> S;
    const int kc = (k + kKC - 1) / kKC;
    const int mt = (m + kBM - 1) / kBM, nt = (n + S::BN - 1) / S::BN;
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_digit_gemm<CX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
    if (!cuda_ok(attr, "digit GEMM shared memory")) return false;
    PEEC_LAUNCH(k_row_exponents<CX>, k, 256, 0, (const double *)B, ldb, n, s.ef, s.exact,
                (const int *)code);
    Mask *ma = static_cast<Mask *>(s.mask), *mb = ma ? ma + round_up(s.m, kBM) : nullptr;
    auto rows = k <= 64 ? k_digits_rows<CX, 8> : k <= 128 ? k_digits_rows<CX, 16> : k_digits_rows<CX, 32>;
    PEEC_LAUNCH(rows, mt * kBM * (k <= 64 ? 8 : k <= 128 ? 16 : 32) / 256, 256, 0, (const double *)A, lda, m, k, kc,
                (unsigned char *)s.a, s.ea, ma, (const int *)s.ef, (const int *)code);
    PEEC_LAUNCH(k_digits_cols<CX>, (nt * S::BN + 63) / 64, 512, 0, (const double *)B, ldb, n, k, kc, (unsigned char *)s.b,
                s.eb, mb, (const int *)s.ef, (const int *)code);
    Args a;
    a.a = (const unsigned char *)s.a;
    a.b = (const unsigned char *)s.b;
    a.ea = s.ea;
    a.eb = s.eb;
    a.ma = ma;
    a.mb = mb;
    a.c = (double *)C;
    a.ldc = ldc;
    a.a64 = (const double *)A;
    a.b64 = (const double *)B;
    a.lda = lda;
    a.ldb = ldb;
    a.m = m;
    a.n = n;
    a.k = k;
    a.kc_count = kc;
    a.exact = s.exact;
    a.exact_limit = (unsigned)std::min(exact_limit, (size_t)UINT_MAX);
    a.code = code;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    PEEC_LAUNCH(k_digit_gemm<CX>, std::min(sms, mt * nt), 32 * (2 + kEpiWarps), S::kSmem, a);
    return launch_ok("digit GEMM");
}

}  // namespace dg

size_t digit_scratch_bytes(bool cplx, size_t m, size_t n, size_t k) {
    const size_t kp = dg::round_up(k, dg::kKC), mp = dg::round_up(m, dg::kBM), np = dg::round_up(n, 96);
    return mp * kp * dg::kDigits * 2 * (cplx ? 2 : 1) + np * kp * dg::kDigits * 2 * (cplx ? 3 : 1) + 4 * (mp + np + kp) +
           (cplx ? (mp + np) * sizeof(dg::Mask) : 0);
}

size_t &digit_scratch_limit() {
    static thread_local size_t limit = ~(size_t)0;
    return limit;
}

bool DigitScratch::alloc(bool cplx_, int m_, int n_, int k_) {
    release();
    if (digit_scratch_bytes(cplx_, m_, n_, k_) > digit_scratch_limit()) return false;
    cplx = cplx_;
    m = m_;
    n = n_;
    k = k_;
    const size_t kp = dg::round_up(k, dg::kKC), mp = dg::round_up(m, dg::kBM), np = dg::round_up(n, 96);
    a = dalloc_if_room(mp * kp * dg::kDigits * 2 * (cplx ? 2 : 1));
    b = dalloc_if_room(np * kp * dg::kDigits * 2 * (cplx ? 3 : 1));
    ea = static_cast<int *>(dalloc_if_room(4 * mp));
    eb = static_cast<int *>(dalloc_if_room(4 * np));
    ef = static_cast<int *>(dalloc_if_room(4 * kp));
    exact = static_cast<unsigned *>(dalloc_if_room(sizeof(unsigned)));
    if (cplx) mask = dalloc_if_room((mp + np) * sizeof(dg::Mask));
    if (a && b && ea && eb && ef && exact && (mask || !cplx)) return true;
    release();
    return false;
}

void DigitScratch::release() {
    dfree(a);
    dfree(b);
    dfree(ea);
    dfree(eb);
    dfree(ef);
    dfree(exact);
    dfree(mask);
    a = b = mask = nullptr;
    ea = eb = ef = nullptr;
    exact = nullptr;
    m = n = k = 0;
}

bool digit_gemm_sub(bool cplx, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc, int m, int n,
                    int k, DigitScratch &s, int *code, size_t exact_limit) {
    if (m <= 0 || n <= 0 || k <= 0) return true;
    if (s.cplx != cplx || m > s.m || n > s.n || k > s.k || k > (cplx ? kDigitMaxKCplx : kDigitMaxKReal)) {
        set_error("digit GEMM: size beyond its scratch");
        return false;
    }
    return cplx ? dg::run<true>(A, lda, B, ldb, C, ldc, m, n, k, s, code, exact_limit)
                : dg::run<false>(A, lda, B, ldb, C, ldc, m, n, k, s, code, exact_limit);
}

}  // namespace peec

extern "C" size_t peec_gb300_set_digit_scratch_limit(size_t bytes) {
    const size_t before = peec::digit_scratch_limit();
    peec::digit_scratch_limit() = bytes;
    return before;
}

extern "C" int peec_gb300_digit_gemm_sub(int cplx, const void *d_a, size_t lda, const void *d_b, size_t ldb, void *d_c,
                                         size_t ldc, int m, int n, int k) {
    using namespace peec;
    if (!d_a || !d_b || !d_c || m < 1 || n < 1 || k < 1 || lda < (size_t)k || ldb < (size_t)n || ldc < (size_t)n ||
        k > (cplx ? kDigitMaxKCplx : kDigitMaxKReal))
        return -1;
    DigitScratch s;
    DBuf<int> code(1);
    if (!s.alloc(cplx != 0, m, n, k) || !code.p) {
        set_error("digit GEMM: no memory for the digits");
        return -1;
    }
    cudaMemsetAsync(code.p, 0, sizeof(int), stream());
    if (!digit_gemm_sub(cplx != 0, d_a, lda, d_b, ldb, d_c, ldc, m, n, k, s, code.p)) return -1;
    int h = 0;
    cudaMemcpyAsync(&h, code.p, sizeof(int), cudaMemcpyDeviceToHost, stream());
    if (!sync("digit GEMM")) return -1;
    if (h != 0) {
        set_error("digit GEMM: a wait ran out");
        return -1;
    }
    return 0;
}
