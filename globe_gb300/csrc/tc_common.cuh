// tc_common.cuh -- what the tensor-core genotype kernels share: the tile and
// digit constants, the K permutation of the decoded operand, the e4m3 digit
// encoding, the exact recombination of split partials, and the host launch
// of k_tc_gemm (defined in k_tc_geno.cu).
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "internal.cuh"

namespace globe {
namespace tc {

constexpr int BM = 128;           // rows per MMA tile (TMEM lanes)
constexpr int BK = 128;           // K elements per stage (one 128-byte swizzle panel of e4m3)
constexpr int PKB = BK / 4;       // packed bytes per row per stage
constexpr int DBITS = 5;          // digit base 32
constexpr int DHALF = 1 << (DBITS - 1);   // 16: digits in [-16, 16]
constexpr int NDIG = 9;           // digits per right-hand-side column by default (45 bits)
constexpr int MIN_DIG = 2;        // fewest digits a context may ask for (globe_set_digits)
constexpr int ND64 = 12;          // digits per column of the GLOBE_PREC_FP64 products (59 bits: |I| < 2^59)
constexpr int NDZ = 16;           // ... of the dense ones: 12 and 4 more, which hold what those leave

// The tile-blocked genotype copies hold "tile codes", 2 bits per genotype like the PLINK
// codes they are made from (re-encoded once, by recode_tile), equal to the genotype:
//   00 = genotype 0 or missing, 01 = genotype 1, 10 = genotype 2 (11 is not produced).
// A field masked in place is then an e4m3 byte proportional to its genotype: at bit offset 0
// of a byte 0x00 / 0x01 / 0x02 = 0, 2^-9, 2^-8 (subnormals); at offset 2 0x00 / 0x04 / 0x08 =
// 0, 2^-7, 2^-6.  So the decode is four masks and one shift (decode_word in k_tc_geno.cu).
__host__ __device__ __forceinline__ uint32_t recode_tile(uint32_t w) {
    const uint32_t lo = w & 0x55555555u, hi = (w >> 1) & 0x55555555u;   // PLINK bit 0 / bit 1 of each code
    // PLINK 00 (g=2) -> 10, 10 (g=1) -> 01, 11 (g=0) and 01 (missing) -> 00
    return ((~hi & ~lo & 0x55555555u) << 1) | (hi & ~lo);
}
// the PLINK code each tile code stands for (missing and genotype 0 share tile code 00)
__host__ __device__ constexpr int tile_to_plink(int t) { return t == 1 ? 2 : (t == 2 ? 0 : 3); }

// (sh, sl) += (h, l) in double-float: Knuth's two-sum of the high parts, the rounding error and
// the low parts into sl (GB300's FP32 pipe is many times its FP64 pipe)
__device__ __forceinline__ void df_add(float& sh, float& sl, float h, float l) {
    const float s = __fadd_rn(sh, h);
    const float bp = __fsub_rn(s, sh);
    const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bp)), __fsub_rn(h, bp));
    sl = __fadd_rn(sl, __fadd_rn(err, l));
    sh = s;
}

// Byte b of row `row` in a tile-blocked copy with nch 32-byte chunks per row: block (row / 128,
// b / 32) of 128 rows x 32 bytes, the two 16-byte halves of a row swapped when bit 2 of the row
// (within its tile) is set.
__host__ __device__ __forceinline__ int64_t blk_offset(int64_t row, int64_t b, int nch) {
    const int64_t t = row >> 7;
    const int r = (int)(row & 127);
    const int w = (int)(b & 31);
    const int h = (w >> 4) ^ ((r >> 2) & 1);
    return (((t * nch + (b >> 5)) * 128 + r) * 32) + h * 16 + (w & 15);
}

// K position of genotype i of a 16-genotype word after decode_word (k_tc_geno.cu): word r holds
// the genotypes at field r of the word's four bytes, so position 4 (i % 4) + i / 4.  Its own
// inverse.  Even genotypes (fields 0 and 2) decode to 2^-9 g, odd ones to 2^-7 g, so the digit
// operand of the genotype products carries 4 d at even genotypes (geno_digit_mult): every
// product is then g d 2^-7.
__host__ __device__ __forceinline__ int kpos_g(int64_t i) {
    const int q = (int)(i & 15);
    return (int)(i & ~15ll) + 4 * (q & 3) + (q >> 2);
}
__host__ __device__ constexpr int geno_digit_mult(int64_t i) { return (i & 1) ? 1 : 4; }
constexpr float GENO_UNIT_INV = 128.0f;   // genotype-product partials are multiples of 2^-7

__device__ __forceinline__ uint32_t e4m3_int(int d) {   // d in [-16, 16], or 4x that: exact in e4m3
    return (uint32_t)__nv_cvt_float_to_fp8((float)d, __NV_SATFINITE, __NV_E4M3);
}

// Exact int64 -> FP64 conversion scaled by a power of two, from the bits: GB300's FP64 pipe,
// which also runs its int64 -> FP64 conversion instruction, is small, and the recombinations
// convert two or three integers per value.  It gives the bits of the FP64 route it replaces.
// (The digit kernels' FP64 -> int64 rounding stays on the conversion instruction: an integer
// form of it measured slower there.)

// v s for |v| < 2^53 and s a power of two: (double)v * s, built from the bits when the result
// is a normal double (both the conversion and the product are exact then), else computed so
__device__ __forceinline__ double ll_times_pow2(long long v, double s) {
    if (v == 0) return 0.0;
    const int es = (int)((__double_as_longlong(s) >> 52) & 0x7ff);
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    const int msb = 63 - __clzll((long long)a);
    const int ex = es + msb;   // biased exponent of v s
    if (es == 0 || msb > 52 || ex <= 0 || ex >= 2047) return (double)v * s;
    const unsigned long long mant = (a << (52 - msb)) & 0xfffffffffffffull;
    return __longlong_as_double((long long)((v < 0 ? 0x8000000000000000ull : 0ull) | ((unsigned long long)ex << 52) |
                                            mant));
}

// 2^e, from its bits where it is a normal double (ldexp runs on the FP64 pipe)
__device__ __forceinline__ double pow2i(int e) {
    return (e >= -1022 && e <= 1023) ? __longlong_as_double((long long)(e + 1023) << 52) : ldexp(1.0, e);
}

// 2^e sum_j 32^-j P_j of one row of a genotype product, ND digits per column (rows c*ND + j
// of the partials).  Every FP32 partial is an exact multiple of 2^-7 (|P| < 2^17), so it is
// scaled to an integer, the split partials are summed in int64 and the digits combined in two
// exact int64 halves (hi = digits 0..ND_HI-1, lo = the rest); the only rounding is the final
// FP64 addition.
// With YU > 1, YU splits' ND loads issue together: the kernels wait on them.  Up to 2 splits (the
// large shapes' pass 1) run faster one at a time, from fewer registers.
template <int ND, int YU = 1>
__device__ __forceinline__ void recombine_int(const float* __restrict__ part, int nsplit, int nmma, int64_t ldp, int c,
                                              int64_t row, long long& hi, long long& lo) {
    constexpr int NH = (ND + 1) / 2;
    long long pj[ND];
    if constexpr (YU == 1) {
#pragma unroll
        for (int j = 0; j < ND; ++j)
            pj[j] = (long long)__float2int_rn(part[((int64_t)c * ND + j) * ldp + row] * GENO_UNIT_INV);
        for (int y = 1; y < nsplit; ++y) {
#pragma unroll
            for (int j = 0; j < ND; ++j)
                pj[j] += (long long)__float2int_rn(part[((int64_t)y * nmma + c * ND + j) * ldp + row] * GENO_UNIT_INV);
        }
    } else {
#pragma unroll
        for (int j = 0; j < ND; ++j) pj[j] = 0;
        for (int y0 = 0; y0 < nsplit; y0 += YU) {
            float v[YU][ND];
#pragma unroll
            for (int u = 0; u < YU; ++u)
                if (y0 + u < nsplit) {
#pragma unroll
                    for (int j = 0; j < ND; ++j) v[u][j] = part[((int64_t)(y0 + u) * nmma + c * ND + j) * ldp + row];
                }
#pragma unroll
            for (int u = 0; u < YU; ++u)
                if (y0 + u < nsplit) {
#pragma unroll
                    for (int j = 0; j < ND; ++j) pj[j] += (long long)__float2int_rn(v[u][j] * GENO_UNIT_INV);
                }
        }
    }
    hi = lo = 0;
#pragma unroll
    for (int j = 0; j < NH; ++j) hi = hi * (1 << DBITS) + pj[j];
#pragma unroll
    for (int j = NH; j < ND; ++j) lo = lo * (1 << DBITS) + pj[j];
}
template <int ND, int YU = 1>
__device__ __forceinline__ double recombine(const float* __restrict__ part, int nsplit, int nmma, int64_t ldp, int c,
                                           int64_t row, double s_hi, double s_lo) {
    long long hi, lo;
    recombine_int<ND, YU>(part, nsplit, nmma, ldp, c, row, hi, lo);
    return ll_times_pow2(hi, s_hi) + ll_times_pow2(lo, s_lo);
}

// scale factors of recombine<ND> for exponent e: 2^(e - 5 (ND_HI - 1)) and 2^(e - 5 (ND - 1))
template <int ND>
__device__ __forceinline__ void recombine_scales(int e, double& s_hi, double& s_lo) {
    s_hi = pow2i(e - DBITS * ((ND + 1) / 2 - 1));
    s_lo = pow2i(e - DBITS * (ND - 1));
}

// ---- column statistics of a product's inputs ----------------------------------
//
// A column x is scaled by the power of two 2^-e with |x 2^-e| < 16.  All that e needs is the
// largest high word of |x| (sign dropped): its exponent field, or 0x7ff where a NaN or an
// infinity occurs, which marks the column as bad.  One 32-bit word per column, raised by
// integer maxima (GB300's FP64 pipe does two operations a clock and SM, so the FP64 maxima and
// sums of every element that stood here cost more than the data's reads): zeroed between
// products, filled by k_col_max or by the kernel that writes the column.
__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ bool col_bad(unsigned hi) { return hi >= 0x7ff00000u; }
// the exponent e; a zero or subnormal column takes the smallest (ND64, whose 59 bits then reach
// below the last bit of a double), or the smallest whose scale 2^(5 (ND - 1) - e) is finite
template <int ND>
__device__ __forceinline__ int col_exp(unsigned hi) {
    const int e = (int)(hi >> 20) - 1022 - (DBITS - 1);
    return col_bad(hi) ? 0 : (ND == ND64 ? e : max(e, -983));
}

// CTAs per column of k_col_max: ~8 values per thread
__host__ __forceinline__ int col_parts(int64_t n) {
    const int64_t p = (n + 2047) / 2048;
    return (int)(p < 1 ? 1 : (p > 304 ? 304 : p));
}
// CTAs per column of a combine kernel: a row per thread up to 32768 rows (a chain of four costs a
// small product more than the extra sums do), then ~4; at most 2 per SM.  It depends on the rows
// only, so a column's sums have one order whatever its group.
constexpr int COMBINE_PARTS = 304;
__host__ __forceinline__ int combine_parts(int64_t n) {
    const int64_t p = n <= 32768 ? (n + 255) / 256 : std::max<int64_t>(128, (n + 1023) / 1024);
    return (int)(p < 1 ? 1 : (p > COMBINE_PARTS ? COMBINE_PARTS : p));
}

// sum of v over a CTA of 256 threads, in one order (sm: 256 doubles), valid in thread 0: halves
// through shared memory, since an FP64 addition costs the same for one lane as for 32
__device__ __forceinline__ double cta_sum_256(double v, double* sm) {
    const int t = threadIdx.x;
    sm[t] = v;
    __syncthreads();
#pragma unroll
    for (int s = 128; s >= 32; s >>= 1) {
        if (t < s) {
            v += sm[t + s];
            sm[t] = v;
        }
        __syncthreads();
    }
    if (t < 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}
// max of m over the CTA, raised in *out
__device__ __forceinline__ void cta_raise(unsigned m, unsigned* out) {
    __shared__ unsigned sm[32];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0u;
        m = __reduce_max_sync(0xffffffffu, m);
        if (threadIdx.x == 0 && m) atomicMax(out, m);
    }
}

// (h, l) += (a, b): two-sum of the high parts, everything else into l
__device__ __forceinline__ void dd_add(double& h, double& l, double a, double b) {
    const double s = __dadd_rn(h, a), bp = __dsub_rn(s, h);
    l = __dadd_rn(l, __dadd_rn(b, __dadd_rn(__dsub_rn(h, __dsub_rn(s, bp)), __dsub_rn(a, bp))));
    h = s;
}

// hi[c] raised to the largest abs_hi of column c (n rows)
__global__ void k_col_max(const double* __restrict__ X, int64_t n, int64_t ld, unsigned* __restrict__ hi);

// ND digits of X (n x k, FP64) into D[(c*ND + j) * kpad + pos(r)]  (e4m3); every position
// in [0, kpad) of the column's digit rows is written (rows >= n give digit 0).  One thread
// fills 4 consecutive positions P..P+3 (a 32-bit word).  GENO: the operand of a genotype
// product -- pos = kpos_g (position P + q of a group of 16 holds row 4 q + P/4) and digits
// times geno_digit_mult(row); otherwise the order of the dense product's planes, evens before odds
// in each group of 16 (position P < 8 holds row 2P, P >= 8 row 2(P-8)+1).
// x 2^-e is rounded once to the integer I = round(x 2^-e 32^(ND-1)), |I| <= 2^(5 ND - 1); its
// balanced base-32 digits are peeled off from the least significant end in integer
// arithmetic (d = ((I + 16) mod 32) - 16, in [-16, 15]); the leading digit is what
// remains, in [-16, 16].  sum_j d_j 32^-j equals x 2^-e rounded to 5 (ND-1) fraction bits.
// The scale comes from the column's high word hi[c]; CTA 0 of each column leaves {e, 0 or NaN} in
// colinfo for the epilogues.  With isum the column sum of x, each x rounded to ND64 digits whatever
// ND, is added to isum[2c] 2^30 + isum[2c+1] in units of 2^(e - 55) (integer atomics: the same
// bits in any order); clear[2c], clear[2c+1] are set to zero
// (an isum no longer in use).  The npad digit rows after the last column's are set to zero (the MMA
// width is a multiple of 16; a memset of them cost a launch of its own).  With ND64 digits and more
// (the FP64 products) the scaling takes two factors where one would leave the range of a double.
// NDZ digits: the first ND64 as above, then those of the remainder x 2^-e 32^(ND64-1) - I, which is
// exact in a double and at most 1/2.  An entry more than 2^25 below the column's largest may have bits
// below the last digit still: what the digits leave of such entries goes to rest[c gridDim.x + CTA], by
// rising row; their number is left_any where they do not fit or cannot be told (a bad column, an
// entry that the scaling takes to zero).
constexpr int REST_MAX = 8;       // entries of a Rest
constexpr int left_any = REST_MAX + 1;
struct Rest {
    double v[REST_MAX];           // z = (its digits) + v
    int row[REST_MAX];
    int n, pad;
};
template <int ND, bool GENO>
__global__ void k_digits(const double* __restrict__ X, int64_t n, int64_t ld, const unsigned* __restrict__ hi,
                         double* __restrict__ colinfo, uint8_t* __restrict__ D, int64_t kpad,
                         unsigned long long* __restrict__ isum, unsigned long long* __restrict__ clear, int npad,
                         Rest* __restrict__ rest = nullptr) {
    constexpr int NI = ND < ND64 ? ND : ND64;   // digits of I
    const int c = blockIdx.y;
    const unsigned h = hi[c];
    const int pad = c == (int)gridDim.y - 1 ? npad : 0;
    const int e = col_exp<NI>(h), sh = DBITS * (NI - 1) - e;
    const double sc = pow2i(NI == ND64 ? min(sh, 1000) : sh);   // a power of two: x * sc is exact
    const double sc2 = NI == ND64 ? pow2i(sh - min(sh, 1000)) : 1.0;
    const bool bad = col_bad(h);   // non-finite column: zero digits
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        colinfo[2 * c] = (double)e;
        colinfo[2 * c + 1] = bad ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
        if (clear) clear[2 * c] = clear[2 * c + 1] = 0ull;
    }
    const int64_t nw = kpad >> 2;
    long long sum_hi = 0, sum_lo = 0;
    __shared__ int nrest;
    Rest* left = nullptr;
    if constexpr (ND > ND64) {
        left = rest + (size_t)c * gridDim.x + blockIdx.x;
        if (threadIdx.x == 0) nrest = bad ? left_any : 0;
        __syncthreads();
    }
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (int64_t)gridDim.x * blockDim.x) {
        const int64_t P = w << 2, base = P & ~(int64_t)15;
        const int pl = (int)(P & 15);
        const int mult = GENO ? geno_digit_mult(pl >> 2) : 1;   // GENO: rows 4 q + pl/4 share its parity
        long long I[4];
        int L[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int pq = pl + q;
            const int64_t src = base + (GENO ? 4 * q + (pl >> 2) : (pq < 8 ? 2 * pq : 2 * (pq - 8) + 1));
            const double raw = (src < n && !bad) ? X[src + c * ld] : 0.0;
            double x = raw * sc;
            if (NI == ND64) x *= sc2;
            I[q] = __double2ll_rn(x);
            if constexpr (ND > ND64) {
                const double r = (x - (double)I[q]) * (double)(1 << (DBITS * (ND - ND64)));
                L[q] = __double2int_rn(r);
                const double d = r - (double)L[q];   // exact
                if (x == 0.0 && raw != 0.0) atomicAdd(&nrest, left_any);
                else if (d != 0.0) {
                    const int at = atomicAdd(&nrest, 1);
                    if (at < REST_MAX) {
                        left->v[at] = ldexp(d, e - DBITS * (ND - 1));
                        left->row[at] = (int)src;
                    }
                }
            }
            if (isum) {
                const long long J = NI == ND64 ? I[q] : __double2ll_rn(x * pow2i(DBITS * (ND64 - ND)));
                sum_hi += J >> 30;
                sum_lo += J & ((1ll << 30) - 1);
            }
        }
        uint32_t word[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j) word[j] = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if constexpr (ND > ND64) {
#pragma unroll
                for (int j = ND - 1; j > ND64; --j) {
                    const int d = ((L[q] + DHALF) & (2 * DHALF - 1)) - DHALF;
                    L[q] = (L[q] - d) >> DBITS;
                    word[j] |= e4m3_int(mult * d) << (8 * q);
                }
                word[ND64] |= e4m3_int(mult * L[q]) << (8 * q);   // |L| <= 2^(5 (ND - ND64) - 1): in [-16, 16]
            }
#pragma unroll
            for (int j = NI - 1; j > 0; --j) {
                const int d = (int)((I[q] + DHALF) & (2 * DHALF - 1)) - DHALF;
                I[q] = (I[q] - d) >> DBITS;   // exact: I - d is a multiple of 32
                word[j] |= e4m3_int(mult * d) << (8 * q);
            }
            word[0] |= e4m3_int(mult * (int)I[q]) << (8 * q);
        }
#pragma unroll
        for (int j = 0; j < ND; ++j) *reinterpret_cast<uint32_t*>(D + ((int64_t)c * ND + j) * kpad + P) = word[j];
        for (int j = ND; j < ND + pad; ++j) *reinterpret_cast<uint32_t*>(D + ((int64_t)c * ND + j) * kpad + P) = 0u;
    }
    if (isum) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, o);
            sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(isum + 2 * c, (unsigned long long)sum_hi);
            atomicAdd(isum + 2 * c + 1, (unsigned long long)sum_lo);
        }
    }
    if constexpr (ND > ND64) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int m = min(nrest, left_any);
            left->n = m;
            for (int a = 1; a < m && m <= REST_MAX; ++a)   // into one order, whatever the threads' was
                for (int b = a; b > 0 && left->row[b - 1] > left->row[b]; --b) {
                    const int t = left->row[b];
                    left->row[b] = left->row[b - 1];
                    left->row[b - 1] = t;
                    const double v = left->v[b];
                    left->v[b] = left->v[b - 1];
                    left->v[b - 1] = v;
                }
        }
    }
}

}  // namespace tc

// Extra launch dimension of k_tc_gemm: gridDim.z = nz independent digit
// operands stacked in one tensor map (operand z = map rows z*NMMA ..), partials
// of operand z at part + z * pz.  A CTA whose rows all lie below
// skip0 + z * skipz does nothing (the lower-triangle GRM build uses this).
struct ZGrid {
    int nz = 1;
    int64_t pz = 0;
    int skip0 = 0, skipz = 0;
    int stall = 0;   // test hook (globe_debug_stall_next_gemm): leave the first digit stage unloaded
};

// Words of the columns' statistics (tc_common.cuh's top): zhi and uhi, the high words of Z's and
// u's columns, and isum, the sums of Z's.  Zero between products.
struct TcStat {
    unsigned long long* isum = nullptr;
    unsigned *zhi = nullptr, *uhi = nullptr;
    TcStat from(int c) const { return TcStat{isum + 2 * (size_t)c, zhi + c, uhi + c}; }
};
int tc_stat(globe_ctx* ctx, int k, TcStat* st);
// the words of Z's k columns (n rows), zhi filled unless *ready (then *ready is reset: the product
// that follows consumes it)
int tc_stat_fill(globe_ctx* ctx, const double* Z, int64_t n, int k, bool* ready, TcStat* st);

int make_map(globe_ctx* ctx, CUtensorMap* m, const void* base, uint64_t inner, uint64_t outer, uint32_t box_in,
             uint32_t box_out, bool sw128);
// Tile-blocked genotype copies hold a multiple of TILE_PAD row tiles of 128, so that CTAs of
// 1, 2, 3 or 4 tiles never run past them; gemm_dispatch checks it for each launch (ntiles:
// the row tiles of blk).
constexpr int TILE_PAD = 12;
int gemm_dispatch(globe_ctx* ctx, int nmma, const uint8_t* blk, int ntiles, const CUtensorMap& mB, int rows, int nchunks,
                  int splits, float* part, int64_t ldp, unsigned* err, const ZGrid& zg);
int rows_per_cta(int nmma);
int eff_splits(int nchunks, int splits);

}  // namespace globe
