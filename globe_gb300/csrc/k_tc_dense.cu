// k_tc_dense.cu -- dense GRM product on the 5th-generation tensor cores
// (GLOBE_PREC_MIXED, and GLOBE_PREC_FP64 with more digits).
//
//   out (N x k) = scale * A Z,  A(i,j) = lt[max(i,j)(max(i,j)+1)/2 + min(i,j)]
//   (PCGsolver.cpp:1202-1213, varCompEst.cpp:531-558)
//
// A is held a second time on the device as DA planes of balanced base-32 digits of
// one fixed-point grid: A(i,j) ~ 2^eA sum_d a_d(i,j) 32^-d, integer a_d in [-16,16]
// (exact in e4m3), eA fixed by max|A| (max|A| 2^-eA in [8,16)).  That is A rounded
// once to a step of 2^(eA - 5(DA-1)) <= 2^(-3 - 5(DA-1)) max|A|; with the default
// DA = 7 every entry within 2^-34 max|A|, i.e. within half a float32 ulp for every
// |A(i,j)| >= max|A| / 2^10.  DA = min(7, the context's digit count).
// The right-hand sides are split into ND digits per column exactly as in the
// genotype product.  Every MMA multiplies two digits (|a z| <= 256), so an FP32
// sum over up to 2^16 of them is an exact integer: the tensor-core accumulation
// carries no rounding; the DA x ND digit products are recombined in int64 / FP64.
//
// Layout: plane d, row i, K position P at adig[(d*NP + i) * NP + P] with
// NP = N rounded up to 128 and K permuted within groups of 16 like the digit
// tiles of the right-hand sides (k_digits), rows padded to a multiple of 256.
// The planes are full squares (both triangles), 7 N^2 bytes at DA = 7.
//
// GLOBE_PREC_FP64 takes the 12 to 14 planes that hold every entry of A exactly and 16 digits of Z,
// which hold an entry exactly or to 2^-53 of itself down to 2^-25 of the column's largest; it folds
// the exact sums in double-double with one rounding at the end.  So each row is held to FP64 by
// itself: within 2^-53 (|A| |z|)_i and the rounding, whatever the zeros of A and the magnitudes in z.
// What the digits leave of smaller entries (one normal column in 700 has one at N = 20k) is added on
// the FP64 pipe afterwards; columns with many such entries, or with a NaN or an infinity, are formed
// there, and a matrix that 14 planes do not hold stays there altogether.  N = 20k, k = 16 streams 12
// N^2 = 4.8 GB in 1.0 ms with its epilogue; 25.1 ms on the FP64 pipe, which it was bound by.  (12
// digits of Z and 12 planes whatever A: 0.93 ms, but a row that a column's largest entries do not
// enter lost up to all of its digits.)
//
// Kernel (one CTA = 2 x 128 rows x one K range, M=128 x N=NMMA MMAs per row tile):
//   warp 0     TMA of both operands per stage: two 128 x 128-byte tiles of the
//              digit planes (HBM) and the NMMA x 128-byte digit tile of Z (L2)
//   warps 1-2  one tcgen05.mma issue stream per row tile (kind::f8f6f4, E4M3 x
//              E4M3 -> F32, both operands from 128B-swizzled shared memory)
//   warp 3     TMEM allocation
//   warps 4-7  epilogue (tcgen05.ld of TMEM lane quadrant warp % 4 -> FP32 partials)
// Every mbarrier wait is bounded; on timeout the CTA records an error bit, waits
// (bounded) for its issued copies / MMAs and frees TMEM.
#include <cstring>
#include <type_traits>
#include <vector>

#include "tc_ptx.cuh"

namespace globe {
namespace tc {

constexpr int DA_MAX = 7;        // digit planes of A at most (GLOBE_PREC_MIXED)
constexpr int DA64 = 12;         // digit planes of A at least (GLOBE_PREC_FP64),
constexpr int DA64_MAX = 14;     // and at most
constexpr int DMT = 2;           // row tiles per CTA
constexpr int DROWS = DMT * BM;  // rows per CTA
constexpr int DK_MAX_CHUNKS = 512;   // K <= 2^16 per CTA: |sum| <= 256 * 2^16 = 2^24, exact in FP32

template <int NMMA>
struct DGeo {
    static constexpr int ABYTES = DMT * BM * BK;      // digit-plane bytes per stage (HBM)
    static constexpr int BBYTES = NMMA * BK;          // Z digit bytes per stage (L2)
    static constexpr int ST0 = (210 * 1024) / (ABYTES + BBYTES);
    static constexpr int STAGES = ST0 > 6 ? 6 : ST0;
    static_assert(STAGES >= 3, "stages");
};

template <int NMMA>
struct __align__(1024) DSmem {
    uint8_t a[DGeo<NMMA>::STAGES][DMT][BM * BK];   // 1024-aligned 16 KB tiles
    uint8_t b[DGeo<NMMA>::STAGES][NMMA * BK];      // NMMA * 128 B, a multiple of 2 KB
    uint64_t full[DGeo<NMMA>::STAGES], empty[DGeo<NMMA>::STAGES], accfull[DMT];
    uint32_t tmem_base;
    int abort;
};

template <int NMMA>
__global__ void __launch_bounds__(256, 1)
    k_tc_dense(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int rows,
               int nchunks, int cps, float* __restrict__ part, int64_t ldp, unsigned* __restrict__ err, int stall) {
    constexpr int ST = DGeo<NMMA>::STAGES;
    static_assert(NMMA % 16 == 0 && NMMA >= 16 && NMMA <= 256, "NMMA");
    constexpr uint32_t NCOLS = ncols_alloc(DMT * NMMA);
    extern __shared__ uint8_t smraw[];
    DSmem<NMMA>& S = *reinterpret_cast<DSmem<NMMA>*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * DROWS, split = blockIdx.y;
    const int c0 = split * cps;
    const int nloc = min(nchunks, c0 + cps) - c0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&S.full[s], 1);
            mbar_init(&S.empty[s], DMT);
        }
        for (int m = 0; m < DMT; ++m) mbar_init(&S.accfull[m], 1);
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3) tmem_alloc(&S.tmem_base, NCOLS);
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = S.tmem_base;
    int* abort = &S.abort;

    if (warp == 0) {
        if (lane == 0 && nloc > 0) {
            int issued = 0;
            for (int it = 0; it < nloc; ++it) {
                const int s = it % ST, n = it / ST;
                if (n > 0 && !mbar_wait(&S.empty[s], (n - 1) & 1, abort, err, 1u)) break;
                if (stall && it == 0) {   // test hook: the stage is never loaded, so its waits run out
                    issued = 1;
                    continue;
                }
                mbar_expect_tx(&S.full[s], DGeo<NMMA>::ABYTES + DGeo<NMMA>::BBYTES);
                const int x = (c0 + it) * BK;
                tma_load_2d(S.a[s][0], &tmA, x, row0, &S.full[s]);
                tma_load_2d(S.a[s][1], &tmA, x, row0 + BM, &S.full[s]);
                tma_load_2d(S.b[s], &tmB, x, 0, &S.full[s]);
                issued = it + 1;
            }
            for (int it = issued - 1; it >= 0 && it >= issued - ST; --it) mbar_drain(&S.full[it % ST], (it / ST) & 1);
        }
    } else if (warp == 1 || warp == 2) {
        const int m = warp - 1;
        if (lane == 0 && nloc > 0) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(NMMA >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            const uint32_t dcol = tmem + (uint32_t)(m * NMMA);
            for (int it = 0; it < nloc; ++it) {
                const int s = it % ST;
                if (!mbar_wait(&S.full[s], (it / ST) & 1, abort, err, 2u)) break;
                tc_after();
                const uint64_t ad = desc_sw128(saddr(S.a[s][m])), bd = desc_sw128(saddr(S.b[s]));
#pragma unroll
                for (int kk = 0; kk < BK / 32; ++kk)
                    mma_f8(dcol, ad + (uint64_t)(2 * kk), bd + (uint64_t)(2 * kk), idesc, (it | kk) != 0);
                mma_commit(&S.empty[s]);
            }
            mma_commit(&S.accfull[m]);   // tracks every MMA this thread issued
        }
    } else if (warp >= 4) {
        const int quad = warp & 3;   // a warp reaches TMEM lanes 32 (warp % 4) ..
        const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
#pragma unroll 1
        for (int m = 0; m < DMT; ++m) {
            bool go = nloc > 0 && mbar_wait(&S.accfull[m], 0, abort, err, 4u);
            go = __all_sync(0xffffffffu, go);   // tcgen05.ld is warp-collective
            if (!go) continue;
            tc_after();
            const int rr = row0 + m * BM + quad * 32 + lane;
#pragma unroll 1
            for (int cb = 0; cb < NMMA; cb += 16) {
                uint32_t acc[16];
                tmem_ld16(tmem + lane_addr + (uint32_t)(m * NMMA + cb), acc);
                if (rr < rows) {
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj)
                        part[((int64_t)split * NMMA + cb + jj) * ldp + rr] = __uint_as_float(acc[jj]);
                }
            }
        }
    }
    // leave: MMAs that were issued must finish before TMEM is released
    if ((warp == 1 || warp == 2) && nloc > 0) mbar_drain(&S.accfull[warp - 1], 0);
    tc_before();
    __syncthreads();
    if (warp == 3) {
        tc_after();
        tmem_dealloc(tmem, NCOLS);
    }
}

// max |A| over the packed triangle as float bits (non-negative floats order like their bits),
// whether any entry is not finite, and LSB0 + the exponent of the lowest bit that any entry holds
constexpr int LSB0 = 256;
__global__ void k_dense_scan(const float* __restrict__ lt, int64_t n, unsigned* __restrict__ out) {
    unsigned mx = 0, bad = 0, lsb = 0x7fffffffu;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = t0; e < n; e += nt) {
        const float v = lt[e];
        const unsigned b = __float_as_uint(v) & 0x7fffffffu, ex = b >> 23;
        if (!isfinite(v)) bad = 1;
        else if (b) {
            mx = max(mx, b);
            const unsigned m = ex ? (b & 0x7fffffu) | 0x800000u : b;   // v = m 2^(max(ex, 1) - 150)
            lsb = min(lsb, LSB0 + max(ex, 1u) - 150u + (unsigned)__ffs((int)m) - 1u);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        lsb = min(lsb, __shfl_xor_sync(0xffffffffu, lsb, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, mx);
        if (bad) atomicOr(out + 1, 1u);
        atomicMin(out + 2, lsb);
    }
}

// The DA digit planes of one 64 x 64 block (I0, J0) of the full square: the block is staged
// through shared memory (rows of the triangle left of the diagonal, columns of it right of
// the diagonal: coalesced either way), then each thread writes 4 words of 4 K positions per
// plane.  Position P of a group of 16 holds column 2P (P < 8) or 2(P-8)+1.  x 2^-eA is rounded once
// to I = round(x 2^-eA 32^(DA-1)); its balanced base-32 digits are peeled off from the least
// significant end (d = ((I + 16) mod 32) - 16); the leading digit is what remains, in [-16, 16].
// More than DA64 planes: those of the remainder of the first DA64, as k_digits has them.
template <int DA>
__global__ void __launch_bounds__(256) k_dense_digits(const float* __restrict__ lt, int32_t N, int eA,
                                                      uint8_t* __restrict__ D, int64_t np) {
    constexpr int DT = 64;
    __shared__ float At[DT][DT + 1];
    const int tid = threadIdx.x;
    const int64_t I0 = (int64_t)blockIdx.y * DT, J0 = (int64_t)blockIdx.x * DT;
    if (J0 + DT <= I0) {
        const int jj = tid & (DT - 1);
        for (int m = tid >> 6; m < DT; m += 4) {
            const int64_t i = I0 + m, j = J0 + jj;
            At[m][jj] = (i < N) ? lt[i * (i + 1) / 2 + j] : 0.0f;
        }
    } else if (J0 >= I0 + DT) {
        const int ii = tid & (DT - 1);
        for (int m = tid >> 6; m < DT; m += 4) {
            const int64_t i = I0 + ii, j = J0 + m;
            At[ii][m] = (i < N && j < N) ? lt[j * (j + 1) / 2 + i] : 0.0f;
        }
    } else {
        const int jj = tid & (DT - 1);
        for (int m = tid >> 6; m < DT; m += 4) {
            const int64_t i = I0 + m, j = J0 + jj;
            float v = 0.0f;
            if (i < N && j < N) v = (i >= j) ? lt[i * (i + 1) / 2 + j] : lt[j * (j + 1) / 2 + i];
            At[m][jj] = v;
        }
    }
    __syncthreads();
    constexpr int DI = DA < DA64 ? DA : DA64;
    const double sc = ldexp(1.0, DBITS * (DI - 1) - eA);   // a power of two: x * sc is exact
#pragma unroll 1
    for (int w = tid; w < DT * (DT / 4); w += 256) {
        const int m = w >> 4, pl = (w & 15) * 4;   // row in the block, first K position in the block
        long long I[4];
        int L[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int p = pl + q, base = p & ~15, pp = p & 15;
            const int jl = base + (pp < 8 ? 2 * pp : 2 * (pp - 8) + 1);
            const double x = (double)At[m][jl] * sc;
            I[q] = __double2ll_rn(x);
            if constexpr (DA > DA64) L[q] = __double2int_rn((x - (double)I[q]) * (double)(1 << (DBITS * (DA - DA64))));
        }
        uint32_t word[DA];
#pragma unroll
        for (int d = 0; d < DA; ++d) word[d] = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if constexpr (DA > DA64) {
#pragma unroll
                for (int d = DA - 1; d > DA64; --d) {
                    const int dg = ((L[q] + DHALF) & (2 * DHALF - 1)) - DHALF;
                    L[q] = (L[q] - dg) >> DBITS;
                    word[d] |= e4m3_int(dg) << (8 * q);
                }
                word[DA64] |= e4m3_int(L[q]) << (8 * q);
            }
#pragma unroll
            for (int d = DI - 1; d > 0; --d) {
                const int dg = (int)((I[q] + DHALF) & (2 * DHALF - 1)) - DHALF;
                I[q] = (I[q] - dg) >> DBITS;   // exact: I - dg is a multiple of 32
                word[d] |= e4m3_int(dg) << (8 * q);
            }
            word[0] |= e4m3_int((int)I[q]) << (8 * q);
        }
#pragma unroll
        for (int d = 0; d < DA; ++d)
            *reinterpret_cast<uint32_t*>(D + ((int64_t)d * np + I0 + m) * np + J0 + pl) = word[d];
    }
}

// out[i,c] = sA 2^e_c sum_{d,j} 32^-(d+j) P[plane d, digit j](i,c), sA = scale 2^eA.  Each
// split partial is an exact integer in FP32; they are summed in int64 by total weight
// s = d + j (T_s, |T_s| <= 12 * 256 N), and the weights folded in exact int64 chunks of
// five (C_q = sum_{s=5q}^{5q+4} 32^(5q+4-s) T_s, |C_q| < 2^31 N): a conversion and an FP64 addition
// per chunk instead of a recombination per plane.  With G = 4, four threads in warps of their own
// share an output: each sums DG planes, and the first adds the others' weights up through shared
// memory.  That shortens the chain of loads where few CTAs run (6007 x 5 in FP64: 18.9 -> 13.4
// us), and costs where many do (20k x 16 mixed: 24.6 -> 36.9 us), so it is taken up to
// DC_SPLIT_CTAS CTAs of one thread per output.
constexpr int DC_SPLIT_CTAS = 2 * 152;

// T_0 .. T_{DA + ND - 2} of output i, column c, in the first 256 / G threads; every thread calls it
template <int DA, int ND, int G>
__device__ __forceinline__ void dense_weights(const float* __restrict__ part, int nsplit, int nmma, int64_t ldp,
                                              int64_t np, int da, int64_t i, bool in, int c, long long (&T)[DA + ND - 1]) {
    constexpr int DG = (DA + G - 1) / G, NW = DG + ND - 1, DC_I = 256 / G;
    __shared__ long long sm[G > 1 ? G - 1 : 1][G > 1 ? NW : 1][DC_I];
    const int pg = threadIdx.x / DC_I, il = threadIdx.x % DC_I;
    long long w[NW];
#pragma unroll
    for (int q = 0; q < NW; ++q) w[q] = 0;
    if (in) {
#pragma unroll
        for (int d = 0; d < DG; ++d) {
            if (pg * DG + d < da) {   // the ND digit loads of split 0 issued together, further splits after
                const float* src = part + (int64_t)c * ND * ldp + (int64_t)(pg * DG + d) * np + i;
                long long pj[ND];
#pragma unroll
                for (int j = 0; j < ND; ++j) pj[j] = (long long)__float2int_rn(src[(int64_t)j * ldp]);
                for (int y = 1; y < nsplit; ++y) {
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        pj[j] += (long long)__float2int_rn(src[((int64_t)y * nmma + j) * ldp]);
                }
#pragma unroll
                for (int j = 0; j < ND; ++j) w[d + j] += pj[j];
            }
        }
    }
    if constexpr (G > 1) {
        if (pg > 0) {
#pragma unroll
            for (int q = 0; q < NW; ++q) sm[pg - 1][q][il] = w[q];
        }
        __syncthreads();
        if (pg > 0) return;
    }
#pragma unroll
    for (int q = 0; q < DA + ND - 1; ++q) T[q] = q < NW ? w[q] : 0;
#pragma unroll
    for (int g = 1; g < G; ++g)
#pragma unroll
        for (int q = 0; q < NW; ++q)
            if (g * DG + q < DA + ND - 1) T[g * DG + q] += sm[g - 1][q][il];
}

template <int ND, int G>
__global__ void __launch_bounds__(256) k_dense_combine(const float* __restrict__ part, int nsplit, int nmma, int64_t ldp,
                                                       int32_t N, int64_t np, int da, const double* __restrict__ colinfo,
                                                       double sA, double* __restrict__ out, int64_t ldo,
                                                       unsigned* __restrict__ zhi) {
    constexpr int NT = DA_MAX + ND - 1;
    static_assert(NT <= 15, "three chunks of five weights");
    const int c = blockIdx.y;
    constexpr int DC_I = 256 / G;
    const int64_t i = (int64_t)blockIdx.x * DC_I + threadIdx.x % DC_I;
    if (blockIdx.x == 0 && threadIdx.x == 0) zhi[c] = 0u;   // cleared for the next product
    long long T[NT];
    dense_weights<DA_MAX, ND, G>(part, nsplit, nmma, ldp, np, da, i, i < N, c, T);
    if (threadIdx.x >= DC_I || i >= N) return;
    const double s0 = sA * pow2i((int)colinfo[2 * c] - 20);   // 2^(e_c - 5*4) for chunk 0
    const bool bad = isnan(colinfo[2 * c + 1]);   // a non-finite column: NaN out
    long long C[3] = {0, 0, 0};
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int m = 0; m < 5; ++m) C[q] = C[q] * 32 + (5 * q + m < NT ? T[5 * q + m] : 0);
    const double v = s0 * (ll_times_pow2(C[0], 1.0) + ll_times_pow2(C[1], 0x1p-25) + ll_times_pow2(C[2], 0x1p-50));
    out[i + c * ldo] = bad ? colinfo[2 * c + 1] : v;
}

// The FP64 product's epilogue: up to DA64_MAX + NDZ - 1 = 29 weights in six exact chunks, added in
// double-double, and 2^e_c in two factors.
template <int G>
__global__ void __launch_bounds__(256) k_dense_combine64(const float* __restrict__ part, int nsplit, int nmma,
                                                         int64_t ldp, int32_t N, int64_t np, int da,
                                                         const double* __restrict__ colinfo, double sA, double scale,
                                                         double* __restrict__ out, int64_t ldo,
                                                         unsigned* __restrict__ zhi) {
    constexpr int NT = DA64_MAX + NDZ - 1;
    static_assert(NT <= 30, "six chunks of five weights");
    const int c = blockIdx.y;
    constexpr int DC_I = 256 / G;
    const int64_t i = (int64_t)blockIdx.x * DC_I + threadIdx.x % DC_I;
    if (blockIdx.x == 0 && threadIdx.x == 0) zhi[c] = 0u;
    long long T[NT];
    dense_weights<DA64_MAX, NDZ, G>(part, nsplit, nmma, ldp, np, da, i, i < N, c, T);
    if (threadIdx.x >= DC_I || i >= N) return;
    const int e = (int)colinfo[2 * c];
    const double ea = pow2i(e / 2), eb = pow2i(e - e / 2), bad = colinfo[2 * c + 1];
    double h = 0.0, l = 0.0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        long long C = 0;
#pragma unroll
        for (int m = 0; m < 5; ++m) C = C * 32 + (5 * q + m < NT ? T[5 * q + m] : 0);
        constexpr double W[6] = {1.0, 0x1p-25, 0x1p-50, 0x1p-75, 0x1p-100, 0x1p-125};
        dd_add(h, l, ll_times_pow2(C, W[q]), 0.0);
    }
    out[i + c * ldo] = (h + l) * sA * scale * ea * eb + bad;
}

}  // namespace tc

// ---- host side ---------------------------------------------------------------

using namespace tc;

// (Re)builds digit planes: set 0 for the context's digit count, set 1 for the FP64 products, which
// take the DA64 to DA64_MAX planes that hold every entry of A exactly
static int dense_digit_planes(globe_ctx* ctx, int set) {
    auto& g = ctx->gen;
    auto& a = g.adig[set];
    int da = set ? DA64 : std::min(DA_MAX, ctx->digits);
    if (a.state != 0 && (set || a.da == da)) return GLOBE_OK;
    dfree(ctx, a.p);
    a.p = nullptr;
    a.state = -1;   // until the planes are complete
    a.da = da;
    const int32_t N = ctx->coh.N;
    unsigned* mx;   // words 1-3 of the error-flag slot (word 0 is the kernels' flag): max |A| bits, non-finite, lowest bit
    GLOBE_RET(tc_err_word(ctx, &mx));
    GLOBE_CK(ctx, cudaMemsetAsync(mx + 1, 0, 2 * sizeof(unsigned), ctx->stream));
    GLOBE_CK(ctx, cudaMemsetAsync(mx + 3, 0x7f, sizeof(unsigned), ctx->stream));
    const int64_t nelt = (int64_t)N * (N + 1) / 2;
    k_dense_scan<<<(unsigned)std::min<int64_t>(div_up(nelt, 256), 152 * 8), 256, 0, ctx->stream>>>(g.grm, nelt, mx + 1);
    GLOBE_LAUNCHED(ctx, "k_dense_scan");
    unsigned h[3] = {0, 0, 0};
    GLOBE_CK(ctx, cudaMemcpyAsync(h, mx + 1, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    GLOBE_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (h[1]) return GLOBE_OK;   // a non-finite entry: the other kernels propagate it
    float amax;
    std::memcpy(&amax, &h[0], sizeof(float));
    int E = 0;
    if (amax > 0.0f) std::frexp((double)amax, &E);
    a.e = E - (DBITS - 1);   // max|A| 2^-eA in [8, 16)
    if (set && amax > 0.0f) {   // the grid's step 2^(eA - 5 (da - 1)) down to the lowest bit of any entry
        da = std::max(DA64, 1 + div_up(a.e - ((int)h[2] - LSB0), DBITS));
        if (da > DA64_MAX) return GLOBE_OK;
        a.da = da;
    }
    const int64_t np = ((int64_t)N + BM - 1) / BM * BM;
    const int64_t rows = ((int64_t)da * np + DROWS - 1) / DROWS * DROWS;
    const size_t bytes = (size_t)rows * (size_t)np;
    // the planes must fit beside what is resident, with room for a product's workspaces (set 1:
    // its split partials are 1 KB a plane row and split); otherwise the other kernels stay in use
    size_t fr = 0, tot = 0;
    GLOBE_CK(ctx, cudaMemGetInfo(&fr, &tot));
    const size_t room = ((size_t)2 << 30) + (set ? (size_t)rows * 1024 * 4 : 0);
    if (set == 0 && bytes + room > fr && g.adig[1].p) {   // the mixed planes come first
        dfree(ctx, g.adig[1].p);
        g.adig[1] = Genetic::Planes();
        GLOBE_CK(ctx, cudaMemGetInfo(&fr, &tot));
    }
    if (bytes + room > fr || rows > INT32_MAX) return GLOBE_OK;
    GLOBE_RET(dalloc(ctx, &a.p, bytes));
    if (rows > da * np)
        GLOBE_CK(ctx, cudaMemsetAsync(a.p + (size_t)da * np * np, 0, (size_t)(rows - da * np) * np, ctx->stream));
    const dim3 grid((unsigned)(np / 64), (unsigned)(np / 64));
    switch (da) {
        case 2: k_dense_digits<2><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 3: k_dense_digits<3><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 4: k_dense_digits<4><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 5: k_dense_digits<5><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 6: k_dense_digits<6><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 12: k_dense_digits<12><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 13: k_dense_digits<13><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        case 14: k_dense_digits<14><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
        default: k_dense_digits<7><<<grid, 256, 0, ctx->stream>>>(g.grm, N, a.e, a.p, np); break;
    }
    GLOBE_LAUNCHED(ctx, "k_dense_digits");
    GLOBE_CK(ctx, cudaStreamSynchronize(ctx->stream));
    a.np = np;
    a.rows = rows;
    a.state = 1;
    return GLOBE_OK;
}

template <int NMMA>
static int launch_dense(globe_ctx* ctx, const CUtensorMap& mA, const CUtensorMap& mB, int rows, int nchunks,
                        int cps, float* part, int64_t ldp, unsigned* err, int stall) {
    const size_t smem = sizeof(DSmem<NMMA>) + 1024;
    static std::atomic<uint64_t> attr_set{0};   // the shared-memory opt-in is per device
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(attr_set.load() & bit)) {
        GLOBE_CK(ctx, cudaFuncSetAttribute(k_tc_dense<NMMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set.fetch_or(bit);
    }
    const int splits = (nchunks + cps - 1) / cps;
    const dim3 grid((unsigned)(rows / DROWS), (unsigned)splits);
    k_tc_dense<NMMA><<<grid, 256, smem, ctx->stream>>>(mA, mB, rows, nchunks, cps, part, ldp, err, stall);
    ctx->tc_used = true;
    GLOBE_LAUNCHED(ctx, "k_tc_dense");
    return GLOBE_OK;
}

static int dense_dispatch(globe_ctx* ctx, int nmma, const CUtensorMap& mA, const CUtensorMap& mB, int rows,
                          int nchunks, int cps, float* part, int64_t ldp, unsigned* err, int stall) {
    switch (nmma) {
#define GLOBE_DENSE_CASE(n) \
    case n: return launch_dense<n>(ctx, mA, mB, rows, nchunks, cps, part, ldp, err, stall);
        GLOBE_DENSE_CASE(16) GLOBE_DENSE_CASE(32) GLOBE_DENSE_CASE(48) GLOBE_DENSE_CASE(64)
        GLOBE_DENSE_CASE(80) GLOBE_DENSE_CASE(96) GLOBE_DENSE_CASE(112) GLOBE_DENSE_CASE(128)
        GLOBE_DENSE_CASE(144) GLOBE_DENSE_CASE(160) GLOBE_DENSE_CASE(176) GLOBE_DENSE_CASE(192)
        GLOBE_DENSE_CASE(208) GLOBE_DENSE_CASE(224) GLOBE_DENSE_CASE(240) GLOBE_DENSE_CASE(256)
#undef GLOBE_DENSE_CASE
    }
    return set_err(ctx, GLOBE_ERR_ARG, "unsupported MMA width %d", nmma);
}

// K stages per CTA.  One CTA runs per SM; the product takes about ceil(CTAs / SMs) waves of
// (stages per CTA + a fixed cost: setup, pipeline fill, and the epilogue's partials, written
// here and read again by the combine: 8 NMMA bytes per row, in units of a 128-byte stage).
// Fewest waves-weighted stages win, within K <= 2^16 per CTA (exact FP32 sums).
static int dense_cps(globe_ctx* ctx, int tiles, int nchunks, int nmma) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device) != cudaSuccess || sms < 1) sms = 152;
    const double fixed = 4.0 + 8.0 * nmma / BK;
    const int lo = std::max(1, (nchunks + DK_MAX_CHUNKS - 1) / DK_MAX_CHUNKS);
    const int hi = std::max(lo, std::min(64, nchunks / 8));
    int best = (nchunks + lo - 1) / lo;
    double best_cost = 1e300;
    for (int s = lo; s <= hi; ++s) {
        const int cps = (nchunks + s - 1) / s;
        const int se = (nchunks + cps - 1) / cps;
        const double cost = std::ceil((double)tiles * se / sms) * (cps + fixed);
        if (cost < best_cost * 0.999) {
            best_cost = cost;
            best = cps;
        }
    }
    return best;
}

static int digit_ctas(int64_t np) { return (int)std::min<int64_t>(div_up(np / 4, 256), 1024); }

// out (N x kg) = scale * A Z for one group of <= 256 / ND columns; rest: k_digits' (NDZ)
template <int ND>
static int dense_group(globe_ctx* ctx, const double* Z, int kg, double scale, double* out, const TcStat& st, Rest* rest) {
    constexpr bool F64 = ND == NDZ;
    const auto& a = ctx->gen.adig[F64 ? 1 : 0];
    const int32_t N = ctx->coh.N;
    const int64_t np = a.np;
    const int nch = (int)(np / BK);
    const int nmma = ((kg * ND + 15) / 16) * 16;
    const int rows = (int)a.rows, tiles = rows / DROWS;
    const int cps = dense_cps(ctx, tiles, nch, nmma);
    const int splits = (nch + cps - 1) / cps;
    const int64_t ldp = rows;
    uint8_t* D;
    float* P;
    double* col;
    unsigned* err;
    GLOBE_RET(ws(ctx, WS_TC_D1, (size_t)nmma * np, &D));
    GLOBE_RET(ws(ctx, WS_TC_P1, (size_t)splits * nmma * ldp, &P));
    GLOBE_RET(ws(ctx, WS_TC_SCAL, (size_t)2 * kg, &col));
    GLOBE_RET(tc_err_word(ctx, &err));
    CUtensorMap mA, mB;
    GLOBE_RET(make_map(ctx, &mA, a.p, (uint64_t)np, (uint64_t)rows, BK, BM, true));
    GLOBE_RET(make_map(ctx, &mB, D, (uint64_t)np, (uint64_t)nmma, BK, (uint32_t)nmma, true));
    k_digits<ND, false><<<dim3((unsigned)digit_ctas(np), kg), 256, 0, ctx->stream>>>(
        Z, N, N, st.zhi, col, D, np, nullptr, nullptr, nmma - kg * ND, rest);
    GLOBE_LAUNCHED(ctx, "k_digits");
    {
        ProfScope p(ctx, GLOBE_PROF_GRM_PASS1);
        const int stall = ctx->stall_next_gemm;   // test hook (globe_debug_stall_next_gemm)
        ctx->stall_next_gemm = 0;
        GLOBE_RET(dense_dispatch(ctx, nmma, mA, mB, rows, nch, cps, P, ldp, err, stall));
    }
    const auto combine = [&](auto split) {
        constexpr int G = decltype(split)::value;
        const dim3 gc((unsigned)div_up(N, 256 / G), kg);
        if constexpr (F64)
            k_dense_combine64<G><<<gc, 256, 0, ctx->stream>>>(P, splits, nmma, ldp, N, np, a.da, col,
                                                              std::ldexp(1.0, a.e - 20), scale, out, N, st.zhi);
        else
            k_dense_combine<ND, G><<<gc, 256, 0, ctx->stream>>>(P, splits, nmma, ldp, N, np, a.da, col,
                                                                std::ldexp(scale, a.e), out, N, st.zhi);
    };
    if (div_up(N, 256) * kg <= DC_SPLIT_CTAS) combine(std::integral_constant<int, 4>());
    else combine(std::integral_constant<int, 1>());
    GLOBE_LAUNCHED(ctx, "k_dense_combine");
    return GLOBE_OK;
}

static int dense_group_nd(globe_ctx* ctx, int nd, const double* Z, int kg, double scale, double* out, const TcStat& st,
                          Rest* rest) {
    switch (nd) {
        case 2: return dense_group<2>(ctx, Z, kg, scale, out, st, rest);
        case 3: return dense_group<3>(ctx, Z, kg, scale, out, st, rest);
        case 4: return dense_group<4>(ctx, Z, kg, scale, out, st, rest);
        case 5: return dense_group<5>(ctx, Z, kg, scale, out, st, rest);
        case 6: return dense_group<6>(ctx, Z, kg, scale, out, st, rest);
        case 7: return dense_group<7>(ctx, Z, kg, scale, out, st, rest);
        case 8: return dense_group<8>(ctx, Z, kg, scale, out, st, rest);
        case 9: return dense_group<9>(ctx, Z, kg, scale, out, st, rest);
        case NDZ: return dense_group<NDZ>(ctx, Z, kg, scale, out, st, rest);
    }
    return set_err(ctx, GLOBE_ERR_ARG, "unsupported digit count %d", nd);
}

// out (N x k) = scale * A Z from the planes, nd digits per column
static int dense_apply_nd(globe_ctx* ctx, int nd, const double* Z, int k, double scale, double* out, bool zhi_ready) {
    PinScope pin(ctx, nd == NDZ ? PIN_TC | PIN_PLANES64 : PIN_TC);
    const int nw = digit_ctas(ctx->gen.adig[nd == NDZ ? 1 : 0].np);
    Rest* rest = nullptr;
    if (nd == NDZ) GLOBE_RET(ws(ctx, WS_TC_U, (size_t)k * nw, &rest));
    TcStat st;
    GLOBE_RET(tc_stat_fill(ctx, Z, ctx->coh.N, k, &zhi_ready, &st));
    const int gmax = 256 / nd;   // MMA width <= 256; near-equal groups
    const int ng = (k + gmax - 1) / gmax;
    for (int gi = 0, c0 = 0; gi < ng; ++gi) {
        const int kg = k / ng + (gi < k % ng ? 1 : 0);
        GLOBE_RET(dense_group_nd(ctx, nd, Z + (size_t)c0 * ctx->coh.N, kg, scale, out + (size_t)c0 * ctx->coh.N,
                                 st.from(c0), rest ? rest + (size_t)c0 * nw : nullptr));
        c0 += kg;
    }
    ctx->stat_dirty = false;
    return rest ? dense_rest_fp64_pipe(ctx, Z, k, scale, out, rest, nw) : GLOBE_OK;
}

int dense_apply_tc(globe_ctx* ctx, const double* Z, int k, double scale, double* out, bool zhi_ready) {
    GLOBE_RET(dense_digit_planes(ctx, 0));
    if (ctx->gen.adig[0].state != 1) return dense_apply_df(ctx, Z, k, scale, out);
    return dense_apply_nd(ctx, ctx->digits, Z, k, scale, out, zhi_ready);
}

// The FP64 product, by its size N N k (FP64 pipe / planes, us a product):
//  - inside a solve, which repeats the product and so pays for building the planes (0.2 ms at
//    N = 200, 4.4 ms at 20k), the planes from 1e5 on (2e5: 64 / 36; 1.6e7: 471 / 44;
//    6.4e9: 25118 / 1010);
//  - a single operator call from 4e6 on, where the first call, with the planes to build, costs
//    about the same on either (1e6: 191 / 288; 4e6: 352 / 314; 4e8: 8484 / 5179).
// The choice depends on the sizes only; the FP64 pipe also runs where the planes cannot be held or
// do not hold A exactly, and for single columns (top of the file).
// Error against 128-bit sums (N = 2500; normal, constant, count, lognormal and unit columns): at most
// 1.0e-16 of the column and of (|A| |z|)_i row by row; FP64 pipe (and a column over 12 decades, which
// it forms) up to 2.4e-15.
#ifndef F64_DENSE_SOLVE_MIN
#define F64_DENSE_SOLVE_MIN 1e5
#endif
#ifndef F64_DENSE_CALL_MIN
#define F64_DENSE_CALL_MIN 4e6
#endif
static bool f64_dense_size(const globe_ctx* ctx, int k) {
    return (double)ctx->coh.N * ctx->coh.N * k >= (ctx->in_solve ? F64_DENSE_SOLVE_MIN : F64_DENSE_CALL_MIN);
}
bool dense_f64_tc(const globe_ctx* ctx, int k) { return ctx->gen.adig[1].state == 1 && f64_dense_size(ctx, k); }

int dense_apply_f64(globe_ctx* ctx, const double* Z, int k, double scale, double* out, bool zhi_ready) {
    auto& a = ctx->gen.adig[1];
    const size_t len = (size_t)ctx->coh.N * k;
    if (Z < out + len && out < Z + len) {   // every column is read again after out is written
        double* zc;
        GLOBE_RET(ws(ctx, WS_W, len, &zc));
        GLOBE_CK(ctx, cudaMemcpyAsync(zc, Z, sizeof(double) * len, cudaMemcpyDeviceToDevice, ctx->stream));
        Z = zc;
    }
    if (a.state >= 0 && f64_dense_size(ctx, k)) {
        int rc = dense_digit_planes(ctx, 1);
        if (rc == GLOBE_OK && a.state == 1) rc = dense_apply_nd(ctx, NDZ, Z, k, scale, out, zhi_ready);
        if (a.state == 1 && rc != GLOBE_ERR_NOMEM) return rc;
        if (rc != GLOBE_OK && rc != GLOBE_ERR_NOMEM) return rc;
        if (rc == GLOBE_ERR_NOMEM) {
            release_optional(ctx);
            a.state = -1;
        }
    }
    return dense_apply_fp64_pipe(ctx, Z, k, scale, out);
}

}  // namespace globe
