// k_grm_geno.cu -- on-the-fly genotype GRM product on the FP64 pipe: the small GLOBE_PREC_FP64
// products, and all of them where the second genotype copy does not fit (geno_apply_f64 in
// k_tc_geno.cu chooses).
//
//   out (N x k) = scale * Zs' (Zs Z),  zs(s,i) = (g - 2 f_s) inv_std_s,
//   missing -> g = 0, scale = sig2g / M            (PCGsolver.cpp:1130-1201)
//
// The genotypes are read from the SNP-major tile-blocked copy of the
// tensor-core path (blk1, tile codes; the only SNP-major copy kept).
// Pass 1 (w = Zs Z): one to eight warps per two SNP rows, a lane per
// sample.  Pass 2 (Zs' w): a CTA owns 128 consecutive
// samples (one 32-byte chunk of every SNP row), stages SNP tiles in shared
// memory and splits the SNP range across CTAs (partials reduced in a fixed
// order).  zs per SNP is a table indexed by the 2-bit code, so the decode is a
// select, not arithmetic.  Latency bounds the smallest products, FP64
// throughput the largest.
#include "tc_common.cuh"

namespace globe {

__device__ __forceinline__ double zsel(unsigned code, double t0, double t1, double t2) {
    // tile code 00 -> t1 (g=0 or missing), 01 -> t2 (g=1), 10 -> t0 (g=2)
    return code == 1u ? t2 : (code == 2u ? t0 : t1);
}

// W = Zs Z: wp warps (1, 2, 4 or 8) per two SNPs, a lane per individual, so that the lanes' loads of
// Z lie side by side and each 16 of them share a word of codes (64 individuals a lane: every load of
// Z touched 32 lines).  Bound by latency at most sizes that come here, hence wp (p1_warps).
// N = 601, M = 1503: 15.1 -> 8.5 us; a call of N = 100, M = 100000: 453 -> 148 us.
template <int KC>
__global__ void __launch_bounds__(256) k_geno_p1(const uint8_t* __restrict__ blk, int nch, int64_t Mk,
                                                 int32_t N, const double* __restrict__ zs,
                                                 const double* __restrict__ Z, int64_t ldz, int kc,
                                                 double* __restrict__ W, int64_t ldw, int wp) {
    __shared__ double sm[8][2][KC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = warp & (wp - 1);
    const int64_t s = ((int64_t)blockIdx.x * (8 / wp) + warp / wp) * 2;
    const bool one = s < Mk, two = s + 1 < Mk;   // the copy's rows are padded: the second SNP's codes may be read anyway
    double t[2][3], acc[2][KC];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 3; ++q) t[u][q] = s + u < Mk ? zs[4 * (s + u) + q] : 0.0;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int c = 0; c < KC; ++c) acc[u][c] = 0.0;
    const int sh = 2 * (lane & 15);
#pragma unroll 4
    for (int i = one ? sub * 32 + lane : N; i < N; i += 32 * wp) {
        double z[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(blk + tc::blk_offset(s + u, (int64_t)(i >> 4) << 2, nch)));
            z[u] = zsel((w >> sh) & 3u, t[u][0], t[u][1], t[u][2]);
        }
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c < kc) {
                const double x = __ldg(Z + i + (size_t)c * ldz);
                acc[0][c] += z[0] * x;
                acc[1][c] += z[1] * x;
            }
    }
#pragma unroll
    for (int c = 0; c < KC; ++c) {
        double a = acc[0][c], b = acc[1][c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            sm[warp][0][c] = a;
            sm[warp][1][c] = b;
        }
    }
    __syncthreads();
    if (sub == 0 && lane < 2 * KC) {
        const int u = lane / KC, c = lane % KC;
        double a = sm[warp][u][c];
        for (int q = 1; q < wp; ++q) a += sm[warp + q][u][c];
        if (c < kc && s + u < Mk) W[s + u + (size_t)c * ldw] = a;
    }
}

// Warps per two SNPs: 16 warps an SM where the individuals give each four loads or more; fewer with
// more columns, which give a warp as many chains and whose sums over its lanes each warp pays for
// (N = 2000, M = 3000, 6 columns: 329 us a call with 2, 305 with 1; N = 20000, M = 1000, one column:
// 344 us with 1, 151 with 8).
static int p1_warps(int64_t Mk, int32_t N, int kc) {
    int wp = 1;
    while (wp < 8 && (Mk + 1) / 2 * wp * std::max(1, kc / 2) < 16 * 152 && N > 128 * wp) wp *= 2;
    return wp;
}

constexpr int P2_THREADS = 128;  // samples per CTA (32 bytes per SNP row)
constexpr int P2_TS = 64;        // SNPs per shared-memory tile

template <int KC>
__global__ void __launch_bounds__(P2_THREADS) k_geno_p2(const uint8_t* __restrict__ blk, int nch,
                                                        int64_t Mk, int32_t N, const double* __restrict__ zs,
                                                        const double* __restrict__ W, int64_t ldw, int kc,
                                                        int64_t s_per, double* __restrict__ part) {
    __shared__ __align__(16) uint8_t gb[P2_TS][32];
    __shared__ double zt[P2_TS][4];
    __shared__ double wt[P2_TS][KC];
    const int tid = threadIdx.x;
    const int64_t i = (int64_t)blockIdx.x * P2_THREADS + tid;
    const int64_t byte0 = (int64_t)blockIdx.x * 32;   // this CTA's 32-byte chunk of every row
    const int64_t s_beg = (int64_t)blockIdx.y * s_per;
    int64_t s_end = s_beg + s_per;
    if (s_end > Mk) s_end = Mk;
    double acc[KC];
#pragma unroll
    for (int c = 0; c < KC; ++c) acc[c] = 0.0;
    const int sh = 2 * (tid & 3);
    const int bi = tid >> 2;
    for (int64_t s0 = s_beg; s0 < s_end; s0 += P2_TS) {
        const int ns = (int)((s_end - s0) < P2_TS ? (s_end - s0) : P2_TS);
        {   // 64 rows x 32 bytes, 16 bytes per thread
            const int rs = tid >> 1, half = tid & 1;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (rs < ns)
                v = __ldg(reinterpret_cast<const uint4*>(blk + tc::blk_offset(s0 + rs, byte0 + half * 16, nch)));
            *reinterpret_cast<uint4*>(&gb[rs][half * 16]) = v;
        }
        for (int e = tid; e < P2_TS * 4; e += P2_THREADS) {
            const int rs = e >> 2;
            zt[rs][e & 3] = rs < ns ? zs[(s0 + rs) * 4 + (e & 3)] : 0.0;
        }
        for (int e = tid; e < P2_TS * KC; e += P2_THREADS) {
            const int rs = e / KC, c = e % KC;
            wt[rs][c] = (rs < ns && c < kc) ? W[(s0 + rs) + (size_t)c * ldw] : 0.0;
        }
        __syncthreads();
        for (int rs = 0; rs < ns; ++rs) {
            const unsigned code = (gb[rs][bi] >> sh) & 3u;
            const double z = zsel(code, zt[rs][0], zt[rs][1], zt[rs][2]);
#pragma unroll
            for (int c = 0; c < KC; ++c) acc[c] += z * wt[rs][c];
        }
        __syncthreads();
    }
    if (i < N) {
        const size_t base = (size_t)blockIdx.y * (size_t)N * kc;
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c < kc) part[base + i + (size_t)c * N] = acc[c];
    }
}

// out[e] = scale * sum_y part[y * n + e] (fixed order): 32 entries a CTA, eight threads each
__global__ void __launch_bounds__(256) k_sum_splits(const double* __restrict__ part, int nsplit, int64_t n, double scale,
                                                    double* __restrict__ out, int64_t ldo, int64_t rows) {
    __shared__ double sm[8][32];
    const int x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * 32 + x;
    double a = 0;
    if (e < n) {
#pragma unroll 4
        for (int y = y0; y < nsplit; y += 8) a += __ldg(part + (size_t)y * n + e);
    }
    sm[y0][x] = a;
    __syncthreads();
    if (y0 == 0 && e < n) {
#pragma unroll
        for (int y = 1; y < 8; ++y) a += sm[y][x];
        const int64_t r = e % rows, c = e / rows;
        out[r + c * ldo] = scale * a;
    }
}

static int pick_splits(int64_t ctas_x, int64_t Mk) {
    int64_t want = (2 * 152 + ctas_x - 1) / ctas_x;
    int64_t maxs = (Mk + P2_TS - 1) / P2_TS;
    if (want > maxs) want = maxs;
    if (want < 1) want = 1;
    if (want > 256) want = 256;
    return (int)want;
}

template <int KC>
static int geno_chunk(globe_ctx* ctx, const double* Z, int kc, double scale, double* out, double* W,
                      double* part, int nsplit, int64_t s_per) {
    auto& g = ctx->gen;
    const int32_t N = ctx->coh.N;
    {
        ProfScope ps(ctx, GLOBE_PROF_GRM_PASS1);
        const int wp = p1_warps(g.Mk, N, kc);
        k_geno_p1<KC><<<div_up(g.Mk, 16 / wp), 256, 0, ctx->stream>>>(g.blk1, g.nch1, g.Mk, N, g.zs, Z, N, kc, W, g.Mk, wp);
        GLOBE_LAUNCHED(ctx, "k_geno_p1");
    }
    dim3 grid(div_up(N, P2_THREADS), nsplit);
    {
        ProfScope ps(ctx, GLOBE_PROF_GRM_PASS2);
        k_geno_p2<KC><<<grid, P2_THREADS, 0, ctx->stream>>>(g.blk1, g.nch1, g.Mk, N, g.zs, W, g.Mk, kc, s_per, part);
        GLOBE_LAUNCHED(ctx, "k_geno_p2");
    }
    int64_t n = (int64_t)N * kc;
    k_sum_splits<<<(unsigned)div_up(n, 32), 256, 0, ctx->stream>>>(part, nsplit, n, scale, out, N, N);
    GLOBE_LAUNCHED(ctx, "k_sum_splits");
    return GLOBE_OK;
}

int geno_apply_fp64_pipe(globe_ctx* ctx, const double* Z, int k, double scale, double* out) {
    auto& g = ctx->gen;
    const int32_t N = ctx->coh.N;
    if (g.Mk == 0) {
        GLOBE_CK(ctx, cudaMemsetAsync(out, 0, sizeof(double) * (size_t)N * k, ctx->stream));
        return GLOBE_OK;
    }
    const int kcmax = 8;
    int kc0 = k < kcmax ? k : kcmax;
    double* W;
    GLOBE_RET(ws(ctx, WS_W, (size_t)g.Mk * kc0, &W));
    int64_t ctas_x = div_up(N, P2_THREADS);
    int nsplit = pick_splits(ctas_x, g.Mk);
    int64_t s_per = ((g.Mk + nsplit - 1) / nsplit + P2_TS - 1) / P2_TS * P2_TS;
    nsplit = (int)((g.Mk + s_per - 1) / s_per);
    double* part;
    GLOBE_RET(ws(ctx, WS_GPART, (size_t)nsplit * N * kc0, &part));
    for (int c0 = 0; c0 < k; c0 += kcmax) {
        int kc = (k - c0) < kcmax ? (k - c0) : kcmax;
        const double* Zc = Z + (size_t)c0 * N;
        double* oc = out + (size_t)c0 * N;
        int rc;
        if (kc == 1) rc = geno_chunk<1>(ctx, Zc, kc, scale, oc, W, part, nsplit, s_per);
        else if (kc == 2) rc = geno_chunk<2>(ctx, Zc, kc, scale, oc, W, part, nsplit, s_per);
        else if (kc <= 4) rc = geno_chunk<4>(ctx, Zc, kc, scale, oc, W, part, nsplit, s_per);
        else rc = geno_chunk<8>(ctx, Zc, kc, scale, oc, W, part, nsplit, s_per);
        GLOBE_RET(rc);
    }
    return GLOBE_OK;
}

// ---- A_ii = (1/M) sum_s zs(s,i)^2 (PCGsolver.cpp:924-989) --------------------------
//
// zs^2 takes one of three values per SNP, so four SNPs' share of an individual is one entry of a
// 256-entry table indexed by their four codes (one byte).  Entries are fixed-point int64 on one
// grid for the whole matrix, so any split of the SNPs sums to the same bits.  The grid's step is
// 2^-61 to 2^-62 of S, the sum over the SNPs of the largest zs^2 of any genotype (present or not;
// rounded up to an integer), and A_ii is within half a step, and the rounding of the zs^2, of the
// exact one.  (With the largest zs^2 of all times M in S's place one singleton among common SNPs made
// the step 2000 times wider, at N = 2000.)
// A CTA covers 16384 individuals (16 per thread: one word of each SNP row) and a range of SNPs,
// eight (two tables) a step.  A table is held 16 times over, entry e of copy l at (16 e + l): the
// 16 lanes of a half warp read 16 different bank pairs whatever their codes.  Two pair tables of
// 16 entries build it.  One barrier a step: while a step's tables are read, the next step's are
// written to the other half and the pair tables of the one after it are formed.  Bound by shared
// memory (N = 100k, M = 200k: 2.8 ms, L1 at 72 %; 8192 individuals a CTA and two barriers per four
// SNPs, where writing the tables was a third of the traffic: 3.7 ms).
constexpr int DG_THREADS = 1024;
constexpr int DG_LUT = 256 * 16 * 8;                  // bytes of a table
constexpr int DG_SMEM = 4 * DG_LUT + DG_LUT;          // two steps of two tables, aligned to a table's size

// *sum += S (integers: the same whatever the order).  zs^2 < 4 N, so S < 2^63 for 2^30 SNPs
__global__ void __launch_bounds__(256) k_zs_bound(const double* __restrict__ zs, int64_t Mk,
                                                  unsigned long long* __restrict__ sum) {
    unsigned long long m = 0;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < Mk; s += (int64_t)gridDim.x * blockDim.x) {
        const double a = zs[4 * s], b = zs[4 * s + 1], c = zs[4 * s + 2];
        m += (unsigned long long)ceil(fmax(a * a, fmax(b * b, c * c)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(sum, m);
}
// fraction bits of the fixed-point sums: S 2^bits < 2^62
__device__ __forceinline__ int diag_bits(const unsigned long long* sum) { return __clzll((long long)*sum) - 2; }

// One round of a transpose of the four 2-bit codes of each byte over four words.
template <int S>
__device__ __forceinline__ void dg_round(uint32_t (&r)[4], uint32_t m) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if ((k & S) == 0) {
            const uint32_t t = ((r[k] >> (2 * S)) ^ r[k + S]) & m;
            r[k + S] ^= t;
            r[k] ^= t << (2 * S);
        }
}

__global__ void __launch_bounds__(DG_THREADS, 1) k_geno_diag(const uint8_t* __restrict__ blk, int nch, int64_t Mk,
                                                             int32_t N, const double* __restrict__ zs,
                                                             const unsigned long long* __restrict__ bound, int64_t sper,
                                                             long long* __restrict__ part) {
    extern __shared__ __align__(16) char dg_smem[];
    __shared__ long long pt[2][4][16];   // step parity; pairs of SNPs of a step
    const int tid = threadIdx.x;
    const uint32_t lut0 = ((uint32_t)__cvta_generic_to_shared(dg_smem) + (DG_LUT - 1)) & ~(uint32_t)(DG_LUT - 1);
    const int64_t c = (int64_t)blockIdx.x * (DG_THREADS / 8) + (tid >> 3);   // 128-individual chunk
    const int w = tid & 7;                                                   // its word of 16 individuals
    const bool in = c < nch;
    const int64_t nst = (Mk + 7) / 8, st0 = (int64_t)blockIdx.y * sper, st1 = min(nst, st0 + sper);
    if (st0 >= st1) return;
    const double sc = ldexp(1.0, diag_bits(bound));
    long long acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = 0;
    // four words of a table's SNPs, loaded one table ahead of their use (a step's rows lie in one block)
    uint32_t r[4], rn[4] = {0u, 0u, 0u, 0u};
    auto fetch = [&](int64_t s0) {
        if (!in) return;
        const int rr = (int)(s0 & 127);   // a multiple of 4: the four rows share their half swap
        const uint8_t* p = blk + (((s0 >> 7) * nch + c) * 128 + rr) * 32 + (((w >> 2) ^ ((rr >> 2) & 1)) * 16) + (w & 3) * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) rn[q] = __ldg(reinterpret_cast<const uint32_t*>(p + 32 * q));
    };
    // threads 0 .. 63: entry tid & 15 of pair table tid >> 4 of step st
    const int ca = tc::tile_to_plink(tid & 3), cb = tc::tile_to_plink((tid >> 2) & 3);
    double za = 0.0, zb = 0.0;
    auto fetch_zs = [&](int64_t st) {
        if (tid >= 64) return;
        const int64_t sa = 8 * st + 2 * (tid >> 4);
        za = st < st1 && sa < Mk ? zs[4 * sa + ca] : 0.0;
        zb = st < st1 && sa + 1 < Mk ? zs[4 * sa + 4 + cb] : 0.0;
    };
    auto put_pairs = [&](int64_t st) {
        if (tid < 64) pt[st & 1][tid >> 4][tid & 15] = __double2ll_rn(za * za * sc) + __double2ll_rn(zb * zb * sc);
    };
    // thread tid writes copies 2 (tid & 7) and the next of entries tid >> 3 and 128 + (tid >> 3)
    auto put_luts = [&](int64_t st) {
        const int e = tid >> 3, el = e & 15, eh = e >> 4;
        const uint32_t base = lut0 + (uint32_t)(st & 1) * (2 * DG_LUT) + (uint32_t)(e * 128 + (tid & 7) * 16);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const long long vl = pt[st & 1][2 * t][el];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const long long v = vl + pt[st & 1][2 * t + 1][eh + 8 * q];
                asm volatile("st.shared.v2.b64 [%0], {%1, %1};" ::"r"(base + (uint32_t)(t * DG_LUT + q * (DG_LUT / 2))), "l"(v)
                             : "memory");
            }
        }
    };
    fetch(8 * st0);
    fetch_zs(st0);
    put_pairs(st0);
    fetch_zs(st0 + 1);
    __syncthreads();
    put_luts(st0);
    put_pairs(st0 + 1);
    fetch_zs(st0 + 2);
    __syncthreads();
    for (int64_t st = st0; st < st1; ++st) {
        if (st + 1 < st1) put_luts(st + 1);
        put_pairs(st + 2);   // over those of step st, read before the last barrier
        fetch_zs(st + 3);
        const uint32_t mine = lut0 + (uint32_t)(st & 1) * (2 * DG_LUT) + (uint32_t)(tid & 15) * 8;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
#pragma unroll
            for (int q = 0; q < 4; ++q) r[q] = rn[q];
            if (t == 0 || st + 1 < st1) fetch(8 * st + 4 * (t + 1));
            if (!in) continue;
            dg_round<2>(r, 0x0F0F0F0Fu);   // now byte b of r[m]: the four SNPs' codes of individual 4 b + m
            dg_round<1>(r, 0x33333333u);
            const uint32_t lut = mine + t * DG_LUT;
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t off = (b == 0 ? r[m] << 7 : r[m] >> (8 * b - 7)) & 0x7F80u;   // code x 128 bytes
                    long long v;
                    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(off | lut) : "memory");
                    acc[4 * b + m] += v;
                }
        }
        __syncthreads();
    }
    const int64_t i0 = c * 128 + w * 16;
    long long* out = part + (int64_t)blockIdx.y * N;
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (in && i0 + j < N) out[i0 + j] = acc[j];
}

__global__ void k_geno_diag_sum(const long long* __restrict__ part, int nsplit, int64_t Mk, int32_t N,
                                const unsigned long long* __restrict__ bound, double* __restrict__ d) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    long long a = 0;
    for (int y = 0; y < nsplit; ++y) a += part[(int64_t)y * N + i];
    d[i] = ldexp((double)a, -diag_bits(bound)) / (double)Mk;
}

int geno_diag(globe_ctx* ctx, double* d) {
    auto& g = ctx->gen;
    const int32_t N = ctx->coh.N;
    if (g.Mk == 0) {
        GLOBE_CK(ctx, cudaMemsetAsync(d, 0, sizeof(double) * N, ctx->stream));
        return GLOBE_OK;
    }
    // whole waves of one CTA an SM: four where that leaves a CTA 32 steps of eight SNPs (its first
    // tables and the partial sums' second pass then cost little), else as few as one; at least 4 steps
    const int64_t cx = div_up(div_up(N, 128), DG_THREADS / 8), nst = (g.Mk + 7) / 8;
    const int64_t waves = std::min<int64_t>(4, std::max<int64_t>(1, nst * cx / (32 * 152)));
    int64_t ns = std::max<int64_t>(1, std::min<int64_t>(waves * 152 / cx, nst / 4));
    const int64_t sper = (nst + ns - 1) / ns;
    ns = (nst + sper - 1) / sper;
    long long* part;
    unsigned long long* bound;
    GLOBE_RET(ws(ctx, WS_GPART, (size_t)ns * N + 1, &part));
    bound = reinterpret_cast<unsigned long long*>(part + ns * N);
    GLOBE_CK(ctx, cudaMemsetAsync(bound, 0, sizeof(*bound), ctx->stream));
    k_zs_bound<<<(unsigned)std::min<int64_t>(div_up(g.Mk, 256), 304), 256, 0, ctx->stream>>>(g.zs, g.Mk, bound);
    GLOBE_LAUNCHED(ctx, "k_zs_bound");
    GLOBE_CK(ctx, cudaFuncSetAttribute(k_geno_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_SMEM));
    k_geno_diag<<<dim3((unsigned)cx, (unsigned)ns), DG_THREADS, DG_SMEM, ctx->stream>>>(g.blk1, g.nch1, g.Mk, N, g.zs, bound,
                                                                                        sper, part);
    GLOBE_LAUNCHED(ctx, "k_geno_diag");
    k_geno_diag_sum<<<div_up(N, 256), 256, 0, ctx->stream>>>(part, (int)ns, g.Mk, N, bound, d);
    GLOBE_LAUNCHED(ctx, "k_geno_diag_sum");
    return GLOBE_OK;
}

}  // namespace globe
