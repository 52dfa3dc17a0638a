// k_bed.cu -- PLINK 2-bit genotype statistics, filtering and layout.
//
// Per-SNP counts follow prepGenotypeInput (PCGsolver.cpp:700-743): A1 count
// = 2 #00 + #10 and missing = #01 over the N real samples (the phantom pairs
// of the last byte are excluded, which is what subtractPhantomGenotypes,
// PCGsolver.cpp:589-613, achieves by subtraction).  The float32 frequency,
// missing rate and filter use the same float operations as the reference, so
// the results are bit-exact.  The FP64 standardisation coefficients are the
// float->double restatement of getStdGenotype (PCGsolver.cpp:826-842).
#include <algorithm>

#include "tc_common.cuh"

namespace globe {

// 16 bytes at p, whatever its alignment: one load, or the aligned words around it (which hold at
// least one of the 16 bytes each, so they lie in the buffer's allocation)
__device__ __forceinline__ uint4 load16_any(const uint8_t* __restrict__ p) {
    const unsigned a = (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u);
    if (a == 0) return __ldg(reinterpret_cast<const uint4*>(p));
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (a & 3u));
    if ((a & 3u) == 0) return make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
    const uint32_t w0 = __ldg(q), w1 = __ldg(q + 1), w2 = __ldg(q + 2), w3 = __ldg(q + 3), w4 = __ldg(q + 4);
    const unsigned sh = 8u * (a & 3u);
    return make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh),
                      __funnelshift_r(w3, w4, sh));
}

// A1 alleles and missing codes of two words' 32 samples: the low and the high bits of their codes
// packed into one word each, so that three popc (a quarter-rate instruction) serve both
__device__ __forceinline__ void count_codes(uint32_t x, uint32_t y, int& a, int& ms) {
    const uint32_t L = (x & 0x55555555u) | ((y & 0x55555555u) << 1);
    const uint32_t H = ((x >> 1) & 0x55555555u) | (y & 0xAAAAAAAAu);
    a += 2 * __popc(~(H | L)) + __popc(H & ~L);
    ms += __popc(L & ~H);
}

// One warp per SNP row: 16 bytes per lane and step, four steps' loads in flight, the bytes past
// the last whole 16 (with the last byte's phantom pairs masked) one per lane.  Bound by the
// payload's read (12.5 GB rows of 25 KB: one byte per lane took 8.7 ms, 1.4 TB/s).
__global__ void __launch_bounds__(256) k_bed_stats(const uint8_t* __restrict__ bed, int64_t M, int64_t stride, int32_t N,
                                                   float min_maf, float max_miss, int64_t* __restrict__ alt_out,
                                                   int64_t* __restrict__ miss_out, float* __restrict__ maf_out,
                                                   float* __restrict__ mr_out, uint8_t* __restrict__ keep_out) {
    const int lane = threadIdx.x & 31;
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= M) return;
    const int64_t bps = ((int64_t)N + 3) >> 2;
    const uint8_t* row = bed + s * stride;
    const int last_pairs = N - (int)((bps - 1) * 4);  // 1..4 real pairs in the last byte
    const unsigned last_mask = 0x55u & ((1u << (2 * last_pairs)) - 1u);
    int ai = 0, mi = 0;   // a lane's share of 2 N < 2^32 alleles
    const int nfull = (int)((bps - 1) >> 4);
    int q = lane;
    for (; q + 96 < nfull; q += 128) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = load16_any(row + (int64_t)(q + 32 * u) * 16);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            count_codes(v[u].x, v[u].y, ai, mi);
            count_codes(v[u].z, v[u].w, ai, mi);
        }
    }
    for (; q < nfull; q += 32) {
        const uint4 v = load16_any(row + (int64_t)q * 16);
        count_codes(v.x, v.y, ai, mi);
        count_codes(v.z, v.w, ai, mi);
    }
    for (int64_t b = (int64_t)nfull * 16 + lane; b < bps; b += 32) {
        unsigned x = row[b];
        unsigned m = (b == bps - 1) ? last_mask : 0x55u;
        unsigned L = x & 0x55u, H = (x >> 1) & 0x55u;
        ai += 2 * __popc(~(H | L) & m) + __popc(H & ~L & m);
        mi += __popc(L & ~H & m);
    }
    long long a = ai, ms = mi;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        ms += __shfl_xor_sync(0xffffffffu, ms, o);
    }
    if (lane == 0) {
        int n_obs = N - (int)ms;
        float f = (n_obs > 0) ? (float)a / (2.0f * (float)n_obs) : 0.0f;
        float mr = (float)ms / (float)N;
        bool k = (f >= min_maf && f <= (1.0f - min_maf) && mr <= max_miss);
        if (alt_out) alt_out[s] = a;
        if (miss_out) miss_out[s] = ms;
        if (maf_out) maf_out[s] = f;
        if (mr_out) mr_out[s] = mr;
        keep_out[s] = k ? 1 : 0;
    }
}

int bed_stats(globe_ctx* ctx, const uint8_t* d_bed, int64_t M, int64_t stride, int32_t N,
              float min_maf, float max_miss, int64_t* d_alt, int64_t* d_miss, float* d_maf,
              float* d_mr, uint8_t* d_keep) {
    if (M == 0) return GLOBE_OK;
    k_bed_stats<<<div_up(M, 8), 256, 0, ctx->stream>>>(d_bed, M, stride, N, min_maf, max_miss, d_alt,
                                                        d_miss, d_maf, d_mr, d_keep);
    GLOBE_LAUNCHED(ctx, "k_bed_stats");
    return GLOBE_OK;
}

// ---- indices of the kept SNPs, in order: per-CTA counts, their scan, the scatter ----
constexpr int KEEP_T = 1024;

__global__ void __launch_bounds__(KEEP_T) k_keep_count(const uint8_t* __restrict__ keep, int64_t M,
                                                       int64_t* __restrict__ cnt) {
    const int64_t s = (int64_t)blockIdx.x * KEEP_T + threadIdx.x;
    const int n = __syncthreads_count(s < M && keep[s]);
    if (threadIdx.x == 0) cnt[blockIdx.x] = n;
}
// exclusive scan in place, one CTA; cnt[nb] = the total
__global__ void __launch_bounds__(KEEP_T) k_keep_scan(int64_t* __restrict__ cnt, int nb) {
    __shared__ int64_t sm[KEEP_T];
    int64_t base = 0;
    for (int b0 = 0; b0 < nb; b0 += KEEP_T) {
        const int b = b0 + threadIdx.x;
        const int64_t v = b < nb ? cnt[b] : 0;
        sm[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < KEEP_T; o <<= 1) {
            const int64_t a = threadIdx.x >= o ? sm[threadIdx.x - o] : 0;
            __syncthreads();
            sm[threadIdx.x] += a;
            __syncthreads();
        }
        if (b < nb) cnt[b] = base + sm[threadIdx.x] - v;
        base += sm[KEEP_T - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) cnt[nb] = base;
}
__global__ void __launch_bounds__(KEEP_T) k_keep_scatter(const uint8_t* __restrict__ keep, int64_t M,
                                                         const int64_t* __restrict__ cnt, int64_t* __restrict__ idx) {
    __shared__ int wsum[KEEP_T / 32];
    const int64_t s = (int64_t)blockIdx.x * KEEP_T + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool k = s < M && keep[s];
    const unsigned bal = __ballot_sync(0xffffffffu, k);
    if (lane == 0) wsum[warp] = __popc(bal);
    __syncthreads();
    int64_t at = cnt[blockIdx.x] + __popc(bal & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) at += wsum[w];
    if (k) idx[at] = s;
}

// cnt: keep_blocks(M) + 1 values, left as the offsets and the number of kept SNPs
int keep_blocks(int64_t M) { return div_up(M, KEEP_T); }
int keep_scan(globe_ctx* ctx, const uint8_t* d_keep, int64_t M, int64_t* cnt) {
    if (M > 0) {
        k_keep_count<<<keep_blocks(M), KEEP_T, 0, ctx->stream>>>(d_keep, M, cnt);
        GLOBE_LAUNCHED(ctx, "k_keep_count");
    }
    k_keep_scan<<<1, KEEP_T, 0, ctx->stream>>>(cnt, keep_blocks(M));
    GLOBE_LAUNCHED(ctx, "k_keep_scan");
    return GLOBE_OK;
}
int keep_scatter(globe_ctx* ctx, const uint8_t* d_keep, int64_t M, const int64_t* cnt, int64_t* idx) {
    k_keep_scatter<<<keep_blocks(M), KEEP_T, 0, ctx->stream>>>(d_keep, M, cnt, idx);
    GLOBE_LAUNCHED(ctx, "k_keep_scatter");
    return GLOBE_OK;
}

// Kept rows of the payload -> the SNP-major tile-blocked copy (tile codes), 16 bytes per thread,
// straight from the payload: rows past Mk, bytes past the row and the phantom pairs of its last
// byte become genotype 0.  Bound by its one read and one write (12.5 GB each; the former copy
// of the kept rows moved as much again, a byte per lane, in 10.4 ms).
__global__ void __launch_bounds__(256) k_bed_layout(const uint8_t* __restrict__ bed, int64_t stride,
                                                    const int64_t* __restrict__ idx, int64_t Mk, int64_t bps, int32_t N,
                                                    int64_t ntiles, int64_t nch, uint8_t* __restrict__ dst) {
    using namespace tc;
    const int64_t total = ntiles * nch * (BM * PKB / 16);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t blkid = e / (BM * PKB / 16);
        const int within = (int)(e % (BM * PKB / 16));
        const int r = within >> 1, h = within & 1;
        const int64_t t = blkid / nch, c = blkid % nch;
        const int64_t row = t * BM + r, byte = c * PKB + h * 16;
        uint4 v = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        if (row < Mk && byte < bps) {
            const uint8_t* src = bed + idx[row] * stride + byte;
            if (byte + 16 < bps) {
                v = load16_any(src);
            } else {   // the row's last bytes
                uint32_t w[4] = {v.x, v.y, v.z, v.w};
                const int n = (int)(bps - byte), pairs = N - (int)((bps - 1) * 4);
                const uint32_t real = (1u << (2 * pairs)) - 1u;
                for (int q = 0; q < n; ++q) {
                    uint32_t b = src[q];
                    if (q == n - 1) b = (b & real) | (0xFFu & ~real);
                    w[q >> 2] = (w[q >> 2] & ~(0xFFu << (8 * (q & 3)))) | (b << (8 * (q & 3)));
                }
                v = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        v = make_uint4(recode_tile(v.x), recode_tile(v.y), recode_tile(v.z), recode_tile(v.w));
        const int64_t phys = (blkid * BM + r) * 2 + (h ^ ((r >> 2) & 1));   // halves swapped when bit 2 of r is set
        *reinterpret_cast<uint4*>(dst + phys * 16) = v;
    }
}

int bed_layout(globe_ctx* ctx, const uint8_t* d_bed, int64_t stride, const int64_t* d_idx, int64_t Mk, int64_t bps,
               int ntiles, int nch, uint8_t* dst) {
    const int64_t total = (int64_t)ntiles * nch * (tc::BM * tc::PKB / 16);
    k_bed_layout<<<(unsigned)std::min<int64_t>((total + 255) / 256, 65535), 256, 0, ctx->stream>>>(
        d_bed, stride, d_idx, Mk, bps, ctx->coh.N, ntiles, nch, dst);
    GLOBE_LAUNCHED(ctx, "k_bed_layout");
    return GLOBE_OK;
}

// zs(code) = (g - 2f) * inv_std with g(00)=2, g(01 missing)=0, g(10)=1, g(11)=0.
__global__ void k_snp_coefs(const int64_t* __restrict__ alt, const int64_t* __restrict__ miss,
                            const int64_t* __restrict__ idx, int64_t Mk, int32_t N,
                            double* __restrict__ f_out, double* __restrict__ inv_out,
                            double* __restrict__ zs) {
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Mk) return;
    int64_t s = idx[k];
    int n_obs = N - (int)miss[s];
    double f = (n_obs > 0) ? (double)alt[s] / (double)(2.0f * (float)n_obs) : 0.0;
    double den = 2.0 * f * (1.0 - f);
    double inv = (den > (double)1e-12f) ? 1.0 / sqrt(den) : 1.0;
    f_out[k] = f;
    inv_out[k] = inv;
    zs[k * 4 + 0] = (2.0 - 2.0 * f) * inv;
    zs[k * 4 + 1] = (0.0 - 2.0 * f) * inv;
    zs[k * 4 + 2] = (1.0 - 2.0 * f) * inv;
    zs[k * 4 + 3] = (0.0 - 2.0 * f) * inv;
}

int snp_coefs(globe_ctx* ctx, const int64_t* d_alt, const int64_t* d_miss, const int64_t* d_idx,
              int64_t Mk, int32_t N, double* d_f, double* d_inv, double* d_zs) {
    if (Mk == 0) return GLOBE_OK;
    k_snp_coefs<<<div_up(Mk, 256), 256, 0, ctx->stream>>>(d_alt, d_miss, d_idx, Mk, N, d_f, d_inv, d_zs);
    GLOBE_LAUNCHED(ctx, "k_snp_coefs");
    return GLOBE_OK;
}

// ---- synthetic genotypes (counter-based) --------------------------------

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float u21(uint64_t h, int part) {
    return ((float)((h >> (21 * part)) & 0x1FFFFFull) + 0.5f) * (1.0f / 2097152.0f);
}

// One thread per output byte (4 samples).
__global__ void k_synth_bed(uint8_t* __restrict__ bed, int64_t M, int32_t N, int64_t stride,
                            uint64_t seed, float maf_lo, float maf_hi, float miss_rate) {
    const int64_t bps = ((int64_t)N + 3) >> 2;
    const int64_t s = blockIdx.y + (int64_t)blockIdx.z * gridDim.y;
    if (s >= M) return;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < stride;
         b += (int64_t)gridDim.x * blockDim.x) {
        uint8_t v = 0;
        if (b < bps) {
            uint64_t hs = mix64(seed ^ mix64((uint64_t)s * 0x632BE59BD9B4E019ull));
            float p = maf_lo + (maf_hi - maf_lo) * u21(hs, 0);
            float pa1 = (u21(hs, 1) < 0.5f) ? 1.0f - p : p;
            unsigned byte = 0;
            for (int j = 0; j < 4; ++j) {
                int64_t i = b * 4 + j;
                unsigned code = 0;
                if (i < N) {
                    uint64_t h = mix64(hs ^ (uint64_t)(i + 1) * 0xD1342543DE82EF95ull);
                    int g = (u21(h, 0) < pa1) + (u21(h, 1) < pa1);
                    if (u21(h, 2) < miss_rate) code = 1;
                    else code = (g == 2) ? 0u : (g == 1 ? 2u : 3u);
                }
                byte |= code << (2 * j);
            }
            v = (uint8_t)byte;
        }
        bed[s * stride + b] = v;
    }
}

int synth_bed(globe_ctx* ctx, uint8_t* d_bed, int64_t M, int32_t N, int64_t stride, uint64_t seed,
              float maf_lo, float maf_hi, float miss_rate) {
    if (M == 0) return GLOBE_OK;
    int bx = div_up(stride, 256);
    if (bx > 64) bx = 64;
    int64_t gy = M < 65535 ? M : 65535;
    int64_t gz = (M + gy - 1) / gy;
    dim3 grid(bx, (unsigned)gy, (unsigned)gz);
    k_synth_bed<<<grid, 256, 0, ctx->stream>>>(d_bed, M, N, stride, seed, maf_lo, maf_hi, miss_rate);
    GLOBE_LAUNCHED(ctx, "k_synth_bed");
    return GLOBE_OK;
}

}  // namespace globe
