// k_solve.cu -- the record kernels of one block-PCG iteration.
//
// The iteration of the reference (PCGsolver.cpp:1362-1432, varCompEst.cpp:478-528) on V p
// (PCGsolver.cpp:1095-1266) and Q^-1 r (:1014-1049), arranged so that three record vectors
// x, r, p are all that is kept, and each is read and written as few times as the recurrences
// allow:
//   k_dir     x += alpha p (the step before's);  z = Q^-1 r;  p = z + beta p;
//             s0 = sum p, s1 = sum t p, pp = sum p^2 per individual;  Z = s0      (5 vectors)
//   product   GZ = sig2g A Z
//   k_step    per individual a0 = GZ + b0 s0 + b01 s1, a1 = b01 s0 + b1 s1;
//             p'Vp = sum sig2e pp + a0 s0 + a1 s1;  alpha = r'z / p'Vp
//   k_update  r -= alpha V p, V p = sig2e p + a0 + t a1 on the spot;  g = H (sum r, sum t r);
//             |r|^2, r'z with z = Q^-1 r = (r - g0 - t g1) / sig2e on the spot;  beta (3 vectors)
// V p and z are two numbers per individual away from p and r, so neither is stored (they were: 13
// vector transfers an iteration instead of 8), and p'Vp needs no pass over the records.
//
// Layout: the vectors are [record][column], column fastest, and a thread owns an (individual,
// column) pair with the columns of an individual on neighbouring threads: a warp reads whole
// runs of an individual's records, whatever the number of columns.  Individuals are taken in order
// of their record counts (Cohort::order), so the threads of a warp walk equally many records.  One
// thread's walk is a chain of loads and sums, and outlasts the rest where an individual has many
// records for the size of the solve: those are walked by teams of a CTA's threads, several
// individuals at a time, and the longest by a whole CTA each (shape(), which classes them).  The
// kernels are bound by the vectors' transfers (in double-float) or by the FP64 pipe (~16 operations
// a record and column; in FP64).
//
// Two arithmetics: FP64 (GLOBE_PREC_FP64), and double-float pairs (df.cuh) in the 8 bytes of
// each double under GLOBE_PREC_MIXED, column c scaled by a power of two (col_unscale) to a
// unit-size right-hand side.  What stays FP64 there: the GRM product's input and output, and every
// sum past FLUSH individuals of a thread (a team's sums over one individual's records are in
// double-float); alpha and beta are formed from those sums in FP64 and rounded to pairs.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "df.cuh"
#include "solve.cuh"
#include "tc_common.cuh"

namespace globe {

constexpr int ST = 288;            // threads per CTA at most
// Records per step of a thread, whose loads issue together, and resident CTAs per SM, k_dir and
// k_update: more of either was slower (k_update with 4 records and 3 CTAs: 60 against 53 us at
// N = 100k, k = 5, 255 against 204 us at N = 50k, k = 65; k_dir with 2 and 4: 153 and 38 against
// 158 and 36 us), and so was keeping an individual's r and t in registers for k_update's second
// pass over them (83 us: 2 CTAs).  With at most two CTAs an SM to run, where a chain of loads is
// what counts, k_update takes 4 records at a time (mixed, five columns, us an iteration with 2 / 4: 157
// CTAs 66.4 / 64.5, 295 74.9 / 73.4, 324 76.0 / 76.6, 393 78.6 / 82.0).
constexpr int RU_DIR = 4, RU_UPD = 2, RES_DIR = 3, RES_UPD = 4;
// CTAs per SM launched at most: k_dir's take two turns, the kernels that end in column sums one
// (fewer partials)
constexpr int PER_DIR = 2 * RES_DIR, PER_SUM = 4;
constexpr int PER_LONG = 2;        // and for the individuals that take a whole CTA
constexpr int TEAM = 8, TEAM_MOST = 32;   // threads of a team

struct ArithF64 {
    using V = double;
    using S = double;
    static __device__ __forceinline__ V load(const S* p) { return *p; }
    static __device__ __forceinline__ void store(S* p, V v) { *p = v; }
    static __device__ __forceinline__ V zero() { return 0.0; }
    static V host(double d) { return d; }
    static __device__ __forceinline__ V scalar(double d) { return d; }
    static __device__ __forceinline__ V from(double d) { return d; }
    static __device__ __forceinline__ V from_scaled(double d, int sh) { return sh ? ldexp(d, sh) : d; }
    static __device__ __forceinline__ double to_double(V v) { return v; }
    static __device__ __forceinline__ V neg(V a) { return -a; }
    static __device__ __forceinline__ V add(V a, V b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ V mul(V a, V b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ V madd(V a, V b, V c) { return __fma_rn(a, b, c); }
};
struct ArithDF {
    using V = df::D;
    using S = float2;
    static __device__ __forceinline__ V load(const S* p) { return df::load(p); }
    static __device__ __forceinline__ void store(S* p, V v) { df::store(p, v); }
    static __device__ __forceinline__ V zero() { return df::zero(); }
    static V host(double d) { return df::from_double_host(d); }
    static __device__ __forceinline__ V scalar(double d) { return df::from_double(d); }
    static __device__ __forceinline__ V from(double d) { return df::from_double_scaled(d, 0); }
    static __device__ __forceinline__ V from_scaled(double d, int sh) { return df::from_double_scaled(d, sh); }
    static __device__ __forceinline__ double to_double(V v) { return df::to_double(v); }
    static __device__ __forceinline__ V neg(V a) { return df::neg(a); }
    static __device__ __forceinline__ V add(V a, V b) { return df::add(a, b); }
    static __device__ __forceinline__ V mul(V a, V b) { return df::mul(a, b); }
    static __device__ __forceinline__ V madd(V a, V b, V c) { return df::madd(a, b, c); }
};

// A thread's sums over individuals: in the solve's arithmetic over FLUSH of them, past those in FP64,
// in the thread's places of tot (shared memory: registers for them spilled).  FP64 sums stay in `part`.
// (Double-float over all of a CTA's individuals, as many as N asks for: no faster at N = 100k, five
// columns 88.4 ms a solve either way, 37 226 and 228.)
constexpr int FLUSH = 8;
template <class A, int NQ>
struct Sums {
    typename A::V part[NQ];
    double* tot;   // NQ x ST
    int n = 0;
    static constexpr bool FLUSHED = !std::is_same_v<typename A::V, double>;
    __device__ __forceinline__ explicit Sums(double* sm) : tot(sm) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            part[q] = A::zero();
            if (FLUSHED) tot[q * ST + threadIdx.x] = 0.0;
        }
    }
    // after each individual
    __device__ __forceinline__ void next() {
        if (FLUSHED && ++n == FLUSH) {
            n = 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                tot[q * ST + threadIdx.x] += A::to_double(part[q]);
                part[q] = A::zero();
            }
        }
    }
    __device__ __forceinline__ double total(int q) const {
        return A::to_double(part[q]) + (FLUSHED ? tot[q * ST + threadIdx.x] : 0.0);
    }
};

// A class of individuals: n of them from order[i0] on, walked by `ctas` CTAs, rt threads of a CTA to
// each (individual, column)
struct Part {
    int32_t i0, n;
    int ctas, rt;
};
// What the kernels take of a solve (SolveVecs, solve.cuh) in their arithmetic's storage type
template <class A>
struct Args {
    typename A::S *x, *r, *p, *S0, *S1, *PP, *G;
    const typename A::S *t, *H;
    const int4* order;               // {block, first record, one past its last, individual} (Cohort::order)
    const int32_t *bind, *cols;
    int32_t N;
    int64_t Nrec;
    int k, kact, kc, ti;             // columns; active ones; columns per tile, individuals per CTA step
    typename A::V e, inv_e, b0, b01, b1;
    typename A::S *alpha, *beta;     // converted once, where they are formed
    double *rz, *pvp, *rr;
    double* part;
    int slots;                       // partials per column: CTAs
    Part cls[3];                     // who walks what: whole CTAs, teams, single threads
    unsigned* cnt;                   // arrival counts, zero between launches: per tile its groups' and
    unsigned* tiles_done;            // the groups' (sum_last); of the tiles
};

// Thread (il, c): column c of the CTA's tile, individual il of its step
struct Lane {
    int c, il, col;
    bool on;
};
template <class A>
__device__ __forceinline__ Lane lane_of(const Args<A>& a) {
    Lane l;
    const int t = threadIdx.x;
    l.il = t / a.kc;
    l.c = (int)blockIdx.y * a.kc + t - l.il * a.kc;
    l.on = l.il < a.ti && l.c < a.kact;
    l.col = l.on ? (a.cols ? a.cols[l.c] : l.c) : 0;
    return l;
}

// the class of CTA x, and x within it
template <class A>
__device__ __forceinline__ int class_of(const Args<A>& a, int& x) {
    int p = 0;
    for (; p < 2 && x >= a.cls[p].ctas; ++p) x -= a.cls[p].ctas;
    return p;
}
// A thread's place in its CTA's class: individuals come `per` at a time, this one's slot of them
// and its place among the slot's rt threads
struct Team {
    unsigned i0, n, j0, js;   // individuals i0 + j, j = j0 + slot, in steps of js
    int rt, per, slot, rl;
    bool on;
};
template <bool MANY, class A>
__device__ __forceinline__ Team team_of(const Args<A>& a, const Lane& l, const Part& p, int x) {
    Team w;
    w.i0 = p.i0;
    w.n = p.n;
    w.rt = MANY ? p.rt : 1;
    w.per = MANY ? a.ti / p.rt : a.ti;
    w.slot = MANY ? l.il / p.rt : l.il;
    w.rl = MANY ? l.il - w.slot * p.rt : 0;
    w.on = l.on && (!MANY || w.slot < w.per);
    w.j0 = (unsigned)(x * w.per);
    w.js = (unsigned)(p.ctas * w.per);
    return w;
}

// v[q] over the rt threads of each slot and column, in the rl = 0 thread's v and in sm[q ST + its t]
// (every thread of the CTA calls it)
template <int Q, class A>
__device__ __forceinline__ void team_sum(const Args<A>& a, const Team& w, typename A::V (&v)[Q], typename A::V* sm) {
    const int t = threadIdx.x;
#pragma unroll
    for (int q = 0; q < Q; ++q) sm[q * ST + t] = v[q];
    __syncthreads();
    int s = 1;
    while (s < w.rt) s <<= 1;
    for (s >>= 1; s > 0; s >>= 1) {
        if (w.on && w.rl < s && w.rl + s < w.rt) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                v[q] = A::add(v[q], sm[q * ST + t + s * a.kc]);
                sm[q * ST + t] = v[q];
            }
        }
        __syncthreads();
    }
}

// ---- k_dir -----------------------------------------------------------------------

// the CTA's individuals; returns the largest abs_hi of the thread's sums
template <class A, bool MANY>
__device__ __forceinline__ unsigned dir_walk(const Args<A>& a, const Lane& l, int c, int x, const bool first,
                                             typename A::V* sm, double* __restrict__ Zi) {
    using V = typename A::V;
    constexpr int RU = RU_DIR;
    const Team w = team_of<MANY>(a, l, a.cls[c], x);
    const V inv_e = a.inv_e, al = l.on && !first ? A::load(a.alpha + l.col) : A::zero(),
            be = l.on && !first ? A::load(a.beta + l.col) : A::zero();
    const int step = MANY ? w.rt : 1;
    unsigned m = 0;
    for (unsigned j = w.j0; j < w.n; j += w.js) {   // uniform over the CTA
        const unsigned idx = j + w.slot;
        V s0 = A::zero(), s1 = A::zero(), pp = A::zero();
        int b = 0, i = 0;
        bool in = w.on && idx < w.n;
        if (in) {
            const int4 ord = a.order[w.i0 + idx];
            const int st = ord.y, en = ord.z;
            b = ord.x;
            i = ord.w;
            if (!GLOBE_BOUNDS(b >= 0 && b < a.N && st >= 0 && st <= en && en <= a.Nrec && i >= 0 && i < a.N, 0x1601u))
                in = false, b = 0;
            const V g0 = A::load(a.G + 2 * ((size_t)b * a.k + l.col)), g1 = A::load(a.G + 2 * ((size_t)b * a.k + l.col) + 1);
            for (int q0 = st + (MANY ? w.rl : 0); in && q0 < en; q0 += RU * step) {
                V rv[RU], pv[RU], xv[RU], tv[RU];
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int q = q0 + u * step;
                    if (q < en) {
                        const size_t o = (size_t)q * a.k + l.col;
                        rv[u] = A::load(a.r + o);
                        tv[u] = A::load(a.t + q);
                        if (!first) {
                            pv[u] = A::load(a.p + o);
                            xv[u] = A::load(a.x + o);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int q = q0 + u * step;
                    if (q < en) {
                        const size_t o = (size_t)q * a.k + l.col;
                        V v = A::madd(rv[u], inv_e, A::neg(A::madd(g1, tv[u], g0)));   // z
                        if (!first) {
                            A::store(a.x + o, A::madd(al, pv[u], xv[u]));
                            v = A::madd(be, pv[u], v);
                        }
                        A::store(a.p + o, v);
                        s0 = A::add(s0, v);
                        s1 = A::madd(tv[u], v, s1);
                        pp = A::madd(v, v, pp);
                    }
                }
            }
        }
        if (MANY) {
            V v[3] = {s0, s1, pp};
            team_sum(a, w, v, sm);
            s0 = v[0];
            s1 = v[1];
            pp = v[2];
            in = in && w.rl == 0;
        }
        if (in) {
            const size_t o = (size_t)b * a.k + l.col;
            A::store(a.S0 + o, s0);
            A::store(a.S1 + o, s1);
            A::store(a.PP + o, pp);
            const double z = A::to_double(s0);
            Zi[i + (size_t)l.c * a.N] = z;
            m = max(m, tc::abs_hi(z));
        }
    }
    return m;
}

template <class A>
__global__ void __launch_bounds__(ST, RES_DIR) k_dir(Args<A> a, const bool first, double* __restrict__ Zi, unsigned* zhi) {
    __shared__ typename A::V sm[3 * ST];
    __shared__ unsigned smu[ST];
    const Lane l = lane_of(a);
    smu[threadIdx.x] = 0u;
    int x = blockIdx.x;
    const int p = class_of(a, x);
    const unsigned m = p < 2 ? dir_walk<A, true>(a, l, p, x, first, sm, Zi) : dir_walk<A, false>(a, l, 2, x, first, sm, Zi);
    if (zhi) {   // the scale of the product's input (k_col_max's part)
        __syncthreads();
        const int cl = threadIdx.x - l.il * a.kc;
        if (l.on && m) atomicMax(&smu[cl], m);
        __syncthreads();
        if (l.on && l.il == 0 && smu[cl]) atomicMax(zhi + l.c, smu[cl]);
    }
}

// ---- column sums over the CTAs -------------------------------------------------------
//
// An FP64 instruction takes 16 clocks of an SM's FP64 pipe whatever its active lanes, and a
// dependent one ~40: so every sum keeps columns on the lanes and is two steps of ~sqrt terms.  A
// CTA adds up its threads' sums and leaves one partial per column and quantity; the last CTA of
// each group to arrive adds up the group's, and the last group's the groups' (one group where the
// CTA's threads can take 16 partials each: a second round of arrivals costs ~4 us).  (A warp per
// column with shuffles, all partials in one last CTA, took 45 us at 65 columns.)  The order is one,
// so the sums' bits are.

// total of the R rows of nw values in sm, valid in threads t < nw; ends without a barrier
__device__ __forceinline__ double two_step(const double* sm, double* sm2, int R, int nw) {
    const int t = threadIdx.x;
    int ns = 1;
    while (ns * ns < R) ++ns;
    ns = max(1, min(ns, (int)blockDim.x / nw));
    const int j0 = t / nw, w = t - j0 * nw;
    double s = 0.0;
    if (j0 < ns && j0 < R) {
        s = sm[j0 * nw + w];
        for (int j = j0 + ns; j < R; j += ns) s += sm[j * nw + w];
    }
    if (ns == 1) return s;
    sm2[t] = s;
    __syncthreads();
    if (t < nw)
        for (int j = 1; j < min(ns, R); ++j) s += sm2[j * nw + t];
    return s;
}

// v summed over the tile's CTAs into out0[col] (and out1[col], the second quantity); returns true in
// every thread of the last CTA, once they are written and visible to it
template <int NQ, class A>
__device__ __forceinline__ bool sum_last(const Args<A>& a, const Lane& l, const double (&v)[NQ], int slot,
                                         double* __restrict__ out0, double* __restrict__ out1) {
    __shared__ double sm[NQ * ST], sm2[ST], smd[ST], smd2[ST];
    __shared__ bool last;
    const int t = threadIdx.x, kc = a.kc, c0 = blockIdx.y * kc, nc = min(kc, a.kact - c0), nw = NQ * kc;
    // thread t < nw stands for quantity q and column c of the tile
    const int q = t >= kc ? 1 : 0, c = t - q * kc;
    const bool mine = t < nw && c < nc;
    if (l.il < a.ti) {
        const int cl = t - l.il * kc;
#pragma unroll
        for (int p = 0; p < NQ; ++p) sm[(l.il * NQ + p) * kc + cl] = l.on ? v[p] : 0.0;
    }
    __syncthreads();
    const double s = two_step(sm, sm2, a.ti, nw);
    const size_t row = (size_t)NQ * a.kact;
    if (mine) a.part[(size_t)slot * row + (size_t)q * a.kact + c0 + c] = s;
    const int P = (int)blockDim.x / nw;   // threads per column and quantity
    const int gs = min(a.slots, max(32, 16 * P)), ng = (a.slots + gs - 1) / gs, g = slot / gs;
    const int gn = min(gs, a.slots - g * gs);
    unsigned* cnt = a.cnt + blockIdx.y * (ng + 1);
    double* gpart = a.part + (size_t)a.slots * row;
    for (int level = 0;; ++level) {   // 0: this CTA's group; 1: the groups
        if (t < nw) __threadfence();   // what this CTA wrote, then its arrival
        __syncthreads();
        if (t == 0) {
            unsigned* const n = cnt + (level == 0 ? g : ng);
            last = atomicAdd(n, 1u) == (unsigned)(level == 0 ? gn : ng) - 1u;
            if (last) *n = 0u;
        }
        __syncthreads();
        if (!last) return false;
        __threadfence();
        const double* src = level == 0 ? a.part + (size_t)g * gs * row : gpart;
        const int m = level == 0 ? gn : ng;
        const int j0 = t / nw, w = t - j0 * nw, wq = w >= kc ? 1 : 0, wc = w - wq * kc;
        if (j0 < P) {
            double x = 0.0;
            if (wc < nc) {
                const double* pc = src + (size_t)wq * a.kact + c0 + wc;
#pragma unroll 8
                for (int j = j0; j < m; j += P) x += __ldcg(pc + (size_t)j * row);
            }
            smd[j0 * nw + w] = x;
        }
        __syncthreads();
        const double x = two_step(smd, smd2, P, nw);
        const bool fin = level == 1 || ng == 1;
        if (mine) {
            if (fin) (q ? out1 : out0)[a.cols ? a.cols[c0 + c] : c0 + c] = x;
            else gpart[(size_t)g * row + (size_t)q * a.kact + c0 + c] = x;
        }
        if (fin) break;
        __syncthreads();   // smd is written again
    }
    if (t < nw) __threadfence();
    __syncthreads();
    return true;
}

// ---- k_step ----------------------------------------------------------------------

template <class A>
__global__ void __launch_bounds__(ST) k_step(Args<A> a, const double* __restrict__ GZ) {
    using V = typename A::V;
    const Lane l = lane_of(a);
    const V e = a.e, b0 = a.b0, b01 = a.b01, b1 = a.b1;
    __shared__ double tot[ST];
    Sums<A, 1> dot(tot);
    for (int64_t g = blockIdx.x; g * a.ti < a.N; g += gridDim.x) {
        const int64_t b = g * a.ti + l.il;
        if (!l.on || b >= a.N || !GLOBE_BOUNDS(a.bind[b] >= 0 && a.bind[b] < a.N, 0x1701u)) continue;
        const size_t o = (size_t)b * a.k + l.col;
        const V s0 = A::load(a.S0 + o), s1 = A::load(a.S1 + o), pp = A::load(a.PP + o);
        const V gz = A::from(GZ[a.bind[b] + (size_t)l.c * a.N]);
        const V a0 = A::madd(b0, s0, A::madd(b01, s1, gz)), a1 = A::madd(b01, s0, A::mul(b1, s1));
        A::store(a.S0 + o, a0);
        A::store(a.S1 + o, a1);
        dot.part[0] = A::madd(e, pp, A::madd(a0, s0, A::madd(a1, s1, dot.part[0])));
        dot.next();
    }
    const double v[1] = {dot.total(0)};
    if (sum_last<1>(a, l, v, blockIdx.x, a.pvp, nullptr) && threadIdx.x < a.kc) {
        const int c = blockIdx.y * a.kc + threadIdx.x;
        if (c < a.kact) {
            const int col = a.cols ? a.cols[c] : c;
            const double q = __ldcg(a.pvp + col);
            A::store(a.alpha + col, A::scalar(q != 0.0 ? a.rz[col] / q : 0.0));
        }
    }
}

// ---- the stopping rule on the device (solver.cu's device loop) ---------------------------

// the host loop's stopping rule (pcg_run), after iteration st->it + 1, by one warp: a lane per
// column (one thread's square roots and quotients took 0.3 us a column)
__device__ void pcg_check(const PcgLoop& p, const double* rr, const double* pvp, const int32_t* cols, int kact) {
    PcgLoopState* st = p.st;
    const int lane = threadIdx.x & 31;
    int bad = INT_MAX;   // the first active column that broke down
    for (int c = lane; c < kact && bad == INT_MAX; c += 32) {
        const int j = cols[c];
        if (!(__ldcg(pvp + j) > 0.0) || !isfinite(__ldcg(rr + j))) bad = c;
    }
    bad = __reduce_min_sync(0xffffffffu, bad);
    long long mx = 0;    // bits of the largest ratio (non-negative doubles order like their bits)
    bool open = false;   // a column above the tolerance (GLOBE_RULE_AIREML)
    for (int j = lane; j < p.k; j += 32) {
        const double r = sqrt(__ldcg(rr + j)) * (p.unsc ? p.unsc[j] : 1.0), nb = sqrt(p.bb[j]);
        if (p.rule == GLOBE_RULE_PCGSOLVER) {
            const double small_b = (double)1e-12f;  // PCGsolver.cpp:1365, :1393
            const double q = nb > small_b ? r / nb : 0.0;
            if (q > __longlong_as_double(mx)) mx = __double_as_longlong(q);
        } else {
            open = open || (p.bb[j] > 0.0 && !(r < p.tol * nb));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    open = __any_sync(0xffffffffu, open);
    if (lane != 0) return;
    const int it = st->it + 1;
    st->it = it;
    st->rhs_iters += kact;
    if (bad != INT_MAX) {
        st->status = 4;
        st->err_col = cols[bad];
        cudaGraphSetConditional(p.h, 0u);
        return;
    }
    bool stop = false;
    if (p.rule == GLOBE_RULE_PCGSOLVER) {
        const double m = __longlong_as_double(mx);
        if (m < p.tol) {
            st->status = 1;
            stop = true;
        } else {
            const double last = st->last;
            if (last - m < (double)5e-3f * last) ++st->stag;
            else st->stag = 0;
            st->last = m;
            if (st->stag >= 10) {
                st->status = 2;
                stop = true;
            }
        }
    } else if (!open) {
        st->status = 1;
        stop = true;
    }
    if (!stop && it >= p.maxit) {
        st->status = 3;
        stop = true;
    }
    cudaGraphSetConditional(p.h, stop ? 0u : 1u);
}

// ---- k_update ---------------------------------------------------------------------

// the CTA's individuals: |r|^2 and r'z of the thread's records.  INIT: r stays (the solve's
// start): g and r'z only
template <class A, bool MANY, bool INIT, int RU>
__device__ __forceinline__ void update_walk(const Args<A>& a, const Lane& l, int c, int x, typename A::V* sm,
                                            Sums<A, 2>& sums) {
    using V = typename A::V;
    const Team w = team_of<MANY>(a, l, a.cls[c], x);
    const V inv_e = a.inv_e, e = a.e, na = INIT || !l.on ? A::zero() : A::neg(A::load(a.alpha + l.col));
    const int step = MANY ? w.rt : 1;
    for (unsigned j = w.j0; j < w.n; j += w.js) {   // uniform over the CTA
        const unsigned idx = j + w.slot;
        int b = 0, st = 0, en = 0;
        V s0 = A::zero(), s1 = A::zero(), a0 = A::zero(), a1 = A::zero();
        bool in = w.on && idx < w.n;
        if (in) {
            const int4 ord = a.order[w.i0 + idx];
            b = ord.x;
            st = ord.y;
            en = ord.z;
            if (!GLOBE_BOUNDS(b >= 0 && b < a.N && st >= 0 && st <= en && en <= a.Nrec, 0x1801u)) in = false, b = st = en = 0;
        }
        const size_t o = (size_t)b * a.k + l.col;
        if (!INIT && in) {
            a0 = A::load(a.S0 + o);
            a1 = A::load(a.S1 + o);
        }
        // r - alpha V p of record q
        auto next = [&](V rv, V pv, V tv) { return INIT ? rv : A::madd(na, A::madd(e, pv, A::madd(tv, a1, a0)), rv); };
        auto finish = [&](V& g0, V& g1) {   // g / sig2e of the individual, kept for k_dir
            const typename A::S* hb = a.H + 4 * (size_t)b;
            g0 = A::mul(A::madd(A::load(hb), s0, A::mul(A::load(hb + 1), s1)), inv_e);
            g1 = A::mul(A::madd(A::load(hb + 2), s0, A::mul(A::load(hb + 3), s1)), inv_e);
            if (!MANY || w.rl == 0) {
                A::store(a.G + 2 * o, g0);
                A::store(a.G + 2 * o + 1, g1);
            }
        };
        const int q1 = st + (MANY ? w.rl : 0);
        for (int q0 = q1; q0 < en; q0 += RU * step) {
            V rv[RU], pv[RU], tv[RU];
#pragma unroll
            for (int u = 0; u < RU; ++u) {
                const int q = q0 + u * step;
                if (q < en) {
                    const size_t oq = (size_t)q * a.k + l.col;
                    rv[u] = A::load(a.r + oq);
                    tv[u] = A::load(a.t + q);
                    if (!INIT) pv[u] = A::load(a.p + oq);
                }
            }
#pragma unroll
            for (int u = 0; u < RU; ++u) {
                const int q = q0 + u * step;
                if (q < en) {
                    const V rn = next(rv[u], pv[u], tv[u]);
                    if (!INIT) {
                        A::store(a.r + (size_t)q * a.k + l.col, rn);
                        sums.part[1] = A::madd(rn, rn, sums.part[1]);
                    }
                    s0 = A::add(s0, rn);
                    s1 = A::madd(tv[u], rn, s1);
                }
            }
        }
        if (MANY) {
            V v[2] = {s0, s1};
            team_sum(a, w, v, sm);
            const int t0 = threadIdx.x - w.rl * a.kc;   // the slot's first thread of this column
            s0 = sm[t0];
            s1 = sm[ST + t0];
            __syncthreads();
        }
        if (in) {
            V g0, g1;
            finish(g0, g1);
            for (int q0 = q1; q0 < en; q0 += RU * step) {
                V rv[RU], tv[RU];
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int q = q0 + u * step;
                    if (q < en) {
                        rv[u] = A::load(a.r + (size_t)q * a.k + l.col);
                        tv[u] = A::load(a.t + q);
                    }
                }
#pragma unroll
                for (int u = 0; u < RU; ++u)
                    if (q0 + u * step < en)
                        sums.part[0] = A::madd(rv[u], A::madd(rv[u], inv_e, A::neg(A::madd(g1, tv[u], g0))), sums.part[0]);
            }
        }
        sums.next();
    }
}

template <class A, bool INIT, int RU>
__global__ void __launch_bounds__(ST, RU == RU_UPD ? RES_UPD : 2) k_update(Args<A> a, PcgLoop loop) {
    using V = typename A::V;
    __shared__ V sm[2 * ST];
    const Lane l = lane_of(a);
    int x = blockIdx.x;
    const int p = class_of(a, x);
    __shared__ double tot[2 * ST];
    Sums<A, 2> sums(tot);   // r'z, |r|^2
    if (p < 2) update_walk<A, true, INIT, RU>(a, l, p, x, sm, sums);
    else update_walk<A, false, INIT, RU>(a, l, 2, x, sm, sums);
    const double v[2] = {sums.total(0), sums.total(1)};
    // r'z (new) lands in rz's second half (k entries), |r|^2 in rr
    double* rz2 = a.rz + a.k;
    if (!sum_last<2>(a, l, v, blockIdx.x, rz2, INIT ? rz2 + a.k : a.rr)) return;
    if (threadIdx.x < a.kc) {
        const int c = blockIdx.y * a.kc + threadIdx.x;
        if (c < a.kact) {
            const int col = a.cols ? a.cols[c] : c;
            const double old = a.rz[col], nw = __ldcg(rz2 + col);
            if (!INIT) A::store(a.beta + col, A::scalar(old != 0.0 ? nw / old : 0.0));
            a.rz[col] = nw;
        }
    }
    if (loop.st && threadIdx.x < 32) {   // the last tile to finish applies the stopping rule
        bool mine = true;
        if (gridDim.y > 1) {
            __threadfence();
            unsigned n = 0;
            if (threadIdx.x == 0) n = atomicAdd(a.tiles_done, 1u);
            mine = __shfl_sync(0xffffffffu, n, 0) == gridDim.y - 1u;
            if (mine && threadIdx.x == 0) *a.tiles_done = 0u;
            __threadfence();
        }
        if (mine) pcg_check(loop, a.rr, a.pvp, a.cols, a.kact);
    }
}

// ---- between column-major FP64 and the solve's layout ------------------------------------

constexpr int CV_R = 256, CV_C = 8;   // records (and threads) and columns of a tile

// 2^-e for the power of two u = 2^e, from its exponent bits
__device__ __forceinline__ int neg_exp2(double u) { return 1023 - (int)((__double_as_longlong(u) >> 52) & 0x7ff); }

// out[record][column] = in (column-major, n rows) / unsc[column]
template <class A>
__global__ void __launch_bounds__(CV_R) k_to_rows(const double* __restrict__ in, int64_t n, int k,
                                                const double* __restrict__ unsc, typename A::S* __restrict__ out) {
    __shared__ double sm[CV_C][CV_R + 1];
    const int64_t r0 = (int64_t)blockIdx.x * CV_R;
    const int c0 = blockIdx.y * CV_C, nc = min(CV_C, k - c0);
    const int nr = (int)(n - r0 < CV_R ? n - r0 : CV_R);
    for (int c = 0; c < nc; ++c)
        if ((int)threadIdx.x < nr) sm[c][threadIdx.x] = in[r0 + threadIdx.x + (size_t)(c0 + c) * n];
    __syncthreads();
    for (int w = threadIdx.x; w < nr * nc; w += CV_R) {
        const int r = w / nc, c = w - r * nc;
        A::store(out + (size_t)(r0 + r) * k + c0 + c, A::from_scaled(sm[c][r], unsc ? neg_exp2(unsc[c0 + c]) : 0));
    }
}

// out (column-major) = unsc (x + alpha p); without alpha, x alone
template <class A>
__global__ void __launch_bounds__(CV_R) k_from_rows(const typename A::S* __restrict__ x, const typename A::S* __restrict__ p,
                                                  const typename A::S* __restrict__ alpha, int64_t n, int k,
                                                  const double* __restrict__ unsc, double* __restrict__ out) {
    __shared__ double sm[CV_C][CV_R + 1];
    const int64_t r0 = (int64_t)blockIdx.x * CV_R;
    const int c0 = blockIdx.y * CV_C, nc = min(CV_C, k - c0);
    const int nr = (int)(n - r0 < CV_R ? n - r0 : CV_R);
    for (int w = threadIdx.x; w < nr * nc; w += CV_R) {
        const int r = w / nc, c = w - r * nc;
        const size_t o = (size_t)(r0 + r) * k + c0 + c;
        typename A::V v = A::load(x + o);
        if (alpha) v = A::madd(A::load(alpha + c0 + c), A::load(p + o), v);
        sm[c][r] = A::to_double(v) * (unsc ? unsc[c0 + c] : 1.0);
    }
    __syncthreads();
    for (int c = 0; c < nc; ++c)
        if ((int)threadIdx.x < nr) out[r0 + threadIdx.x + (size_t)(c0 + c) * n] = sm[c][threadIdx.x];
}

__global__ void k_to_df(const double* __restrict__ in, int64_t n, float2* __restrict__ out) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        df::store(out + e, df::from_double_scaled(in[e], 0));
}
// unsc[c] = col_unscale(bb[c]), once per solve
__global__ void k_col_unscale(const double* __restrict__ bb, int k, double* __restrict__ unsc) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < k) unsc[c] = col_unscale(bb[c]);
}

// ---- host side ---------------------------------------------------------------------

int to_df(globe_ctx* ctx, const double* in, int64_t n, float2* out) {
    if (n < 1) return GLOBE_OK;
    k_to_df<<<(unsigned)std::min<int64_t>((n + 1023) / 1024, 1024), 256, 0, ctx->stream>>>(in, n, out);
    GLOBE_LAUNCHED(ctx, "k_to_df");
    return GLOBE_OK;
}

int col_unscales(globe_ctx* ctx, const double* bb, int k, double* unsc) {
    k_col_unscale<<<div_up(k, 128), 128, 0, ctx->stream>>>(bb, k, unsc);
    GLOBE_LAUNCHED(ctx, "k_col_unscale");
    return GLOBE_OK;
}

// Column tiles of at most 128, near-equal: whole rows up to 128 columns, since a row's sectors are
// shared with its neighbours' (two tiles of 33 of 65 columns read 1.6 times the vectors).  As many
// individuals as leave at most 256 threads, or one more where that wastes fewer.  At most per_sm
// CTAs per SM over all tiles for each class, each taking every gridDim.x-th group of individuals.
//
// Classes (by_length): one thread walks up to `one` records, ~0.5 us each in a chain: SOLVE_LONG where
// one CTA's threads an SM suffice for the teams of the rest (N = 20k, records geometric with mean 10,
// five columns: 6.44 ms a solve, 6.57 with 43), else the more the larger the solve, which takes
// longer anyway.  Beyond, a team of TEAM threads, and past 32 records for each of those (or half of
// `one`) the whole CTA.  A team doubles while its threads have more than 16 records and all teams
// still run at once.  us an iteration with one
// thread up to 32 and a CTA for each longer individual / with one thread for all / so (mixed; M =
// 1000): N = 2000, 100-200 records, one column 101 / 248 / 62; N = 20000, 33-48, one 542 / 108 / 114;
// 100-200, five 788 / 560 / 341; N = 100000, 40-60, one 2756 / 321 / 331, five 2863 / 592 / 598; N =
// 20000, 3-10 and 600 of 300 records, five 102 / 358 / 98.  (A team from 32 records on whatever the
// size: N = 20000, 28-36, one column 131, 98 so; a mix of single threads and teams has both tails.)
struct Shape {
    int kc, ti, threads, tiles, ctas;
    Part cls[3];
};
static Shape shape(const globe_ctx* ctx, int kact, int per_sm, bool by_length) {
    auto& c = ctx->coh;
    Shape s;
    s.kc = div_up(kact, div_up(kact, 128));
    s.tiles = div_up(kact, s.kc);
    s.ti = 256 / s.kc;
    if (256 - s.ti * s.kc >= 32 && (s.ti + 1) * s.kc <= ST) ++s.ti;
    s.threads = div_up(s.ti * s.kc, 32) * 32;
    auto most = [&](int per) { return std::max(1, per * 152 / s.tiles); };
    auto longer = [&](int64_t records) {   // individuals of more records
        return (int)(std::partition_point(c.long_len.begin(), c.long_len.end(), [&](int32_t l) { return l > records; }) -
                     c.long_len.begin());
    };
    int rt = std::min(TEAM, s.ti);
    const int64_t load = c.Nrec * kact;
    int64_t one = SOLVE_LONG;
    if ((int64_t)c.long_len.size() * TEAM * kact > 152 * 256) one += std::min<int64_t>(32, load / 100000) + load / 1000000;
    const int64_t team = std::max(one, rt * std::max<int64_t>(32, one / 2));   // not below `one`, which may be odd
    const int n1 = by_length ? longer(one) : 0, n0 = by_length ? longer(team) : 0;
    while (n1 > n0 && 2 * rt <= std::min(TEAM_MOST, s.ti) && c.long_len[n0] > 16 * rt &&
           div_up(n1 - n0, s.ti / (2 * rt)) <= most(PER_LONG))
        rt *= 2;
    s.cls[0] = Part{0, n0, std::min(n0, most(PER_LONG)), s.ti};
    s.cls[1] = Part{n0, n1 - n0, std::min(div_up(n1 - n0, s.ti / rt), most(per_sm)), rt};
    s.cls[2] = Part{n1, c.N - n1, std::min(div_up(c.N - n1, s.ti), most(per_sm)), 1};
    s.ctas = s.cls[0].ctas + s.cls[1].ctas + s.cls[2].ctas;
    return s;
}

template <class A>
static int args(globe_ctx* ctx, const SolveVecs& v, int kact, const Shape& s, Args<A>* out) {
    using S = typename A::S;
    auto& c = ctx->coh;
    constexpr bool df = std::is_same_v<A, ArithDF>;
    Args<A> a;
    a.x = (S*)v.x;
    a.r = (S*)v.r;
    a.p = (S*)v.p;
    const size_t nk = (size_t)c.N * v.k;
    a.S0 = (S*)v.ind;
    a.S1 = a.S0 + nk;
    a.PP = a.S1 + nk;
    a.G = a.PP + nk;
    a.t = df ? (const S*)c.tdf : (const S*)c.times();
    a.H = (const S*)ctx->ws[df ? WS_HDF : WS_H].p;
    a.bind = c.bind;
    a.order = c.order;
    a.cols = v.cols;
    a.N = c.N;
    a.Nrec = c.Nrec;
    a.k = v.k;
    a.kact = kact;
    a.kc = s.kc;
    a.ti = s.ti;
    a.e = A::host(ctx->vc[0]);
    a.inv_e = A::host(1.0 / ctx->vc[0]);
    a.b0 = A::host(ctx->vc[2]);
    a.b01 = A::host(ctx->vc[3]);
    a.b1 = A::host(ctx->vc[4]);
    a.alpha = (S*)v.alpha;
    a.beta = (S*)v.beta;
    a.rz = v.rz;
    a.pvp = v.pvp;
    a.rr = v.rr;
    a.slots = s.ctas;
    std::copy(s.cls, s.cls + 3, a.cls);
    const size_t most = (2 * PER_SUM + PER_LONG) * 152 + 3, groups = most / 32 + 1;   // for any number of active columns
    GLOBE_RET(ws(ctx, WS_PART, (most + groups) * 2 * v.k, &a.part));
    GLOBE_RET(tc_counters(ctx, (size_t)div_up(v.k, 128) * (groups + 1) + 1, &a.tiles_done));
    a.cnt = a.tiles_done + 1;
    *out = a;
    return GLOBE_OK;
}

template <class A>
static int dir(globe_ctx* ctx, const SolveVecs& v, int kact, bool first, double* Zi, unsigned* zhi) {
    const Shape s = shape(ctx, kact, PER_DIR, true);
    Args<A> a;
    GLOBE_RET(args(ctx, v, kact, s, &a));
    k_dir<A><<<dim3(s.ctas, s.tiles), s.threads, 0, ctx->stream>>>(a, first, Zi, zhi);
    GLOBE_LAUNCHED(ctx, "k_dir");
    return GLOBE_OK;
}

template <class A>
static int step(globe_ctx* ctx, const SolveVecs& v, int kact, const double* GZ) {
    const Shape s = shape(ctx, kact, PER_SUM, false);
    Args<A> a;
    GLOBE_RET(args(ctx, v, kact, s, &a));
    k_step<A><<<dim3(s.ctas, s.tiles), s.threads, 0, ctx->stream>>>(a, GZ);
    GLOBE_LAUNCHED(ctx, "k_step");
    return GLOBE_OK;
}

template <class A, bool INIT>
static int update(globe_ctx* ctx, const SolveVecs& v, int kact, const PcgLoop& loop) {
    const Shape s = shape(ctx, kact, PER_SUM, true);
    Args<A> a;
    GLOBE_RET(args(ctx, v, kact, s, &a));
    const dim3 grid(s.ctas, s.tiles);
    if (grid.x * grid.y <= 2 * 152) k_update<A, INIT, 4><<<grid, s.threads, 0, ctx->stream>>>(a, loop);
    else k_update<A, INIT, RU_UPD><<<grid, s.threads, 0, ctx->stream>>>(a, loop);
    GLOBE_LAUNCHED(ctx, "k_update");
    return GLOBE_OK;
}

int solve_init(globe_ctx* ctx, const SolveVecs& v) {
    SolveVecs all = v;
    all.cols = nullptr;
    return v.df ? update<ArithDF, true>(ctx, all, v.k, PcgLoop()) : update<ArithF64, true>(ctx, all, v.k, PcgLoop());
}
int solve_dir(globe_ctx* ctx, const SolveVecs& v, int kact, bool first, double* Zi, unsigned* zhi) {
    return v.df ? dir<ArithDF>(ctx, v, kact, first, Zi, zhi) : dir<ArithF64>(ctx, v, kact, first, Zi, zhi);
}
int solve_step(globe_ctx* ctx, const SolveVecs& v, int kact, const double* GZ) {
    return v.df ? step<ArithDF>(ctx, v, kact, GZ) : step<ArithF64>(ctx, v, kact, GZ);
}
int solve_update(globe_ctx* ctx, const SolveVecs& v, int kact, const PcgLoop& loop) {
    return v.df ? update<ArithDF, false>(ctx, v, kact, loop) : update<ArithF64, false>(ctx, v, kact, loop);
}

int solve_load(globe_ctx* ctx, const SolveVecs& v, const double* in, void* out) {
    const int64_t n = ctx->coh.Nrec;
    const dim3 grid((unsigned)div_up(n, CV_R), (unsigned)div_up(v.k, CV_C));
    if (v.df) k_to_rows<ArithDF><<<grid, CV_R, 0, ctx->stream>>>(in, n, v.k, v.unsc, (float2*)out);
    else k_to_rows<ArithF64><<<grid, CV_R, 0, ctx->stream>>>(in, n, v.k, nullptr, (double*)out);
    GLOBE_LAUNCHED(ctx, "k_to_rows");
    return GLOBE_OK;
}
int solve_store(globe_ctx* ctx, const SolveVecs& v, bool pending, double* out) {
    const int64_t n = ctx->coh.Nrec;
    const dim3 grid((unsigned)div_up(n, CV_R), (unsigned)div_up(v.k, CV_C));
    const void* al = pending ? v.alpha : nullptr;
    if (v.df)
        k_from_rows<ArithDF><<<grid, CV_R, 0, ctx->stream>>>((const float2*)v.x, (const float2*)v.p, (const float2*)al, n, v.k, v.unsc, out);
    else
        k_from_rows<ArithF64><<<grid, CV_R, 0, ctx->stream>>>((const double*)v.x, (const double*)v.p, (const double*)al, n, v.k, nullptr, out);
    GLOBE_LAUNCHED(ctx, "k_from_rows");
    return GLOBE_OK;
}

}  // namespace globe
