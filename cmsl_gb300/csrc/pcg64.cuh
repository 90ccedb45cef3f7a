// pcg64.cuh -- the FP64 Jacobi-PCG of the depolarisation solve as one
// persistent cooperative kernel.
//
// The reference's algorithm and stop test (depol_varEPS.cu:458-523: two dot
// products an iteration, z = D^-1 r), every iteration of every film of the
// handle inside one launch.  Per iteration:
//   S: p = z + beta p, q = A p, p.q          all-reduce -> alpha
//   U: x += alpha p, r -= alpha q, z = D^-1 r, r.z (r.r)   all-reduce -> beta
//
// What bounds it.  This part executes FP64 at 2 FMA per clock and SM: one
// warp instruction holds the SM's FP64 pipe for 16 cycles, so a film of many
// cells is bound by the number of FP64 instructions per cell, and a small one
// by the latency of the two all-reduces.
//   * FP64 instructions.  A row is q_c = D_c p_c - sum_f e_f p_f with the face
//     permittivities and the diagonal (all over h^2) looked up in shared
//     memory by a per-cell operator word: 7 FP64 instructions whatever the
//     permittivities (the flux form e_f (p_f - p_c) and the division by h^2
//     took about 30).  p is one FMA; a warp owns R rows of 32 cells and marches
//     through z, so a y or z neighbour's p is formed once for all the rows that
//     read it, x neighbours come by shuffle, and the two x halo cells of all R
//     rows are formed together by one packed FMA.  Update: 4 (5 with r.r).
//     About 15 per cell and iteration, from about 45.
//   * No barrier inside S: warps are independent, with the next plane's loads
//     in flight while one is computed.
//   * All-reduce: every block adds its sums to the film's words as fixed-point
//     integers (FxRed) and waits until the words count every block; all blocks
//     then hold the same scalars and take the same decisions.  152 blocks, one
//     value: 3.6 k cycles; with FP64 trees over partials behind an arrival
//     counter 6.6 k, with per-block slots that every block polls 8.3 k.  Films
//     synchronise only their own blocks: one that has converged leaves, the
//     others go on.
//   * Films small enough keep every vector in registers (k_pcg64r): 64x64x16
//     10.6 -> 6.4 us an iteration, 96x80x20 13.3 -> 8.5, 128x128x16 15.4 -> 13.0
//     (with fixed alpha and beta; their two quotients and the check for a second
//     all-reduce add 0.5).
// One iteration, two kernels in a graph loop before and one launch now:
// 64x64x16 43 -> 6.9 us, 256x256x32 with three permittivities 190 -> 71 us
// (about 15.3 FP64 instructions a cell at the measured 19 cycles each and SM
// are 61 us).
//
// Waits are bounded (Pcg64::spin_limit); a wait that gives up records an error
// and its block leaves.  Where the film's first block leaves so, the solve's
// status is SOLVE_WAIT; where only others do, they gave up on sums that the
// first block still received, and the solve it reports is complete or ends on
// a wait of its own for theirs.
#pragma once
#include "kernels.cuh"

namespace cmsl {

constexpr int P64_NT = 256;
constexpr int P64_NW = P64_NT / 32;
constexpr int P64_BPS = 2;                  // resident blocks per SM at most
constexpr int P64_MAX_BLOCKS = 500;         // blocks of one film at most (the counts of FxRed)
constexpr unsigned long long P64_SPIN_LIMIT = 1500000ull;   // polls of a wait (about 0.7 us each) before it gives up
constexpr int P64_NDIAG = 85;               // 3 materials x 28 neighbour counts, identity

struct Pcg64 {
    const uint32_t *op;         // operator word per cell (k_op64)
    double *z;                  // D^-1 r
    unsigned long long *words;  // [n_films][P64_WORDS] the all-reduces' sums (zeroed by start_solves)
    const int *blk_film;        // film of each block
    int *err;                   // timeout flag
    unsigned long long spin_limit;
    int hold_block;             // failure injection: this block never publishes its sums (-1: none)
};

// Operator word of a cell: six nibbles (faces e, w, n, s, u, d) index the face
// table mat_c * 3 + mat_f (9: no face), bits 24-31 the diagonal table.
// Identity rows (Dirichlet planes, Neumann pin): diagonal 1, no faces.
__host__ __device__ inline int p64_diag_index(int mc, int n0, int n1)   // neighbours of material 0 and 1
{
    return mc * 28 + n0 * 7 - n0 * (n0 - 1) / 2 + n1;
}

static __global__ void k_op64(Dev d, uint32_t *op)
{
    const int4 it = d.items[blockIdx.x];
    const FilmDev *f = d.films + it.x;
    const int z0 = it.w & 0xffff, z1 = it.w >> 16;
    const Geom g = make_geom(f, it.y, it.z);
    if (!g.valid) return;
    const int lx = threadIdx.x % TX, ly = threadIdx.x / TX;
    const int i = g.x0 + lx, j = g.y0 + ly, nx = g.nx, ny = g.ny, nz = g.nz;
    const uint32_t *code = d.code + f->off;
    auto mt = [&](int a, int b, int c) { return code_mat(code[a + (long long)nx * (b + (long long)ny * c)]); };
    for (int k = z0; k < z1; ++k) {
        uint32_t w = 84u << 24 | 0x999999u;
        if (!identity_row(f, k, g.own_pl)) {
            int up = k + 1, dn = k - 1;
            if (f->zbc != 0) {
                if (k == 0) dn = 1;
                else if (k == nz - 1) up = nz - 2;
            }
            const int mc = mt(i, j, k);
            const int mf[6] = {mt((i + 1) % nx, j, k), mt((i - 1 + nx) % nx, j, k), mt(i, (j + 1) % ny, k),
                               mt(i, (j - 1 + ny) % ny, k), mt(i, j, up), mt(i, j, dn)};
            int n0 = 0, n1 = 0;
            w = 0u;
            for (int q = 0; q < 6; ++q) {
                w |= (uint32_t)(mc * 3 + mf[q]) << (4 * q);
                n0 += mf[q] == 0;
                n1 += mf[q] == 1;
            }
            w |= (uint32_t)p64_diag_index(mc, n0, n1) << 24;
        }
        op[f->off + g.own_pl + (long long)k * g.plane] = w;
    }
}

// Fixed-point sums.  A dependent FP64 add takes about 150 cycles here, so the
// trees of a block sum and of the sum over the blocks (17 dependent adds) took
// half of an all-reduce.  A thread's double is cut into six signed 23-bit
// pieces of a 138-bit integer in units of 2^E, 2^-100 of a reference value
// (the current r.z or r.r): the sum is exact in those units and independent of
// the order, and the pieces add with the warps' integer reduction.  The block
// carries them into three words (46 bits each, the top one signed) and adds
// each to the film's word with one 64-bit atomic.  A word counts the blocks
// from bit 55 on, so a completed count delivers the sum with the same load.
// A value that is not finite, or 2^17 above the reference in one thread, puts
// FX_BAD into the top word, far above what sound blocks can sum to; the blocks,
// which all see it, then sum once more in units of 2^-40 of the reference (r.z
// jumps by 2^20 and more where permittivities differ by 1e8), and only a value
// outside those as well (2^77 above, or not finite) makes the total NaN.
constexpr int FX_PIECES = 6, FX_BITS = 23, FX_WORDS = 3;
constexpr int FX_COUNT = 55;                        // first bit of the block count
constexpr long long FX_BIAS = 1ll << 44;            // keeps the top word's payload positive
constexpr long long FX_BAD = 1ll << 43;             // sound: |top word| <= 2^33 a block, 2^42 in all
constexpr int FX_COARSE = 60;                       // the second attempt's units over the first's, as a power of two

__device__ __forceinline__ int fx_exponent(double ref)
{
    return max((int)((__double2hiint(ref) >> 20) & 0x7ff) - 1023 - 100, -1074);     // 2^-1074: the least double
}
__device__ __forceinline__ void fx_split(double v, int E, int (&p)[FX_PIECES], bool &bad)
{
    const long long b = __double_as_longlong(v);
    int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    const int sh = (e ? e : 1) - 1075 - E;      // m 2^sh units
    bad = bad || e == 0x7ff || (sh > 64 && m != 0ull);
    #pragma unroll
    for (int i = 0; i < FX_PIECES; ++i) {
        const int t = FX_BITS * i - sh;
        const unsigned long long w = t >= 0 ? (t < 64 ? m >> t : 0ull) : (t > -FX_BITS ? m << -t : 0ull);
        const int q = (int)(w & ((1u << FX_BITS) - 1u));
        p[i] = b < 0 ? -q : q;
    }
}
// (lo + 2^46 mid + 2^92 hi) 2^E rounded to a double, by integer operations
// (lo, mid >= 0): the leading 64 bits are converted, the bits below them cut.
__device__ __forceinline__ double fx_double(long long lo, long long mid, long long hi, int E)
{
    constexpr int B = 2 * FX_BITS;
    mid += lo >> B;
    lo &= (1ll << B) - 1ll;
    hi += mid >> B;
    mid &= (1ll << B) - 1ll;
    const bool neg = hi < 0;
    unsigned long long w0 = (unsigned long long)lo | ((unsigned long long)mid << B);
    unsigned long long w1 = ((unsigned long long)mid >> (64 - B)) | ((unsigned long long)hi << (2 * B - 64));
    unsigned long long w2 = (unsigned long long)(hi >> (128 - 2 * B));
    if (neg) {
        w0 = ~w0 + 1ull;
        w1 = ~w1 + (w0 == 0ull);
        w2 = ~w2 + (w0 == 0ull && w1 == 0ull);
    }
    int e = E;
    if (w2) e += 128;
    else if (w1) { e += 64; w2 = w1; w1 = w0; }
    else { w2 = w0; w1 = 0ull; }
    if (w2 == 0ull) return 0.0;
    const int lz = __clzll((long long)w2);
    const unsigned long long m = lz ? (w2 << lz) | (w1 >> (64 - lz)) : w2;
    const double v = __ull2double_rn(m);            // in [2^63, 2^64]
    const int k = e - lz, be = (__double2hiint(v) >> 20) + k;
    // the exponent moved by an integer addition where the result is a normal number
    const double s = be >= 1 && be <= 2046 ? __hiloint2double(__double2hiint(v) + k * (1 << 20), __double2loint(v)) : ldexp(v, k);
    return neg ? -s : s;
}

// A film's sums over its nb blocks: two sets of words used in turn, whose
// totals only grow (prev: this lane's word at the set's last use).  A set is
// added to again only when every block has read it: the all-reduce between
// needs that block's arrival.
struct FxRed {
    unsigned long long *words;      // the film's [2 sets][P64_WORDS / 2]: [2 values][3 words] (packed: words on
                                    // lines of their own, or several copies of each, measured no faster)
    unsigned long long prev[2];
    int par;
};
struct FxShared {
    int p[P64_NW][2 * FX_PIECES];
    int bad[P64_NW];
};

// Sums v over the film's blocks, ref: reference values.  tot valid in warp 0
// of every block, the same bits everywhere (all NaN where a value was bad).
// False in warp 0 after a timeout.  Every thread of the block calls it; the
// caller's __syncthreads after warp 0's scalar step publishes the outcome.
// FENCE: the blocks' stores before the call are visible to loads after it
// (about 600 cycles; not needed where only the sums cross blocks).
// COARSE: 0, or FX_COARSE for a second attempt.
template <int NV, bool FENCE, int COARSE = 0>
__device__ __forceinline__ bool p64_allreduce(const Pcg64 &B, FxRed &R, int nb, FxShared &sm, const double (&v)[NV],
                                              const double (&ref)[NV], double (&tot)[NV])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool bad = false;
    int mine = 0;                               // lane 6 i + j: piece j of value i
    #pragma unroll
    for (int i = 0; i < NV; ++i) {
        int p[FX_PIECES];
        fx_split(v[i], fx_exponent(ref[i]) + COARSE, p, bad);
        #pragma unroll
        for (int j = 0; j < FX_PIECES; ++j) {
            const int s = __reduce_add_sync(0xffffffffu, p[j]);
            if (lane == i * FX_PIECES + j) mine = s;
        }
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane < NV * FX_PIECES) sm.p[warp][lane] = mine;
    if (lane == 0) sm.bad[warp] = bad;
    R.par ^= 1;
    __syncthreads();
    if (warp != 0) return true;
    bad = __any_sync(0xffffffffu, lane < P64_NW && sm.bad[lane < P64_NW ? lane : 0] != 0);
    long long ps = 0;
    if (lane < NV * FX_PIECES) {
        #pragma unroll
        for (int q = 0; q < P64_NW; ++q) ps += sm.p[q][lane];
    }
    // lane 3 i + j: word j of value i
    const bool own = lane < FX_WORDS * NV;
    const int vi = own ? lane / FX_WORDS : 0, wi = lane % FX_WORDS;
    long long a = 0;
    {
        long long c[FX_PIECES];
        #pragma unroll
        for (int j = 0; j < FX_PIECES; ++j) c[j] = __shfl_sync(0xffffffffu, ps, vi * FX_PIECES + j);
        #pragma unroll
        for (int j = 0; j + 1 < FX_PIECES; ++j) {
            c[j + 1] += c[j] >> FX_BITS;
            c[j] &= (1ll << FX_BITS) - 1ll;
        }
        a = wi == 0 ? (c[1] << FX_BITS) + c[0] : wi == 1 ? (c[3] << FX_BITS) + c[2]
                                                         : (bad ? FX_BAD : (c[5] << FX_BITS) + c[4]) + FX_BIAS;
    }
    unsigned long long *word = R.words + R.par * (P64_WORDS / 2) + vi * FX_WORDS + wi;
    unsigned long long w = 0ull, diff = 0ull;
    if (FENCE) __threadfence();                 // with the block's stores, ordered before by the barrier above
    if (own && (int)blockIdx.x != B.hold_block) {
        const unsigned long long u = (1ull << FX_COUNT) + (unsigned long long)a;
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(u) : "memory");
    }
    const unsigned long long before = R.par ? R.prev[1] : R.prev[0];
    unsigned long long spins = 0;
    for (;;) {
        bool ok = true;
        if (own) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(word) : "memory");
            diff = w - before;
            ok = (diff >> FX_COUNT) == (unsigned long long)nb;
        }
        if (__all_sync(0xffffffffu, ok)) break;
        if (++spins > B.spin_limit) {
            if (lane == 0) atomicExch(B.err, 1);
            return false;
        }
    }
    if (FENCE) __threadfence();
    if (own) {                                  // the words of values this call did not sum stay as they were
        if (R.par) R.prev[1] = w;
        else R.prev[0] = w;
    }
    const long long pv = (long long)(diff & ((1ull << FX_COUNT) - 1ull)) - (wi == 2 ? nb * FX_BIAS : 0ll);
    #pragma unroll
    for (int i = 0; i < NV; ++i) {
        const long long lo = __shfl_sync(0xffffffffu, pv, i * FX_WORDS), mid = __shfl_sync(0xffffffffu, pv, i * FX_WORDS + 1);
        const long long hi = __shfl_sync(0xffffffffu, pv, i * FX_WORDS + 2);
        tot[i] = hi >= FX_BAD / 2 ? __longlong_as_double(0x7ff8000000000000ll) : fx_double(lo, mid, hi, fx_exponent(ref[i]) + COARSE);
    }
    return true;
}

// The scalars of a film's solve, the same in every block (thread 0 steps them).
struct P64Scal {
    double alpha, beta, rz, rr;
    int go;                     // 1 go on, 2 sum again in coarse units, 0 done, -1 timeout, -2 breakdown
    int ok;                     // p64_again: the second attempt's outcome
    double tot[2];              // and its totals
};

// The second attempt of an all-reduce after which the solve would end as a
// breakdown, out of line: it costs 64x64x16 0.15 us an iteration where a loop
// around the first attempt cost 0.34.  The outcome goes to sc (valid in thread
// 0); returns the words' last totals.
template <int NV>
__device__ __noinline__ ulonglong2 p64_again(FxRed R, int nb, int *err, unsigned long long spin_limit, int hold_block,
                                             FxShared *sm, P64Scal *sc, double v0, double v1, double ref0, double ref1)
{
    Pcg64 B{};
    B.err = err;
    B.spin_limit = spin_limit;
    B.hold_block = hold_block;
    double v[NV], ref[NV], tot[NV];
    v[0] = v0;
    ref[0] = ref0;
    if (NV == 2) { v[NV - 1] = v1; ref[NV - 1] = ref1; }
    const bool ok = p64_allreduce<NV, true, FX_COARSE>(B, R, nb, *sm, v, ref, tot);
    if (threadIdx.x == 0) {
        sc->ok = ok;
        sc->tot[0] = tot[0];
        sc->tot[1] = tot[NV - 1];
    }
    return make_ulonglong2(R.prev[0], R.prev[1]);
}
template <int NV>
__device__ __forceinline__ void p64_second(const Pcg64 &B, FxRed &R, int nb, FxShared &sm, P64Scal &sc, double v0, double v1,
                                           double ref0, double ref1)
{
    const ulonglong2 p = p64_again<NV>(R, nb, B.err, B.spin_limit, B.hold_block, &sm, &sc, v0, v1, ref0, ref1);
    R.prev[0] = p.x;
    R.prev[1] = p.y;
    R.par ^= 1;
}

// After S (thread 0): alpha, or the breakdown of depol_varEPS.cu:486-490 (bad:
// 2 after a first attempt, -2 after a second).
__device__ __forceinline__ void p64_after_s(P64Scal &s, bool ok, double pq, bool force, int bad)
{
    const bool good = ok && isfinite(pq) && pq > 0.0;
    s.go = !ok ? -1 : good || force ? 1 : bad;
    s.alpha = force ? 1e-3 : s.rz / pq;
}
// After U (thread 0): beta and the stop test (depol_varEPS.cu:508-521, :472-474).
__device__ __forceinline__ void p64_after_u(P64Scal &s, const FilmDev *f, bool ok, double rzn, double rrn, int iters,
                                            int max_iter, double rz0, double bb, bool force, int bad)
{
    if (!ok) s.go = -1;
    else if (force) s.go = iters < max_iter;
    else if (!isfinite(rzn) || rzn < 0.0) {
        s.go = bad;
        if (bad == 2) return;           // r.z and r.r of the last iteration stay
    }
    else if (f->crit == 0) s.go = iters < max_iter && rzn > f->tol_abs2 && (rz0 <= 0.0 || rzn / rz0 > f->tol_rel2);
    else s.go = iters < max_iter && rrn > f->tol_rel2 * bb;
    s.beta = force ? 0.5 : rzn / s.rz;
    s.rz = rzn;
    s.rr = rrn;
}

struct P64Tables {
    double e[16], d[P64_NDIAG], v[P64_NDIAG];       // -face permittivity / h^2, diagonal, its inverse
};
__device__ __forceinline__ void p64_tables(P64Tables &T, const FilmDev *f)
{
    if (threadIdx.x < 16) T.e[threadIdx.x] = threadIdx.x < 9 ? -(f->epsf[threadIdx.x] / f->h2) : 0.0;
    if (threadIdx.x < P64_NDIAG) {
        double v = 1.0;
        if (threadIdx.x < 84) {
            const int mc = threadIdx.x / 28;
            int c = threadIdx.x % 28, n0 = 0;
            while (c >= 7 - n0) { c -= 7 - n0; ++n0; }
            const int n1 = c, n2 = 6 - n0 - n1;
            v = (n0 * f->epsf[mc * 3] + n1 * f->epsf[mc * 3 + 1] + n2 * f->epsf[mc * 3 + 2]) / f->h2;
        }
        T.d[threadIdx.x] = v;
        T.v[threadIdx.x] = v > 1e-30 ? 1.0 / v : 1.0;       // depol_varEPS.cu:177-179
    }
}

// The film's solve is over (one thread of its first block).
__device__ __forceinline__ void p64_done(SolveDev *S, const P64Scal &s, int iters)
{
    S->iters = iters;
    S->total_iters += iters;
    S->rz = s.rz;
    S->rr = s.rr;
    S->active = 0;
    if (s.go < 0) {
        S->status = s.go == -2 ? 1 : SOLVE_WAIT;
        S->outer_active = 0;
    }
}

// One row of q = A p from a cell's value, its six neighbours and its operator word.
__device__ __forceinline__ double p64_row(const P64Tables &T, uint32_t w, double c, double xe, double xw, double yn,
                                          double ys, double zu, double zd)
{
    double v = T.d[w >> 24] * c;
    v = fma(T.e[w & 15u], xe, v);
    v = fma(T.e[(w >> 4) & 15u], xw, v);
    v = fma(T.e[(w >> 8) & 15u], yn, v);
    v = fma(T.e[(w >> 12) & 15u], ys, v);
    v = fma(T.e[(w >> 16) & 15u], zu, v);
    return fma(T.e[(w >> 20) & 15u], zd, v);
}

struct P64Geom {
    int nx, ny, nz, plane, xt, nc;
    bool neu;
};

// Phase S over the film's units (R rows x 32 cells x one z chunk), one unit a
// warp: p and q written, p.q accumulated.  s, t select the direction's update
// from two loaded values a, b: p = beta b + a (a = z, b = the old p), on the
// first iteration p = a b (a = r, b = D^-1).
// Lanes past the row's end take the row's start (periodic), so the lane after
// the last cell is its east neighbour, and likewise the rows of a last group.
template <int R>
__device__ __forceinline__ void p64_spmv(const P64Geom &G, const double *__restrict__ A, const double *__restrict__ Bv,
                                         double *__restrict__ pn, double *__restrict__ q,
                                         const uint32_t *__restrict__ op, bool first, double beta, int w0, int nw,
                                         const P64Tables &T, double &acc)
{
    const int lane = threadIdx.x & 31;
    const int nx = G.nx, ny = G.ny, nz = G.nz, yt = (ny + R - 1) / R;
    const int units = G.xt * yt * G.nc;
    auto dir = [&](double a, double b) { return fma(first ? a : beta, b, first ? 0.0 : a); };
    auto zmap = [&](int k) { return k < 0 ? (G.neu ? 1 : 0) : k >= nz ? (G.neu ? nz - 2 : nz - 1) : k; };
    for (int u = w0; u < units; u += nw) {
        const int xq = u % G.xt, t = u / G.xt, yq = t % yt, zq = t / yt;
        const int x0 = xq * 32, y0 = yq * R;
        const int z0 = (int)((long long)zq * nz / G.nc), z1 = (int)((long long)(zq + 1) * nz / G.nc);
        const int x = (x0 + lane) % nx;
        int ro[R];
        #pragma unroll
        for (int r = 0; r < R; ++r) ro[r] = ((y0 + r) % ny) * nx + x;
        const int hs = ((y0 - 1 + ny) % ny) * nx + x, hn = ((y0 + R) % ny) * nx + x;
        const int hr = (lane & 15) < R ? (lane & 15) : 0;
        const int hx = ((y0 + hr) % ny) * nx + ((lane & 16) ? (x0 + 32) % nx : (x0 - 1 + nx) % nx);
        double pd[R], pc[R], na[R], nb[R], ha[3], hb[3];
        uint32_t on[R];
        {
            const long long od = (long long)zmap(z0 - 1) * G.plane, oc = (long long)z0 * G.plane;
            const long long ou = (long long)zmap(z0 + 1) * G.plane;
            double a0[R], b0[R], a1[R], b1[R];
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                a0[r] = A[od + ro[r]]; b0[r] = Bv[od + ro[r]];
                a1[r] = A[oc + ro[r]]; b1[r] = Bv[oc + ro[r]];
                na[r] = A[ou + ro[r]]; nb[r] = Bv[ou + ro[r]];
                on[r] = op[oc + ro[r]];
            }
            ha[0] = A[oc + hs]; hb[0] = Bv[oc + hs];
            ha[1] = A[oc + hn]; hb[1] = Bv[oc + hn];
            ha[2] = A[oc + hx]; hb[2] = Bv[oc + hx];
            #pragma unroll
            for (int r = 0; r < R; ++r) { pd[r] = dir(a0[r], b0[r]); pc[r] = dir(a1[r], b1[r]); }
        }
        for (int k = z0; k < z1; ++k) {
            double pu[R];
            uint32_t o[R];
            #pragma unroll
            for (int r = 0; r < R; ++r) { pu[r] = dir(na[r], nb[r]); o[r] = on[r]; }
            const double ps = dir(ha[0], hb[0]), pnn = dir(ha[1], hb[1]), px = dir(ha[2], hb[2]);
            if (k + 1 < z1) {
                const long long o1 = (long long)(k + 1) * G.plane, o2 = (long long)zmap(k + 2) * G.plane;
                #pragma unroll
                for (int r = 0; r < R; ++r) {
                    na[r] = A[o2 + ro[r]]; nb[r] = Bv[o2 + ro[r]];
                    on[r] = op[o1 + ro[r]];
                }
                ha[0] = A[o1 + hs]; hb[0] = Bv[o1 + hs];
                ha[1] = A[o1 + hn]; hb[1] = Bv[o1 + hn];
                ha[2] = A[o1 + hx]; hb[2] = Bv[o1 + hx];
            }
            const long long oc = (long long)k * G.plane;
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                const double c = pc[r];
                double xe = __shfl_down_sync(0xffffffffu, c, 1), xw = __shfl_up_sync(0xffffffffu, c, 1);
                const double he = __shfl_sync(0xffffffffu, px, 16 + r), hw = __shfl_sync(0xffffffffu, px, r);
                if (lane == 31) xe = he;
                if (lane == 0) xw = hw;
                const double yn = r + 1 < R ? pc[r + 1 < R ? r + 1 : r] : pnn, ys = r > 0 ? pc[r > 0 ? r - 1 : r] : ps;
                const uint32_t w = o[r];
                const double v = p64_row(T, w, c, xe, xw, yn, ys, pu[r], pd[r]);
                if (x0 + lane < nx && y0 + r < ny) {
                    pn[oc + ro[r]] = c;
                    q[oc + ro[r]] = v;
                    acc = fma(c, v, acc);
                }
            }
            #pragma unroll
            for (int r = 0; r < R; ++r) { pd[r] = pc[r]; pc[r] = pu[r]; }
        }
    }
}

// Phase U over the film's n cells (16-byte aligned), pairs of cells a lane.
__device__ __forceinline__ void p64_update(long long n, long long t0, long long stride, double *__restrict__ x,
                                           const double *__restrict__ p, double *__restrict__ r,
                                           const double *__restrict__ q, const double *__restrict__ dinv,
                                           double *__restrict__ z, double alpha, bool want_rr, double &rz, double &rr)
{
    constexpr int U = 2;
    const long long n2 = n >> 1;
    auto cell = [&](double &xv, double &rv, double pv, double qv, double dv) {
        xv = fma(alpha, pv, xv);
        rv = fma(-alpha, qv, rv);
        const double zv = rv * dv;
        rz = fma(rv, zv, rz);
        if (want_rr) rr = fma(rv, rv, rr);
        return zv;
    };
    for (long long i = t0; i < n2; i += U * stride) {
        double2 xv[U], pv[U], rv[U], qv[U], dv[U];
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long c = i + u * stride;
            if (c < n2) {
                xv[u] = ((const double2 *)x)[c]; pv[u] = ((const double2 *)p)[c]; rv[u] = ((const double2 *)r)[c];
                qv[u] = ((const double2 *)q)[c]; dv[u] = ((const double2 *)dinv)[c];
            }
        }
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long c = i + u * stride;
            if (c < n2) {
                double2 zv;
                zv.x = cell(xv[u].x, rv[u].x, pv[u].x, qv[u].x, dv[u].x);
                zv.y = cell(xv[u].y, rv[u].y, pv[u].y, qv[u].y, dv[u].y);
                ((double2 *)x)[c] = xv[u];
                ((double2 *)r)[c] = rv[u];
                ((double2 *)z)[c] = zv;
            }
        }
    }
    if ((n & 1) && t0 == 0) {
        const long long c = n - 1;
        double xv = x[c], rv = r[c];
        z[c] = cell(xv, rv, p[c], q[c], dinv[c]);
        x[c] = xv;
        r[c] = rv;
    }
}

// The solve of every active film, from r and the scalars the set-up kernel
// left (start_solves).  With Dev::step_end the last block ends the step.
// Streaming form: the vectors live in memory, every warp takes the units that
// fall to it.
static __global__ void __launch_bounds__(P64_NT, P64_BPS) k_pcg64(Dev d, Fields<double> F, Pcg64 B)
{
    __shared__ FxShared sm;
    __shared__ P64Tables T;
    __shared__ P64Scal sc;
    const int fi = B.blk_film[blockIdx.x];
    const FilmDev *f = d.films + fi;
    SolveDev *S = d.solve + fi;
    const int b0 = f->pb_begin, lb = (int)blockIdx.x - b0, nb = f->pb_end - b0;
    if (threadIdx.x == 0) {
        sc.go = d.force || *(volatile const int *)&S->active != 0;
        sc.rz = S->rz;
        sc.rr = S->rr;
    }
    p64_tables(T, f);
    __syncthreads();
    if (sc.go) {
        P64Geom G;
        G.nx = f->nx; G.ny = f->ny; G.nz = f->nz; G.plane = f->nx * f->ny; G.xt = (f->nx + 31) / 32; G.nc = f->p64_nc;
        G.neu = f->zbc != 0;
        const int R = f->p64_rows;
        const bool want_rr = f->crit != 0;
        const long long off = f->off, n = (long long)G.plane * G.nz;
        double *x = phi_sel(d, S->phi_cur) + off, *r = F.r + off, *z = B.z + off, *q = F.q + off;
        const double *dinv = F.dinv + off;
        const uint32_t *op = B.op + off;
        const int nw = nb * P64_NW, w0 = (threadIdx.x >> 5) * nb + lb;   // a block's warps spread over the film
        FxRed red{B.words + (size_t)P64_WORDS * fi, {0ull, 0ull}, 0};
        const double rz0 = S->rz0, bb = S->bb;
        const int max_iter = d.force ? S->inner_max : f->max_iter;
        int iters = 0;
        for (;;) {
            const bool first = iters == 0;
            const double *po = F.p[iters & 1] + off;
            double *pn = F.p[(iters & 1) ^ 1] + off;
            const double *A = first ? r : z, *Bv = first ? dinv : po;
            double acc[1] = {0.0}, pq[1];
            const double ref1[1] = {sc.rz};
            const double beta = first ? 0.0 : sc.beta;
            if (R == 4) p64_spmv<4>(G, A, Bv, pn, q, op, first, beta, w0, nw, T, acc[0]);
            else if (R == 2) p64_spmv<2>(G, A, Bv, pn, q, op, first, beta, w0, nw, T, acc[0]);
            else p64_spmv<1>(G, A, Bv, pn, q, op, first, beta, w0, nw, T, acc[0]);
            bool ok = p64_allreduce<1, true>(B, red, nb, sm, acc, ref1, pq);
            if (threadIdx.x == 0) p64_after_s(sc, ok, pq[0], d.force != 0, 2);
            __syncthreads();
            if (sc.go != 1) {
                if (sc.go == 2) {
                    p64_second<1>(B, red, nb, sm, sc, acc[0], 0.0, sc.rz, 0.0);
                    if (threadIdx.x == 0) p64_after_s(sc, sc.ok != 0, sc.tot[0], d.force != 0, -2);
                    __syncthreads();
                }
                if (sc.go <= 0) break;
            }
            double a2[2] = {0.0, 0.0}, tot[2];
            const double ref2[2] = {sc.rz, sc.rr};
            p64_update(n, (long long)lb * P64_NT + threadIdx.x, (long long)nb * P64_NT, x, pn, r, q, dinv, z, sc.alpha,
                       want_rr, a2[0], a2[1]);
            ok = p64_allreduce<2, true>(B, red, nb, sm, a2, ref2, tot);
            ++iters;
            if (threadIdx.x == 0) p64_after_u(sc, f, ok, tot[0], tot[1], iters, max_iter, rz0, bb, d.force != 0, 2);
            __syncthreads();
            if (sc.go != 1) {
                if (sc.go == 2) {
                    p64_second<2>(B, red, nb, sm, sc, a2[0], a2[1], sc.rz, sc.rr);
                    if (threadIdx.x == 0)
                        p64_after_u(sc, f, sc.ok != 0, sc.tot[0], sc.tot[1], iters, max_iter, rz0, bb, d.force != 0, -2);
                    __syncthreads();
                }
                if (sc.go <= 0) break;
            }
        }
        if (lb == 0 && threadIdx.x == 0 && !d.force) p64_done(S, sc, iters);
    }
    if (!d.step_end) return;
    if (!ticket_last(d.counter)) return;
    if (threadIdx.x == 0) *d.counter = 0u;
    step_end(d);
}

// Resident form, for films of at most one unit of R rows x 32 cells x ZC
// planes a warp: x, r, p, q and the halo's p stay in registers for the whole
// solve, and only z crosses warps (every warp stores its cells' z and reads
// its halo's, from which it forms the halo's p itself).  One block per SM.
template <int R, int ZC>
__device__ __forceinline__ void p64_resident(const Dev &d, const Fields<double> &F, const Pcg64 &B, const FilmDev *f,
                                             SolveDev *S, int fi, int lb, int nb, FxShared &sm, const P64Tables &T,
                                             P64Scal &sc)
{
    const int lane = threadIdx.x & 31;
    const int nx = f->nx, ny = f->ny, nz = f->nz, plane = nx * ny;
    const bool neu = f->zbc != 0, want_rr = f->crit != 0;
    const long long off = f->off;
    double *xg = phi_sel(d, S->phi_cur) + off, *rg = F.r + off, *zg = B.z + off;
    const int xt = (nx + 31) / 32, yt = (ny + R - 1) / R, zt = (nz + ZC - 1) / ZC;
    const int unit = (threadIdx.x >> 5) * nb + lb;          // a block's warps spread over the film
    const bool has = unit < xt * yt * zt;
    const int u = has ? unit : 0;
    const int xq = u % xt, t = u / xt, y0 = (t % yt) * R, z0 = (t / yt) * ZC, x0 = xq * 32;
    const int xl = (x0 + lane) % nx;
    int row[R];
    #pragma unroll
    for (int r = 0; r < R; ++r) row[r] = ((y0 + r) % ny) * nx + xl;
    const int hs = ((y0 - 1 + ny) % ny) * nx + xl, hn = ((y0 + R) % ny) * nx + xl;
    const int hr = (lane & 15) < R ? (lane & 15) : 0;
    const int hx = ((y0 + hr) % ny) * nx + ((lane & 16) ? (x0 + 32) % nx : (x0 - 1 + nx) % nx);
    int pl[ZC];                                             // plane offsets (the last chunk's clamped)
    #pragma unroll
    for (int c = 0; c < ZC; ++c) pl[c] = min(z0 + c, nz - 1) * plane;
    const int plb = max(z0 - 1, 0) * plane, plt = min(z0 + ZC, nz - 1) * plane;
    const bool vx = has && x0 + lane < nx;
    double x[R][ZC], r[R][ZC], p[R][ZC], q[R][ZC];
    double hps[ZC], hpn[ZC], hpx[ZC], hpb[R], hpt[R];
    uint32_t op[R][ZC];
    {
        const double *dv = F.dinv + off;
        auto dir = [&](int o) { return rg[o] * dv[o]; };
        #pragma unroll
        for (int c = 0; c < ZC; ++c) {
            #pragma unroll
            for (int a = 0; a < R; ++a) {
                const int o = pl[c] + row[a];
                op[a][c] = B.op[off + o];
                x[a][c] = xg[o];
                r[a][c] = rg[o];
                p[a][c] = dir(o);
            }
            hps[c] = dir(pl[c] + hs);
            hpn[c] = dir(pl[c] + hn);
            hpx[c] = dir(pl[c] + hx);
        }
        #pragma unroll
        for (int a = 0; a < R; ++a) { hpb[a] = dir(plb + row[a]); hpt[a] = dir(plt + row[a]); }
    }
    FxRed red{B.words + (size_t)P64_WORDS * fi, {0ull, 0ull}, 0};
    const double rz0 = S->rz0, bb = S->bb;
    const int max_iter = d.force ? S->inner_max : f->max_iter;
    auto valid = [&](int a, int c) { return vx && y0 + a < ny && z0 + c < nz; };
    int iters = 0;
    for (;;) {
        double acc[1] = {0.0}, pq[1];
        const double ref1[1] = {sc.rz};
        #pragma unroll
        for (int c = 0; c < ZC; ++c) {
            const int k = z0 + c;
            #pragma unroll
            for (int a = 0; a < R; ++a) {
                const double v = p[a][c];
                double xe = __shfl_down_sync(0xffffffffu, v, 1), xw = __shfl_up_sync(0xffffffffu, v, 1);
                const double he = __shfl_sync(0xffffffffu, hpx[c], 16 + a), hw = __shfl_sync(0xffffffffu, hpx[c], a);
                if (lane == 31) xe = he;
                if (lane == 0) xw = hw;
                const double yn = a + 1 < R ? p[a + 1 < R ? a + 1 : a][c] : hpn[c];
                const double ys = a > 0 ? p[a > 0 ? a - 1 : a][c] : hps[c];
                double zu = c + 1 < ZC ? p[a][c + 1 < ZC ? c + 1 : c] : hpt[a];
                double zd = c > 0 ? p[a][c > 0 ? c - 1 : c] : hpb[a];
                if (neu) {                      // mirrored end planes (depol_varEPS.cu:86-99)
                    if (k == nz - 1) zu = zd;
                    else if (k == 0) zd = zu;
                }
                q[a][c] = p64_row(T, op[a][c], v, xe, xw, yn, ys, zu, zd);
                if (valid(a, c)) acc[0] = fma(v, q[a][c], acc[0]);
            }
        }
        bool ok = p64_allreduce<1, false>(B, red, nb, sm, acc, ref1, pq);
        if (threadIdx.x == 0) p64_after_s(sc, ok, pq[0], d.force != 0, 2);
        __syncthreads();
        if (sc.go != 1) {
            if (sc.go == 2) {
                p64_second<1>(B, red, nb, sm, sc, acc[0], 0.0, sc.rz, 0.0);
                if (threadIdx.x == 0) p64_after_s(sc, sc.ok != 0, sc.tot[0], d.force != 0, -2);
                __syncthreads();
            }
            if (sc.go <= 0) break;
        }
        double a2[2] = {0.0, 0.0}, tot[2];
        const double ref2[2] = {sc.rz, sc.rr}, alpha = sc.alpha;
        #pragma unroll
        for (int c = 0; c < ZC; ++c)
            #pragma unroll
            for (int a = 0; a < R; ++a) {
                x[a][c] = fma(alpha, p[a][c], x[a][c]);
                r[a][c] = fma(-alpha, q[a][c], r[a][c]);
                q[a][c] = r[a][c] * T.v[op[a][c] >> 24];            // z
                if (valid(a, c)) {
                    zg[pl[c] + row[a]] = q[a][c];
                    a2[0] = fma(r[a][c], q[a][c], a2[0]);
                    if (want_rr) a2[1] = fma(r[a][c], r[a][c], a2[1]);
                }
            }
        ok = p64_allreduce<2, true>(B, red, nb, sm, a2, ref2, tot);
        ++iters;
        if (threadIdx.x == 0) p64_after_u(sc, f, ok, tot[0], tot[1], iters, max_iter, rz0, bb, d.force != 0, 2);
        __syncthreads();
        if (sc.go != 1) {
            if (sc.go == 2) {
                p64_second<2>(B, red, nb, sm, sc, a2[0], a2[1], sc.rz, sc.rr);
                if (threadIdx.x == 0)
                    p64_after_u(sc, f, sc.ok != 0, sc.tot[0], sc.tot[1], iters, max_iter, rz0, bb, d.force != 0, -2);
                __syncthreads();
            }
            if (sc.go <= 0) break;
        }
        const double beta = sc.beta;
        double ls[ZC], ln[ZC], lx[ZC], lb2[R], lt[R];
        #pragma unroll
        for (int c = 0; c < ZC; ++c) { ls[c] = zg[pl[c] + hs]; ln[c] = zg[pl[c] + hn]; lx[c] = zg[pl[c] + hx]; }
        #pragma unroll
        for (int a = 0; a < R; ++a) { lb2[a] = zg[plb + row[a]]; lt[a] = zg[plt + row[a]]; }
        #pragma unroll
        for (int c = 0; c < ZC; ++c) {
            #pragma unroll
            for (int a = 0; a < R; ++a) p[a][c] = fma(beta, p[a][c], q[a][c]);
            hps[c] = fma(beta, hps[c], ls[c]);
            hpn[c] = fma(beta, hpn[c], ln[c]);
            hpx[c] = fma(beta, hpx[c], lx[c]);
        }
        #pragma unroll
        for (int a = 0; a < R; ++a) { hpb[a] = fma(beta, hpb[a], lb2[a]); hpt[a] = fma(beta, hpt[a], lt[a]); }
    }
    #pragma unroll
    for (int c = 0; c < ZC; ++c)
        #pragma unroll
        for (int a = 0; a < R; ++a)
            if (valid(a, c)) {
                xg[pl[c] + row[a]] = x[a][c];
                rg[pl[c] + row[a]] = r[a][c];
            }
    if (lb == 0 && threadIdx.x == 0 && !d.force) p64_done(S, sc, iters);
}

static __global__ void __launch_bounds__(P64_NT, 1) k_pcg64r(Dev d, Fields<double> F, Pcg64 B)
{
    __shared__ FxShared sm;
    __shared__ P64Tables T;
    __shared__ P64Scal sc;
    const int fi = B.blk_film[blockIdx.x];
    const FilmDev *f = d.films + fi;
    SolveDev *S = d.solve + fi;
    const int b0 = f->pb_begin, lb = (int)blockIdx.x - b0, nb = f->pb_end - b0;
    if (threadIdx.x == 0) {
        sc.go = d.force || *(volatile const int *)&S->active != 0;
        sc.rz = S->rz;
        sc.rr = S->rr;
    }
    p64_tables(T, f);
    __syncthreads();
    if (sc.go) {
        const int shape = f->p64_rows * 16 + f->p64_nc;
        if (shape == 1 * 16 + 1) p64_resident<1, 1>(d, F, B, f, S, fi, lb, nb, sm, T, sc);
        else if (shape == 1 * 16 + 2) p64_resident<1, 2>(d, F, B, f, S, fi, lb, nb, sm, T, sc);
        else if (shape == 2 * 16 + 2) p64_resident<2, 2>(d, F, B, f, S, fi, lb, nb, sm, T, sc);
        else p64_resident<2, 4>(d, F, B, f, S, fi, lb, nb, sm, T, sc);
    }
    if (!d.step_end) return;
    if (!ticket_last(d.counter)) return;
    if (threadIdx.x == 0) *d.counter = 0u;
    step_end(d);
}

}  // namespace cmsl
