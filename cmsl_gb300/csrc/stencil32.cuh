// stencil32.cuh -- the CMSL_FP32_REFINED stencil passes: the TDGL step and
// the double-float residual pass of the depolarisation solve.
//
// Same work items as the FP64 kernels (a TX x TY column tile of one film
// marching through z0..z1), but every plane of every field a pass reads is
// brought into a ring of NS shared-memory stages by cp.async copies, NS-3
// planes ahead of the plane being computed.  The z neighbours are read from
// the ring as well, so a thread carries no plane-to-plane state beyond its
// partial sums, several blocks share an SM, and each plane costs one barrier.
//
// FP32 storage (CMSL_FP32_REFINED): P is kept as three float2 arrays per set,
// the pairs (Pmx, Pmy), (Pmz, Psx), (Psy, Psz) (pair j at j * ncells float2
// of the set's allocation), and every double-float potential interleaves its
// (hi, lo) halves per cell; a stencil point of a pair is one 8-byte copy and
// one 8-byte shared load.
//
// Each thread owns one cell of the tile and copies it and at most one x/y
// halo cell.  The tile is TX x TYc columns (TYc 4, 8 or 16: 128, 256 or 512
// threads), the autotuner's choice; the blocks take the stencil item list
// (Dev::sitems) of that tile height.  (Pair tiles -- two x-adjacent cells per thread -- execute a
// third fewer instructions but halve the warps an SM holds within the same
// shared memory, and measured slower.)
//
// Ring protocol (identical in both kernels): planes zlo = max(z0-1, 0) ..
// zhi = min(z1, nz-1) are staged, plane p in stage (p - zlo) % NS, one
// commit group per plane (empty groups keep the count uniform across
// threads).  Before computing plane k a thread waits until plane k+1 has
// landed (NS-4 younger groups may still be in flight), the block syncs --
// which also retires every read of plane k-2 -- and plane k+NS-2 is issued
// into that stage.
#pragma once
#include "kernels.cuh"

namespace cmsl {

// FP32 rotation per grain: films of orthonormal rotations keep the third row
// and a pad (one 16-byte load), others 9 values and 3 pads (three).
constexpr int TR32_ROT = 4, TR32_GEN = 12;

// Warm start of a step's first refinement pass (own cell): 0 the previous
// potential a, 1 linear 2a - q, 2 quadratic 3(a - q) + u, 3 cubic
// 4(a + u) - 6q - v, with a, q, u, v the potentials of steps n .. n-3.  In
// double-float: FP32 rounding noise in the start would be amplified by the
// operator's high-frequency end (~12/h^2) well above the smooth truncation
// error, and the first residual would miss the update pass's 1e-4 ||b||.
__device__ __forceinline__ df extrap_phi(int warm, df a, df q, df u, df v)
{
    if (warm == 1) return df_sub(df{2.f * a.h, 2.f * a.l}, q);
    if (warm == 2) return df_add(df_mul_f(df_sub(a, q), 3.f), u);
    if (warm == 3) return df_sub(df_sub(df_mul_f(df_add(a, u), 4.f), df_mul_f(q, 6.f)), v);
    return a;
}

// The extrapolation order a film's next warm start can take: its warm start
// order, lowered while fewer potentials than it needs are valid (after a
// state upload; a state without a potential starts from zero).
__device__ __forceinline__ int warm_order(const FilmDev *f, const SolveDev *S)
{
    return min(f->warm, max(S->hist - 1, 0));
}

// Difference of two double-float potentials rounded to FP32, for E: the hi
// difference of neighbouring values is exact when they lie within a factor
// of two of each other (Sterbenz) and one FP32 rounding off otherwise; the
// lo difference is added.  E enters the FP32 step, which rounds at that
// level anyway.
__device__ __forceinline__ float phi_diff32(df a, df b) { return (a.h - b.h) + (a.l - b.l); }

// The free one of the five potential buffers of film S.
__device__ __forceinline__ int phi_free(const SolveDev *S)
{
    return 10 - S->phi_cur - S->phi_prev - S->phi_prev2 - S->phi_prev3;
}

// The (hi, lo) pairs of double-float potential buffer i.
__device__ __forceinline__ float2 *phi2_sel(const Dev &d, int i) { return (float2 *)phi_sel(d, i); }
__device__ __forceinline__ df ld_df(const float2 *p)
{
    const float2 v = *p;
    return df{v.x, v.y};
}
// The three P pairs of FP32 set s (pair j at j * ncells).
__device__ __forceinline__ float2 *pairs32(const Fields<float> &F, int s) { return (float2 *)F.P[s][0]; }

// Stage bookkeeping of the ring: s is the stage of the plane being computed.
template <int NS> struct RingIdx {
    int s;
    __device__ __forceinline__ int up(bool top) const { return top ? s : (s + 1 == NS ? 0 : s + 1); }
    __device__ __forceinline__ int dn(bool bottom) const { return bottom ? s : (s == 0 ? NS - 1 : s - 1); }
    __device__ __forceinline__ int ahead() const { return s >= 2 ? s - 2 : s + NS - 2; }   // plane k + NS - 2
    __device__ __forceinline__ void next() { s = s + 1 == NS ? 0 : s + 1; }
};

// A compile-time choice of a loop's form.
template <int V> struct Mode { static constexpr int value = V; };

// The plane of the pinned cell where it lies in this thread's column, else -1.
__device__ __forceinline__ int pin_plane(const Geom &g, int ref)
{
    const int plane = (int)g.plane, k = ref / plane;
    return ref - k * plane == (int)g.own_pl ? k : -1;
}

// The neighbourhood of one cell as a residual pass sees it.
struct RCell {
    df xc, xe, xw, xn, xs, xu, xd;          // x = phi + dx (z neighbours as loaded, k+1 / k-1 clamped)
    float dc, de, dw, dn, ds, du, dd;        // pending correction (update passes)
    float pxe, pxw, pyn, pys, pzu, pzd;      // Pm for the divergence (z clamped)
    int mc, me, mw, mn, ms, mu, md;          // materials (general eps only)
};

// Film constants of a residual pass, held in registers.
struct RConst {
    df cb, cu;                  // eps_0_nd / (2h); eps / h^2 on every face (one eps)
    float dinv_u;               // Jacobi weight of the non-identity rows (one eps)
    int nz;
    bool neu;                   // Neumann z boundary (mirrored end rows, one pinned cell)
    long long ref;              // the pinned cell (film-local)
    const float *cf_h, *cf_l;   // general eps: face coefficient tables (through the film table)
};

// z neighbours of the operator (depol_varEPS.cu:86-99), given the loaded
// k+1 and k-1 values (clamped at the ends).
template <class V>
__device__ __forceinline__ void zpick(const RConst &rc, int k, V up, V dn, V &u, V &dd)
{
    if (!rc.neu || (k > 0 && k < rc.nz - 1)) { u = up; dd = dn; }
    else if (k == 0) { u = up; dd = up; }
    else { u = dn; dd = dn; }
}

// -A dx of one non-identity row in FP32 (dx: the pending correction).
template <bool UNI>
__device__ __forceinline__ float minus_adx(const RConst &rc, int k, const RCell &c)
{
    float du, ddn;
    zpick<float>(rc, k, c.du, c.dd, du, ddn);
    if (UNI) {
        // Neumann: modes of a whole side, and the constant that meets the pinned
        // cell, are far larger than their differences; the sum below rounds at
        // 6 |dx|, 1e-3 of A dx for a mode of 512 cells
        if (rc.neu)
            return rc.cu.h * (((c.de - c.dc) + (c.dw - c.dc)) + ((c.dn - c.dc) + (c.ds - c.dc)) +
                              ((du - c.dc) + (ddn - c.dc)));
        return rc.cu.h * ((c.de + c.dw) + (c.dn + c.ds) + (du + ddn) - 6.f * c.dc);
    }
    int mu, md;
    zpick<int>(rc, k, c.mu, c.md, mu, md);
    const float *ch = rc.cf_h + c.mc * 3;
    return ch[c.me] * (c.de - c.dc) - ch[c.mw] * (c.dc - c.dw) + ch[c.mn] * (c.dn - c.dc) -
           ch[c.ms] * (c.dc - c.ds) + ch[mu] * (du - c.dc) - ch[md] * (c.dc - ddn);
}

// ------------------------------------------------------------ TDGL step
// kernelCalc_antiferro (kernels_evol.cu:47-231) with E_dep of the current
// potential (depol_varEPS.cu:223-276) and the sweep-row sums
// (evolve.cu:256-357) in FP32, plus the warm start of the coming solve:
// the extrapolated potential is written to the film's free buffer, which the
// step's first residual pass then reads.

// Coefficients of one (material, interface) class as three float4: (relax, A,
// LdT, ag), (ags, b4, b12, g6), (a02, -, -, -); ROT: FilmDev::coef_rot.
template <bool ROT> __device__ __forceinline__ void load_coef4(const FilmDev *f, float4 (*sC)[3])
{
    if (threadIdx.x < 6) {
        if (ROT) {
            const float *c = f->coef_rot[threadIdx.x];
            #pragma unroll
            for (int q = 0; q < 3; ++q) sC[threadIdx.x][q] = make_float4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
            return;
        }
        const Coef<float> &c = f->coef32[threadIdx.x];
        sC[threadIdx.x][0] = make_float4(c.relax, c.A, c.LdT, c.ag);
        sC[threadIdx.x][1] = make_float4(c.ags, c.b4, c.b12, c.g6);
        sC[threadIdx.x][2] = make_float4(c.a02, 0.f, 0.f, 0.f);
    }
}

// One cell: P^{n+1} (pn) from P^n (pc), the 6-neighbour sums, -E (ex, ey, ez)
// and -Ez_applied (mEz); pMZl, pSZl (crystal frame) for the sweep rows.
// The grain's rotation t (row major) given.
__device__ __forceinline__ void tdgl_cell32t(const float4 *K, const float (&t)[9], const float (&pc)[6],
                                             const float (&sum)[6], float ex, float ey, float ez, float mEz,
                                             float (&pn)[6], float &pMZl, float &pSZl)
{
    const float4 ka = K[0], kb = K[1], kc = K[2];
    const float relax = ka.x, A = ka.y, LdT = ka.z, ag = ka.w, ags = kb.x, b4 = kb.y, b12 = kb.z, g6 = kb.w;
    const float a02 = kc.x;
    // crystal frame (kernels_evol.cu:162-168)
    const float pMXl = t[0] * pc[0] + t[1] * pc[1] + t[2] * pc[2];
    const float pMYl = t[3] * pc[0] + t[4] * pc[1] + t[5] * pc[2];
    pMZl = t[6] * pc[0] + t[7] * pc[1] + t[8] * pc[2];
    const float pSXl = t[0] * pc[3] + t[1] * pc[4] + t[2] * pc[5];
    const float pSYl = t[3] * pc[3] + t[4] * pc[4] + t[5] * pc[5];
    pSZl = t[6] * pc[3] + t[7] * pc[4] + t[8] * pc[5];
    // two-sublattice Landau derivative (kernels_evol.cu:178-199)
    const float dmx = a02 * pMXl, dmy = a02 * pMYl;
    const float dsx = a02 * pSXl, dsy = a02 * pSYl;
    const float m2 = pMZl * pMZl, m3 = m2 * pMZl, m4 = m3 * pMZl, m5 = m4 * pMZl;
    const float q2 = pSZl * pSZl, q3 = q2 * pSZl, q4 = q3 * pSZl, q5 = q4 * pSZl;
    float dmz = ag * pMZl + b4 * m3;
    dmz = dmz + b12 * pMZl * q2;
    dmz = dmz + g6 * (m5 + 10.f * m3 * q2 + 5.f * pMZl * q4);
    float dsz = ags * pSZl + b4 * q3;
    dsz = dsz + b12 * pSZl * m2;
    dsz = dsz + g6 * (q5 + 10.f * m2 * q3 + 5.f * pSZl * m4);
    // back to the lab frame (kernels_evol.cu:202-208) + fields (:210-220)
    float b[6];
    b[0] = t[0] * dmx + t[3] * dmy + t[6] * dmz + ex;
    b[1] = t[1] * dmx + t[4] * dmy + t[7] * dmz + ey;
    b[2] = t[2] * dmx + t[5] * dmy + t[8] * dmz + (mEz + ez);
    b[3] = t[0] * dsx + t[3] * dsy + t[6] * dsz;
    b[4] = t[1] * dsx + t[4] * dsy + t[7] * dsz;
    b[5] = t[2] * dsx + t[5] * dsy + t[8] * dsz;
    // explicit Euler with the 6-neighbour Laplacian (kernels_evol.cu:223-229)
    #pragma unroll
    for (int q = 0; q < 6; ++q) pn[q] = pc[q] * relax + A * sum[q] - LdT * b[q];
}

__device__ __forceinline__ void load_tr32(const float4 *tr, float (&t)[9])
{
    const float4 t0 = __ldg(tr), t1 = __ldg(tr + 1), t2 = __ldg(tr + 2);
    t[0] = t0.x; t[1] = t0.y; t[2] = t0.z; t[3] = t0.w;
    t[4] = t1.x; t[5] = t1.y; t[6] = t1.z; t[7] = t1.w; t[8] = t2.x;
}

// The same for orthonormal rotations T (rows t1, t2, t3).  The transverse
// restoring terms a02 act alike on both transverse directions, so
//   T^T diag(a02, a02, d) T P = a02 P + (d - a02) (t3 . P) t3:
// only the polar axis t3 is needed, one load of 16 bytes instead of three, and
// the step is, with m = t3 . Pm, s = t3 . Ps and every coefficient times LdT,
//   Pm' = Pm + (A sum - (6 A + LdT a02) Pm - m p(m, s) t3 - LdT E),
//   p(m, s) = ag - a02 + m^2 (b4 + g6 (m^2 + 10 s^2)) + s^2 (b12 + 5 g6 s^2)
// (kernels_evol.cu:162-229): 51 FP32 instructions for the two rotations there
// and back, the Landau polynomials and the update, from about 97.  The
// increment is formed apart: the rounding of a factor 1 - 6 A - LdT a02 would
// recur every step (2.4e-6 instead of 7e-7 of error in P after 120 steps).
// K: (6 A + LdT a02, A, LdT, ag'), (ags', b4', b12', g6'), (5 g6', -, -, -).
__device__ __forceinline__ void tdgl_cell32r(const float4 *K, const float4 t, const float (&pc)[6],
                                             const float (&sum)[6], float ex, float ey, float ez, float mEz,
                                             float (&pn)[6], float &pMZl, float &pSZl)
{
    const float4 ka = K[0], kb = K[1];
    const float g65 = K[2].x;
    const float m = fmaf(t.z, pc[2], fmaf(t.y, pc[1], t.x * pc[0]));
    const float s = fmaf(t.z, pc[5], fmaf(t.y, pc[4], t.x * pc[3]));
    pMZl = m;
    pSZl = s;
    const float m2 = m * m, s2 = s * s;
    const float um = fmaf(kb.w, fmaf(10.f, s2, m2), kb.y), us = fmaf(kb.w, fmaf(10.f, m2, s2), kb.y);
    const float vm = fmaf(g65, s2, kb.z), vs = fmaf(g65, m2, kb.z);
    const float qm = -m * fmaf(m2, um, fmaf(s2, vm, ka.w));
    const float qs = -s * fmaf(s2, us, fmaf(m2, vs, kb.x));
    const float tt[3] = {t.x, t.y, t.z}, e[3] = {ex, ey, mEz + ez};
    #pragma unroll
    for (int q = 0; q < 3; ++q) {
        pn[q] = pc[q] + fmaf(-ka.x, pc[q], fmaf(ka.y, sum[q], fmaf(qm, tt[q], -ka.z * e[q])));
        pn[3 + q] = pc[3 + q] + fmaf(-ka.x, pc[3 + q], fmaf(ka.y, sum[3 + q], qs * tt[q]));
    }
}

// One cell of grain entry gid of the film's rotations TR4.
template <bool ROT>
__device__ __forceinline__ void tdgl_cell32(const float4 *K, const float4 *TR4, int gid, const float (&pc)[6],
                                            const float (&sum)[6], float ex, float ey, float ez, float mEz,
                                            float (&pn)[6], float &pMZl, float &pSZl)
{
    if (ROT) {
        tdgl_cell32r(K, __ldg(TR4 + gid), pc, sum, ex, ey, ez, mEz, pn, pMZl, pSZl);
    } else {
        float t[9];
        load_tr32(TR4 + 3LL * gid, t);
        tdgl_cell32t(K, t, pc, sum, ex, ey, ez, mEz, pn, pMZl, pSZl);
    }
}

// z neighbours of the potential for E (depol_varEPS.cu:246-273): zero beyond
// the Dirichlet planes, mirrored for the Neumann boundary.
__device__ __forceinline__ void efield_z(bool neumann, int k, int nz, df fu, df fd, df &pu, df &pd)
{
    if (!neumann) {
        pu = (k == nz - 1) ? df{0.f, 0.f} : fu;
        pd = (k == 0) ? df{0.f, 0.f} : fd;
    } else {
        pu = (k == nz - 1) ? fd : fu;         // mirrored (depol_varEPS.cu:86-99)
        pd = (k == 0) ? fu : fd;
    }
}

template <int NV>
__device__ __forceinline__ void row_acc(float (&acc)[NV], int mat, const float (&pn)[6], float pMZl, float pSZl)
{
    acc[0] += pn[2];
    acc[1] += pn[5];
    acc[2] += pMZl;
    acc[3] += pSZl;
    acc[4] += (mat == 1) ? pn[2] : 0.f;
    acc[5] += (mat == 0) ? pn[2] : 0.f;
    acc[6] += (mat == 2) ? pn[2] : 0.f;
}

constexpr int T32_NS = 4;
// Stage layout (own + halo slots): P as three float2 planes (P0, P1), (P2, P3),
// (P4, P5), the potential as one (hi, lo) float2 plane, then the code (own),
// and with DEF the pending correction dx (own + halo): a stencil point of a
// pair is one 8-byte shared load.
template <int TYc, bool DEF = false> __host__ __device__ constexpr int t32_stage()      // floats
{
    return 8 * TileShape<TYc>::SPLt + TileShape<TYc>::NTt + (DEF ? TileShape<TYc>::SPLt : 0);
}
template <int TYc, bool DEF = false> constexpr size_t t32_smem()
{
    return sizeof(float) * T32_NS * t32_stage<TYc, DEF>();
}

__device__ __forceinline__ void tdgl_def_film(const Dev &d, int rs, int fi, FilmTail &T);
__device__ __forceinline__ void tdgl_def_grid(const Dev &d, int rs);
__device__ __forceinline__ void tdgl_def_grid1(const Dev &d, int rs, FilmTail &T);

// TYc: the tile height (TX x TYc threads, one column each).
// DEF: a film whose previous step ended on its direct solve (SolveDev::pending;
// every depolarised film under kernel timing) has the potential x0 + dx -- the
// warm start in phi_cur plus the pending correction dx.  The step takes E
// from x0 + dx, writes x0 + dx to the free buffer (where the update pass
// would have put it), extrapolates the next warm start into the third-oldest
// potential's buffer (a warm start of at most quadratic order never reads
// it), and forms the check the update pass would have formed: r <- r - A dx
// in FP32 (r.r in the eighth partial sum).  The last block decides whether
// the previous step stands (tdgl_def_film, tdgl_def_grid).
// The check's values raise the registers a thread needs: the DEF kernels are
// built for three quarters of the blocks per SM (80 registers at 32 x 8
// tiles, where the 64 of four blocks spilled and ran 15 % slower).
template <int TYc, bool DEF> constexpr int tdgl32_minb()
{
    return DEF && TYc < 16 ? TileShape<TYc>::MINB * 3 / 4 : TileShape<TYc>::MINB;
}

template <int NS, int TYc = TY, bool DEF = false, bool FB = false, bool ROT = true>
__global__ void __launch_bounds__(TileShape<TYc>::NTt, tdgl32_minb<TYc, DEF>()) k_tdgl32(Dev d, Fields<float> F)
{
    static_assert(NS >= 4, "the ring holds planes k-1, k, k+1 and at least one in flight");
    constexpr int SPL = TileShape<TYc>::SPLt, NT = TileShape<TYc>::NTt, T32_STAGE = t32_stage<TYc, DEF>();
    constexpr int NV = DEF ? 8 : 7;         // row sums (+ the check's r.r)
    constexpr int DXO = 8 * SPL + NT;       // DEF: the dx plane of a stage
    extern __shared__ float4 smem_t32[];
    float *ring = (float *)smem_t32;
    __shared__ float4 sC[6][3];
    __shared__ double sRed[NT / 32][NV];
    __shared__ FilmTail tail;
    const int4 it = d.sitems[blockIdx.x];
    const FilmDev *f = d.films + it.x;
    const int z0 = it.w & 0xffff, z1 = it.w >> 16;
    load_coef4<ROT>(f, sC);
    const Geom g = make_geom<TYc>(f, it.y, it.z);
    const int cur = d.ctl->cur, rs = d.ctl->run_step;
    const float mEz = (float)(-d.wave[(long long)it.x * d.wstride + rs]);   // dfdPmz_app, kernels_evol.cu:210
    const int row = d.rows[(long long)it.x * d.wstride + rs];
    // film constants in registers (the stores below might alias the film table)
    const SolveDev *S = d.solve + it.x;
    const int nz = g.nz, warm_ = warm_order(f, S);
    const bool dep_ = f->dep_flag != 0, neu_ = f->zbc != 0;
    const float inv_2hf = f->inv_2hf;
    const long long off = f->off, lo = d.ncells, fs = d.ncells;
    const bool pend_ = DEF && dep_ && (d.force || S->pending != 0);
    const float2 *ph = phi2_sel(d, S->phi_cur) + off;
    const float2 *qh = phi2_sel(d, S->phi_prev) + off;
    const float2 *uh = phi2_sel(d, S->phi_prev2) + off;
    const float2 *vh = phi2_sel(d, S->phi_prev3) + off;
    float2 *nh = phi2_sel(d, pend_ ? S->phi_prev3 : phi_free(S)) + off;
    float2 *xh = phi2_sel(d, phi_free(S)) + off;     // DEF: the checked potential x0 + dx
    const float *dxg = F.x + off, *rg = F.r + off;
    const uint32_t *code = d.code + off;
    const float4 *TR4 = (const float4 *)(F.TR + (long long)(ROT ? TR32_ROT : TR32_GEN) * f->g_off);
    const float2 *Po = pairs32(F, cur) + off;   // the three pairs of a set at j * fs
    float2 *Pn = pairs32(F, cur ^ 1) + off;
    const int zlo = max(z0 - 1, 0), zhi = min(z1, nz - 1);
    (void)lo;
    // the check's operator (one eps) and identity rows, as the update pass has them
    RConst rc;
    rc.cu = df{f->cf_h[0], f->cf_l[0]};
    rc.nz = nz;
    rc.neu = neu_;
    const int kpin = neu_ ? pin_plane(g, f->ref_id) : -1;

    // copies of plane p (planes are issued in order, p = zlo, zlo + 1, ...)
    long long own_o = g.own_pl + (long long)zlo * g.plane, halo_o = g.halo_pl + (long long)zlo * g.plane;
    auto issue = [&](int p, float *st, bool dep, bool pend) {
        if (p <= zhi) {
            if (g.valid) {
                #pragma unroll
                for (int j = 0; j < 3; ++j) cp8(st + 2 * (j * SPL + g.own_slot), Po + j * fs + own_o);
                if (dep) cp8(st + 2 * (3 * SPL + g.own_slot), ph + own_o);
                cp4(st + 8 * SPL + threadIdx.x, code + own_o);
                if (pend) cp4(st + DXO + g.own_slot, dxg + own_o);
            }
            if (g.halo) {
                #pragma unroll
                for (int j = 0; j < 3; ++j) cp8(st + 2 * (j * SPL + g.halo_slot), Po + j * fs + halo_o);
                if (dep) cp8(st + 2 * (3 * SPL + g.halo_slot), ph + halo_o);
                if (pend) cp4(st + DXO + g.halo_slot, dxg + halo_o);
            }
        }
        cp_commit();
        own_o += g.plane;
        halo_o += g.plane;
    };
    for (int p = zlo; p <= z0 + NS - 3; ++p) issue(p, ring + (p - zlo) * T32_STAGE, dep_, pend_);

    float acc[NV];
    #pragma unroll
    for (int q = 0; q < NV; ++q) acc[q] = 0.f;
    const int s0 = g.own_slot;
    // The usual step (a depolarised Dirichlet film, quadratic warm start, DEF:
    // a pending check) without the tests of the others in its loop.  The loop
    // is bound by the instructions it issues (500 a cell, 180 of them FP32
    // arithmetic): 256x256x32 62.4 -> 59.2 us, 512x512x64 348 -> 332.
    // (Packed FP32 additions for the sums and the update measured the same;
    // one wave of blocks with equal shares of planes instead of chunks saved
    // 4 us here and lost 40 at 512x512x64, whose neighbouring columns then
    // stand at different planes and miss L2.)
    auto planes = [&](auto mode) {
        constexpr bool STD = decltype(mode)::value != 0;
        const bool dep = STD || dep_, pend = DEF && (STD || pend_), neu = !STD && neu_, sums = STD || row >= 0;
        const int warm = STD ? 2 : warm_;
        RConst rq = rc;
        rq.neu = neu;
        RingIdx<NS> ri{z0 - zlo};
        long long o = g.own_pl + (long long)z0 * g.plane;
        for (int k = z0; k < z1; ++k, o += g.plane, ri.next()) {
            cp_wait<NS - 4>();
            __syncthreads();
            issue(k + NS - 2, ring + ri.ahead() * T32_STAGE, dep, pend);
            if (!g.valid) continue;
            // older potentials for the warm start (consumed after the step's arithmetic)
            df wq{0.f, 0.f}, wu{0.f, 0.f}, wv{0.f, 0.f};
            if (dep && warm >= 1) wq = ld_df(qh + o);
            if (dep && warm >= 2) wu = ld_df(uh + o);
            if (dep && warm >= 3) wv = ld_df(vh + o);
            const float rold = pend ? rg[o] : 0.f;          // DEF: r of the step's first pass
            const float *sk = ring + ri.s * T32_STAGE;
            const float *su = ring + ri.up(k == nz - 1) * T32_STAGE, *sd = ring + ri.dn(k == 0) * T32_STAGE;
            const uint32_t c = ((const uint32_t *)sk)[8 * SPL + threadIdx.x];
            const float2 *k2 = (const float2 *)sk, *u2 = (const float2 *)su, *d2 = (const float2 *)sd;
            float pc[6], sum[6];
            #pragma unroll
            for (int p = 0; p < 3; ++p) {
                const float2 *a = k2 + p * SPL;
                const float2 cc = a[s0], xe = a[s0 + 1], xw = a[s0 - 1], yn = a[s0 + SX], ys = a[s0 - SX];
                const float2 zu = u2[p * SPL + s0], zd = d2[p * SPL + s0];
                pc[2 * p] = cc.x;
                pc[2 * p + 1] = cc.y;
                // neighbour sums e, w, n, s, u, d (kernels_evol.cu:101-122); z clamped
                sum[2 * p] = ((((xe.x + xw.x) + yn.x) + ys.x) + zu.x) + zd.x;
                sum[2 * p + 1] = ((((xe.y + xw.y) + yn.y) + ys.y) + zu.y) + zd.y;
            }
            float ex = 0.f, ey = 0.f, ez = 0.f;
            df a0{0.f, 0.f};
            float chk = 0.f;                                // DEF: the check's r, formed here
            if (dep) {
                const float2 *f2 = k2 + 3 * SPL;
                const float2 fc = f2[s0], fu = u2[3 * SPL + s0], fd = d2[3 * SPL + s0];
                const float2 fe = f2[s0 + 1], fw = f2[s0 - 1], fn = f2[s0 + SX], fsth = f2[s0 - SX];
                a0 = df{fc.x, fc.y};
                df pu, pd;
                efield_z(neu, k, nz, df{fu.x, fu.y}, df{fd.x, fd.y}, pu, pd);
                // -1 * E with E = -(phi_+ - phi_-) / (2h)
                ex = phi_diff32(df{fe.x, fe.y}, df{fw.x, fw.y});
                ey = phi_diff32(df{fn.x, fn.y}, df{fsth.x, fsth.y});
                ez = phi_diff32(pu, pd);
                if (pend) {
                    // phi = x0 + dx: the differences of dx added, the own value
                    // resolved and stored; the update pass's r <- r - A dx
                    // (identity rows: x - g with g = 0)
                    RCell cd;
                    const float *dk = sk + DXO;
                    cd.dc = dk[s0]; cd.de = dk[s0 + 1]; cd.dw = dk[s0 - 1]; cd.dn = dk[s0 + SX]; cd.ds = dk[s0 - SX];
                    cd.du = su[DXO + s0]; cd.dd = sd[DXO + s0];
                    df du{cd.du, 0.f}, dd{cd.dd, 0.f};
                    efield_z(neu, k, nz, du, dd, du, dd);
                    ex += cd.de - cd.dw;
                    ey += cd.dn - cd.ds;
                    ez += du.h - dd.h;
                    a0 = df_add_f(a0, cd.dc);
                    xh[o] = make_float2(a0.h, a0.l);
                    const bool ident = neu ? k == kpin : (k == 0 || k == nz - 1);
                    chk = ident ? -(a0.h + a0.l) : rold + minus_adx<true>(rq, k, cd);
                }
                ex *= inv_2hf;
                ey *= inv_2hf;
                ez *= inv_2hf;
            }
            float pn[6], pMZl, pSZl;
            tdgl_cell32<ROT>(sC[code_mat(c) * 2 + code_iface(c)], TR4, code_gid(c), pc, sum, ex, ey, ez, mEz, pn, pMZl, pSZl);
            #pragma unroll
            for (int j = 0; j < 3; ++j) Pn[j * fs + o] = make_float2(pn[2 * j], pn[2 * j + 1]);
            if (sums) row_acc(acc, code_mat(c), pn, pMZl, pSZl);
            if (dep) {
                const df w = extrap_phi(warm, a0, wq, wu, wv);
                nh[o] = make_float2(w.h, w.l);
            }
            if (pend) acc[NV - 1] = fmaf(chk, chk, acc[NV - 1]);
        }
    };
    if (dep_ && pend_ == DEF && warm_ == 2 && !neu_) planes(Mode<1>{});
    else planes(Mode<0>{});
    cp_wait<0>();

    if (row >= 0 || pend_) block_total32<NV>(d, it.x, 0, acc, sRed);
    if constexpr (DEF)
        finish32<FB>(d, [&](int fi) { tdgl_def_film(d, rs, fi, tail); },
                     [&] { if (FB) tdgl_def_grid(d, rs); else tdgl_def_grid1(d, rs, tail); });
    else
        finish32<FB>(d, [&](int fi) { tdgl_film32(d, rs, fi, tail); }, [&] { tdgl_grid32(d, rs); });
}

// The end of a TDGL step that may carry deferred checks (finish32): every
// pending film's r.r of its check decides whether its previous step stands
// (the update pass's test, ||r|| <= refine_tol ||b||).  If every check
// passes, the checked potentials become current and the step begins as
// tdgl_grid32 begins it.  If one fails, the previous step is reopened: the
// step counters and the P sets roll back, the failed films are set up for
// the update pass that the step's next residual pass then is, the films
// whose checks passed stay pending (the repeated step checks them again, to
// the same result), and the step loop runs this step again after that pass
// has ended the previous one.
// Film fi's part: its sweep row and its check's r.r (S->rr64).
__device__ __forceinline__ void tdgl_def_film(const Dev &d, int rs, int fi, FilmTail &T)
{
    const FilmDev *ff = d.films + fi;
    const int frow = d.rows[(long long)fi * d.wstride + rs], dep = ff->dep_flag;
    film_tail<8>(d, fi, 0, T);
    if (!d.force) {             // kernel timing: the totals as a step forms them; the state stays as it is
        if (frow >= 0) row_write(d, fi, frow, T.tot, T.c.step);
        if (threadIdx.x == 0 && dep && T.S.pending) d.solve[fi].rr64 = T.tot[7];
    }
}

// A pending film's check passed (NaN fails): the update pass's test, with what
// the update may have rounded off (refine_film).
__device__ __forceinline__ bool check_met(const FilmDev *f, double rr, double bb, float upd_err)
{
    if (rr == 0.0) return true;
    if (!(rr <= f->refine_tol2 * bb)) return false;
    const float uc = f->upd_c;
    if (uc == 0.f) return true;
    const float q = rel_norm(rr, bb);
    return q + (upd_err + uc * q) <= f->refine_tolf;
}
// The same of film fi's slot; rr read past this block's L1.
__device__ __forceinline__ bool def_check_ok(const Dev &d, int fi)
{
    const double rr = *(volatile const double *)&d.solve[fi].rr64;
    return check_met(d.films + fi, rr, d.solve[fi].bb, d.solve[fi].upd_err);
}

// What depends on every film: resolve and begin, or reopen.
__device__ __forceinline__ void tdgl_def_grid(const Dev &d, int rs)
{
    if (threadIdx.x != 0) return;
    if (d.force) {
        *d.counter = 0u;
        return;
    }
    bool fail = false;
    for (int fi = 0; fi < d.n_films; ++fi)
        if (d.films[fi].dep_flag && d.solve[fi].pending && !def_check_ok(d, fi)) fail = true;
    if (!fail) {
        for (int fi = 0; fi < d.n_films; ++fi) {
            SolveDev *S = d.solve + fi;
            if (S->pending) {
                // this launch wrote x0 + dx to the free buffer; the warm start
                // buffer (x0) takes the third-oldest slot, which held the next
                // warm start and now becomes the free one
                const int fr = phi_free(S);
                S->phi_prev3 = S->phi_cur;
                S->phi_cur = fr;
                S->pending = 0;
            }
            step_reset(d, fi);
        }
        step_begin(d, rs);
    } else {
        for (int fi = 0; fi < d.n_films; ++fi) {
            SolveDev *S = d.solve + fi;
            if (S->pending && !def_check_ok(d, fi)) {
                S->pending = 0;
                S->outer_active = 1;
                S->active = 0;
                S->refine = 1;
                S->upd = 1;
            }
        }
        step_reopen(d);
        set_cond(d, d.h_steps, 1);
    }
    *d.counter = 0u;
}

// The same for a single film, from its tail T (thread 0): the slot's fields
// are at hand, so the step begins or reopens with stores alone.
__device__ __forceinline__ void tdgl_def_grid1(const Dev &d, int rs, FilmTail &T)
{
    if (threadIdx.x != 0) return;
    if (!d.force) {
        SolveDev *S = d.solve;
        const FilmDev *f = d.films;
        const double rr = T.tot[7];
        const bool pend = f->dep_flag && T.S.pending;
        const bool ok = !pend || check_met(f, rr, T.S.bb, T.S.upd_err);
        if (ok) {
            if (T.S.pending) {
                // this launch wrote x0 + dx to the free buffer; the warm start
                // buffer (x0) takes the third-oldest slot, which held the next
                // warm start and now becomes the free one
                S->phi_prev3 = T.S.phi_cur;
                S->phi_cur = 10 - T.S.phi_cur - T.S.phi_prev - T.S.phi_prev2 - T.S.phi_prev3;
                S->pending = 0;
            }
            step_reset(d, 0);
            step_begin(d, rs);
        } else {
            S->pending = 0;
            S->outer_active = 1;
            S->active = 0;
            S->refine = 1;
            S->upd = 1;
            step_reopen(d);
            set_cond(d, d.h_steps, 1);
        }
    }
    *d.counter = 0u;
}

// Warm start alone (own cells): the free buffer of every depolarised film
// gets the extrapolated potential.  Used before a solve that does not follow
// a TDGL step (cmsl_film_depol).
static __global__ void __launch_bounds__(NT) k_extrap(Dev d)
{
    const int4 it = d.items[blockIdx.x];
    const FilmDev *f = d.films + it.x;
    const int z0 = it.w & 0xffff, z1 = it.w >> 16;
    const Geom g = make_geom(f, it.y, it.z);
    if (!f->dep_flag || !g.valid) return;
    const SolveDev *S = d.solve + it.x;
    const long long off = f->off;
    const float2 *ph = phi2_sel(d, S->phi_cur) + off;
    const float2 *qh = phi2_sel(d, S->phi_prev) + off;
    const float2 *uh = phi2_sel(d, S->phi_prev2) + off;
    const float2 *vh = phi2_sel(d, S->phi_prev3) + off;
    float2 *nh = phi2_sel(d, phi_free(S)) + off;
    const int warm = warm_order(f, S);
    for (int k = z0; k < z1; ++k) {
        const long long o = g.own_pl + (long long)k * g.plane;
        const df w = extrap_phi(warm, ld_df(ph + o), ld_df(qh + o), ld_df(uh + o), ld_df(vh + o));
        nh[o] = make_float2(w.h, w.l);
    }
}

// ------------------------------------------------- double-float residual
// One refinement pass of CMSL_FP32_REFINED's depolarisation solve: with x the
// potential -- on a step's first pass the warm start in the free buffer, on
// later passes the current potential plus the pending FP32 correction dx of
// the inner solve, written to the free buffer -- form b = -eps_0_nd div Pm
// (depol_varEPS.cu:279-329, zero on the Dirichlet planes / Neumann pin) and
// r = b - A x in double-float, and the partial sums r.r, b.b, r.D^-1.r.
// x = phi + dx is formed in double-float at every stencil point (dx can be
// as large as phi itself, e.g. the first solve after a cold start).  UNI:
// every material has the same eps, the operator is eps/h^2 times the 7-point
// Laplacian (one double-float product per cell, no material codes).
// An update pass (after the direct solve, once ||r|| <= 1e-4 ||b|| and while
// its FP32 rounding stays within a quarter of the refinement target,
// refine_film) instead forms r <- r - A dx in FP32.  With several eps, whose steps
// take five to eight passes, it reads dx and the codes where the full pass
// reads the potential, P and D^-1 with halos and works in double-float: 53.4
// -> 24.7 us a pass at 256x256x32, the step 692 -> 499 us.
// No FP64 instruction is executed.
// Stages of the ring.  Several eps: four, since the codes and D^-1 make a stage
// 10 KB and four blocks' five stages leave the L1 28 KB (256x256x32 with
// 50 / 30 / 15: a step 498 -> 489 us); one eps: five of 8 KB (four: 512x512x64
// first pass 128 -> 142 us).
template <bool UNI> constexpr int r32_ns() { return UNI ? 5 : 4; }

// sum of six double-float values minus 6 c; the hi parts are summed error-free
__device__ __forceinline__ df lap7(df e, df w, df n, df s, df u, df dn, df c)
{
    df t = two_sum(e.h, w.h);
    float l = t.l + (e.l + w.l);
    df t2 = two_sum(t.h, n.h);
    l += t2.l + n.l;
    t = two_sum(t2.h, s.h);
    l += t.l + s.l;
    t2 = two_sum(t.h, u.h);
    l += t2.l + u.l;
    t = two_sum(t2.h, dn.h);
    l += t.l + dn.l;
    const df p = two_prod(c.h, -6.f);
    l += fmaf(c.l, -6.f, p.l);
    t2 = two_sum(t.h, p.h);
    l += t2.l;
    return fast_two_sum(t2.h, l);
}

// (a - b) + (c - e) + (g - h) of FP32 values as double-float (hi parts error-free)
__device__ __forceinline__ df div3(float a, float b, float c, float e, float g, float h)
{
    const df x = two_sum(a, -b), y = two_sum(c, -e), z = two_sum(g, -h);
    const df s = two_sum(x.h, y.h);
    float l = s.l + (x.l + y.l);
    const df s2 = two_sum(s.h, z.h);
    l += s2.l + z.l;
    return fast_two_sum(s2.h, l);
}

// r (FP32 value of b - A x, double-float arithmetic) and b.h of one non-identity row.
template <bool UNI>
__device__ __forceinline__ void refine_row(const RConst &rc, int k, const RCell &c, float &rv, float &bh)
{
    const df bm = df_mul(div3(c.pxe, c.pxw, c.pyn, c.pys, c.pzu, c.pzd), rc.cb);   // -b
    df xu, xd;
    zpick<df>(rc, k, c.xu, c.xd, xu, xd);
    df s;            // b - A phi
    if (UNI) {
        s = df_sub(df_mul(rc.cu, lap7(c.xe, c.xw, c.xn, c.xs, xu, xd, c.xc)), bm);
    } else {
        int mu, md;
        zpick<int>(rc, k, c.mu, c.md, mu, md);
        const int m3 = c.mc * 3;
        auto cf = [&](int i) { return df{rc.cf_h[m3 + i], rc.cf_l[m3 + i]}; };
        df a = df_sub(df_mul(cf(c.me), df_sub(c.xe, c.xc)), df_mul(cf(c.mw), df_sub(c.xc, c.xw)));
        a = df_add(a, df_mul(cf(c.mn), df_sub(c.xn, c.xc)));
        a = df_sub(a, df_mul(cf(c.ms), df_sub(c.xc, c.xs)));
        a = df_add(a, df_mul(cf(mu), df_sub(xu, c.xc)));
        a = df_sub(a, df_mul(cf(md), df_sub(c.xc, xd)));
        s = df_sub(a, bm);
    }
    rv = s.h + s.l;
    bh = -bm.h;
}

// The last part of a residual pass of one cell: r and the partial sums.
// upd: r = r_old - A dx (b.b is not formed); otherwise r = b - A x.
template <bool UNI>
__device__ __forceinline__ void refine_cell(const RConst &rc, int k, bool ident, bool upd, const RCell &c,
                                            float r_old, float dinv, float &rv, float (&acc)[3])
{
    float bh = 0.f, wj = 1.f;
    if (ident) {
        rv = -(c.xc.h + c.xc.l);              // x - g with g = 0, b = 0
    } else {
        if (upd) rv = r_old + minus_adx<UNI>(rc, k, c);
        else refine_row<UNI>(rc, k, c, rv, bh);
        wj = UNI ? rc.dinv_u : upd ? 1.f : dinv;    // several eps: only the sign of the update's third sum is used
    }
    acc[0] = fmaf(rv, rv, acc[0]);
    acc[1] = fmaf(bh, bh, acc[1]);
    acc[2] = fmaf(rv, rv * wj, acc[2]);
}

// Stage layout (floats): x = phi (+ dx) as one (hi, lo) float2 plane, dx,
// the (Pmx, Pmy) pair plane, Pmz (own), then the general-eps code and D^-1.
// The update pass keeps the old r of the own cell in the Pmz slot.
template <bool UNI, int TYc = TY> struct R32Lay {
    static constexpr int SPL = TileShape<TYc>::SPLt, NT = TileShape<TYc>::NTt;
    static constexpr int FX = 0, DX = 2 * SPL, PA = 3 * SPL, PZ = 5 * SPL;
    static constexpr int CODE = 5 * SPL + NT, DINV = 6 * SPL + NT;   // general eps only
    static constexpr int STAGE = UNI ? 5 * SPL + NT : 6 * SPL + 2 * NT;
};
template <bool UNI, int TYc = TY> constexpr size_t r32_smem()
{
    return sizeof(float) * r32_ns<UNI>() * R32Lay<UNI, TYc>::STAGE;
}

template <bool UNI, int NS, int TYc = TY, bool FB = false>
__global__ void __launch_bounds__(TileShape<TYc>::NTt, TileShape<TYc>::MINB) k_refine32(Dev d, Fields<float> F)
{
    static_assert(NS >= 4, "the ring holds planes k-1, k, k+1 and at least one in flight");
    using L = R32Lay<UNI, TYc>;
    constexpr int NT = TileShape<TYc>::NTt;
    extern __shared__ float4 smem_r32[];
    float *ring = (float *)smem_r32;
    __shared__ double sRed[NT / 32][3];
    __shared__ FilmTail tail;
    const int4 it = d.sitems[blockIdx.x];
    const FilmDev *f = d.films + it.x;
    const SolveDev *S = d.solve + it.x;
    const int z0 = it.w & 0xffff, z1 = it.w >> 16;
    const Geom g = make_geom<TYc>(f, it.y, it.z);
    const int nz = g.nz;
    // film constants in registers (the stores below might alias the film table)
    RConst rc;
    rc.cb = df{f->cb_h, f->cb_l};
    rc.cu = df{f->cf_h[0], f->cf_l[0]};
    rc.dinv_u = f->dinv_uni;
    rc.nz = nz;
    rc.neu = f->zbc != 0;
    rc.ref = f->ref_id;
    rc.cf_h = f->cf_h;
    rc.cf_l = f->cf_l;
    const bool run_ = f->dep_flag != 0 && (d.force || S->outer_active);
    const bool apply_ = S->refine > 0;                  // later pass: x = phi + dx; first: the warm start
    const bool upd_ = apply_ && S->upd && f->upd_ok;     // r <- r - A dx (after the direct solve)
    const int cur = d.ctl->cur, fr = phi_free(S);
    const long long off = f->off, fs = d.ncells;
    const float2 *xh = phi2_sel(d, apply_ ? S->phi_cur : fr) + off;
    float2 *nh = phi2_sel(d, fr) + off;
    const float *dx = F.x + off;
    const float2 *PA = pairs32(F, cur ^ 1) + off;            // the new (Pmx, Pmy)
    const float *PZ = (const float *)(PA + fs);              // the new Pmz: .x of the (Pmz, Psx) pairs
    const uint32_t *code = d.code + off;
    const float *dinv = F.dinv + off;
    float *r = F.r + off;
    const int zlo = max(z0 - 1, 0), zhi = min(z1, nz - 1);

    // copies of plane p (planes are issued in order, p = zlo, zlo + 1, ...)
    long long own_o = g.own_pl + (long long)zlo * g.plane, halo_o = g.halo_pl + (long long)zlo * g.plane;
    auto issue = [&](int p, float *st, bool run, bool apply, bool upd) {
        if (run && p <= zhi) {
            const int so = g.own_slot, sh = g.halo_slot;
            if (upd) {
                // update pass: dx (several eps: and the codes) with its halo; phi and the old r of the own cell
                if (g.valid) {
                    cp8(st + L::FX + 2 * so, xh + own_o);
                    cp4(st + L::DX + so, dx + own_o);
                    cp4(st + L::PZ + threadIdx.x, r + own_o);
                    if (!UNI) cp4(st + L::CODE + so, code + own_o);
                }
                if (g.halo) {
                    cp4(st + L::DX + sh, dx + halo_o);
                    if (!UNI) cp4(st + L::CODE + sh, code + halo_o);
                }
            } else {
                if (g.valid) {
                    cp8(st + L::FX + 2 * so, xh + own_o);
                    if (apply) cp4(st + L::DX + so, dx + own_o);
                    cp8(st + L::PA + 2 * so, PA + own_o);
                    cp4(st + L::PZ + threadIdx.x, PZ + 2 * own_o);
                    if (!UNI) {
                        cp4(st + L::CODE + so, code + own_o);
                        cp4(st + L::DINV + threadIdx.x, dinv + own_o);
                    }
                }
                if (g.halo) {
                    cp8(st + L::FX + 2 * sh, xh + halo_o);
                    if (apply) cp4(st + L::DX + sh, dx + halo_o);
                    cp8(st + L::PA + 2 * sh, PA + halo_o);
                    if (!UNI) cp4(st + L::CODE + sh, code + halo_o);
                }
            }
        }
        cp_commit();
        own_o += g.plane;
        halo_o += g.plane;
    };
    for (int p = zlo; p <= z0 + NS - 3; ++p) issue(p, ring + (p - zlo) * L::STAGE, run_, apply_, upd_);

    const int s0 = g.own_slot, tz = threadIdx.x;
    const int kpin = rc.neu ? pin_plane(g, rc.ref) : -1;
    float acc[3] = {0.f, 0.f, 0.f};
    // The loop of each kind of pass of a Dirichlet film (1 first, 2 later, 3
    // update) without the tests of the others: 70 % of the issue slots were
    // taken.  First pass at 256x256x32 32.8 -> 26.7 us, 512x512x64 163 -> 128;
    // later pass with three permittivities 57.7 -> 53.4.
    auto planes = [&](auto mode) {
        constexpr int MODE = decltype(mode)::value;
        const bool run = MODE != 0 || run_, apply = MODE ? MODE >= 2 : apply_, upd = MODE ? MODE == 3 : upd_;
        RConst rq = rc;
        rq.neu = MODE == 0 && rc.neu;
        RingIdx<NS> ri{z0 - zlo};
        long long o = g.own_pl + (long long)z0 * g.plane;
        for (int k = z0; k < z1; ++k, o += g.plane, ri.next()) {
            cp_wait<NS - 4>();
            __syncthreads();
            issue(k + NS - 2, ring + ri.ahead() * L::STAGE, run, apply, upd);
            if (!run || !g.valid) continue;
            const float *sk = ring + ri.s * L::STAGE;
            const float *su = ring + ri.up(k == nz - 1) * L::STAGE, *sd = ring + ri.dn(k == 0) * L::STAGE;
            auto D = [&](const float *st, int s) { return st[L::DX + s]; };
            auto X = [&](const float *st, int s) {        // x = phi (+ dx on later passes)
                const float2 v = ((const float2 *)(st + L::FX))[s];
                const df p{v.x, v.y};
                return apply ? df_add_f(p, D(st, s)) : p;
            };
            auto PAx = [&](const float *st, int s) { return ((const float2 *)(st + L::PA))[s].x; };
            auto PAy = [&](const float *st, int s) { return ((const float2 *)(st + L::PA))[s].y; };
            auto M = [&](const float *st, int s) { return UNI ? 0 : code_mat(((const uint32_t *)st)[L::CODE + s]); };
            RCell c;
            c.xc = X(sk, s0);
            c.mc = M(sk, s0); c.me = M(sk, s0 + 1); c.mw = M(sk, s0 - 1); c.mn = M(sk, s0 + SX); c.ms = M(sk, s0 - SX);
            c.mu = M(su, s0); c.md = M(sd, s0);
            if (upd) {
                c.dc = D(sk, s0); c.de = D(sk, s0 + 1); c.dw = D(sk, s0 - 1); c.dn = D(sk, s0 + SX);
                c.ds = D(sk, s0 - SX); c.du = D(su, s0); c.dd = D(sd, s0);
            } else {
                c.xe = X(sk, s0 + 1); c.xw = X(sk, s0 - 1); c.xn = X(sk, s0 + SX); c.xs = X(sk, s0 - SX);
                c.xu = X(su, s0); c.xd = X(sd, s0);
                c.pxe = PAx(sk, s0 + 1); c.pxw = PAx(sk, s0 - 1);
                c.pyn = PAy(sk, s0 + SX); c.pys = PAy(sk, s0 - SX);
                c.pzu = su[L::PZ + tz]; c.pzd = sd[L::PZ + tz];
            }
            // identity rows: the Dirichlet planes, or the Neumann pin
            const bool ident = rq.neu ? k == kpin : (k == 0 || k == nz - 1);
            float rv;
            refine_cell<UNI>(rq, k, ident, upd, c, upd ? sk[L::PZ + tz] : 0.f, UNI || upd ? 0.f : sk[L::DINV + tz], rv, acc);
            r[o] = rv;
            if (apply) nh[o] = make_float2(c.xc.h, c.xc.l);
        }
    };
    if (!run_ || rc.neu) planes(Mode<0>{});
    else if (!apply_) planes(Mode<1>{});
    else if (upd_) planes(Mode<3>{});
    else planes(Mode<2>{});
    cp_wait<0>();
    if (run_) block_total32<3>(d, it.x, 1, acc, sRed);
    finish32<FB>(d, [&](int fi) { refine_film(d, fi, tail); }, [&] { if (FB) refine_grid(d); else refine_grid1(d, tail); });
}

}  // namespace cmsl
