/*
 * k_pair64.cu -- the FP64 mode of the force kernels (md_set_precision(ctx,
 * 64)): the same pair and bonded force laws as the FP32 kernels, evaluated
 * in FP64 on the FP64 positions.  Pair forces take the
 * Coulomb term from a piecewise polynomial within 1e-16 of it and 1/r from
 * an iteration (rsqrt64), which together come closer to the force law than
 * FP64 arithmetic on the form as written; energies and bonded terms use exp,
 * log and IEEE divide and square root.
 *
 * This is the "plain FP64" form of the path run on the GPU: the reference
 * point of the precision gates (RMS force error, NVE drift) and the per-system
 * FP64 runs the adjoint's throughput is compared with.  The force law follows
 * pair_forces.cu:34-205 with the reference's A&S 7.1.26 erfc
 * (simulation.h:39-44, its float coefficients widened to FP64) and Wolf
 * shift W = rc Ft(rc) (forces.cu:104-110); bonds and angles follow
 * bonded_forces.cu:34-193 (U = k (r - r0)^2 with bnd1 = 2k, U = k (th -
 * th0)^2 with ang1 = 2k).  Forces go into the same int64 fixed-point arrays
 * (2^-32 kJ/mol/A: the rounding, ~1e-10 kJ/mol/A, is far below FP32's), so
 * the integrators, thermostats and reductions are shared with the FP32 mode.
 *
 * Layout: 8 lanes per atom, 4 or 16 atoms per block; lane l takes
 * the list entries l, l+8, ... of its atom's padded row (the padding entries
 * point at the atom itself, r = 0, and are skipped); each lane sums in FP64,
 * rounds its sums to fixed point once, and the lanes combine with integer
 * shuffles, so the result is deterministic.
 */
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "md_pair.cuh"

namespace {

constexpr int P64_TPA = 8;
constexpr int P64_THREADS = 128;   /* per block, at most */

/* What a thread keeps of its md_p64 (the table goes to shared memory). */
struct md_p64_model {
    int ni;
    float nih;
    double rcsq, rc, rcinv, rc6i, reacf, alpha, spi, pex, a[5], qfac, wolfw, ucc;
    double L[3], Li[3];
};

/* 1 / sqrt(s) for s in FP32's normal range: the FP32 approximation and one
 * step of Halley's iteration, whose error is about e^3 / 3 for a seed of
 * relative error e / 2 ~ 2^-23.  y y is exact (48 bits) and e rounded once,
 * so what remains is the rounding of the result: half an ulp and 2^-22 of
 * one, against one ulp for a square root and a divide. */
__device__ __forceinline__ double rsqrt64(double s, float &seed)
{
    seed = rsqrt_approx((float)s);
    const double y = (double)seed;
    const double e = fma(-s, y * y, 1.0);
    return fma(e * y, fma(e, 0.375, 0.5), y);
}

/* One pair: ff (F_i = ff d) and the pair energy (consistent potential,
 * LJ shifted to zero at rc) for r^2 <= rc^2.  The FP64 pipe issues one warp
 * instruction in 20 cycles, so its operations are what counts: the force's
 * Coulomb term comes from a piecewise polynomial (tab, 8 FP64 operations;
 * exp and the divide of the A&S form, which the energy takes, over 40).  4082 ions,
 * per launch: 230 us as written, 102 us so (77% of the FP64 pipe).  Its argument r - centre is one
 * fma of r^2 and 1/r: r itself is never rounded.  Against quad precision, at
 * distances from 1.5 A to rc (a rc 0.5 to 3.2): the largest error of G 1.2e-16
 * to 2.3e-16 (rms 4e-17), the form as written in FP64 4.1e-16 to 7.7e-16 (rms
 * 6e-17 to 1.8e-16).  Every rounding of the force is written out (no
 * contraction is left to the compiler), so that it has the same bits with and
 * without ENERGY and a trajectory does not depend on its energy steps. */
template <int KIND, bool ENERGY>
__device__ __forceinline__ void pair64_eval(const md_p64_model &m, const double *tab, double rsq,
                                            double qq, double lja, double ljc, double &ff, double &u)
{
    float seed;
    const double ri = rsqrt64(rsq, seed), ri2 = __dmul_rn(ri, ri);
    double fc, uc = 0.0;
    if (KIND == 1) {
        const bool table = m.ni > 0;
        double ec = 0.0, ex = 0.0, r = 0.0;
        if (ENERGY || !table) {   /* the form as written */
            r = __dmul_rn(rsq, ri);
            r = fma(fma(-r, r, rsq), __dmul_rn(0.5, ri), r);
            const double xa = __dmul_rn(m.alpha, r);
            const double t = __ddiv_rn(1.0, fma(m.pex, xa, 1.0));
            const double p = fma(fma(fma(fma(m.a[4], t, m.a[3]), t, m.a[2]), t, m.a[1]), t, m.a[0]);
            ex = exp(-__dmul_rn(xa, xa));
            ec = __dmul_rn(__dmul_rn(p, t), ex);
        }
        if (table) {
            const double *c = tab + (MD_P64_DEG + 2) * min((int)((float)rsq * seed * m.nih), m.ni - 1);
            const double y = fma(rsq, ri, -c[0]);
            double g = c[MD_P64_DEG + 1];
#pragma unroll
            for (int k = MD_P64_DEG; k > 0; k--) g = fma(g, y, c[k]);
            fc = __dmul_rn(qq, fma(g, ri, -m.wolfw));
        } else {
            fc = __dmul_rn(qq, __dsub_rn(fma(ec, ri, __dmul_rn(m.spi, ex)), m.wolfw));
        }
        if (ENERGY) uc = qq * (ec * ri - m.ucc + m.wolfw * log(r * m.rcinv));
    } else {
        fc = __dmul_rn(qq, fma(-m.reacf, rsq, ri));
        if (ENERGY) uc = qq * (ri + 0.5 * m.reacf * rsq - m.ucc);
    }
    const double ri6 = __dmul_rn(__dmul_rn(ri2, ri2), ri2);
    ff = __dmul_rn(ri2, fma(ri6, fma(lja, ri6, -ljc), fc));
    if (ENERGY)
        u = uc + (lja * (1.0 / 12.0) * (ri6 * ri6 - m.rc6i * m.rc6i) - ljc * (1.0 / 6.0) * (ri6 - m.rc6i));
}

/* Pair forces in FP64 of a single system (tab == nullptr: block b holds the
 * A = blockDim / 8 atoms from A b on) or of a batch (block b holds up to A
 * atoms of replica tab[b].x from tab[b].y on; geometry, model and LJ table per
 * replica). */
template <int KIND, bool ENERGY>
__global__ void __launch_bounds__(P64_THREADS) k_pair64(int n, int pitch, int cap, int centered,
                                                       const int2 *__restrict__ tab,
                                                       const md_rep *__restrict__ reps,
                                                       const md_p64 *__restrict__ models,
                                                       const float2 *__restrict__ ljtab,
                                                       const double *__restrict__ x,
                                                       const float4 *__restrict__ pos4,
                                                       const int *__restrict__ type,
                                                       const unsigned *__restrict__ nl,
                                                       const int *__restrict__ nl_n, long long *f,
                                                       float *vir, float *epot)
{
    __shared__ double2 lj[MD_MAXTYPE * MD_MAXTYPE];
    extern __shared__ double s_g[];   /* the replica's table */
    pdl_trigger();   /* the integrator may be scheduled; it waits for this grid */
    int rep = 0, i0, end;
    if (tab) {
        const int2 bt = tab[blockIdx.x];
        rep = bt.x;
        i0 = bt.y;
        end = reps[rep].atom0 + reps[rep].natom;
    } else {
        i0 = blockIdx.x * (blockDim.x / P64_TPA);
        end = n;
    }
    md_p64_model m;
    {
        const md_p64 &M = models[rep];
        m.ni = M.ni;
        m.nih = M.nih;
        m.rcsq = M.rcsq;
        m.rc = M.rc;
        m.rcinv = M.rcinv;
        m.rc6i = M.rc6i;
        m.reacf = M.reacf;
        m.alpha = M.alpha;
        m.spi = M.spi;
        m.pex = M.pex;
        for (int k = 0; k < 5; k++) m.a[k] = M.a[k];
        m.qfac = M.qfac;
        m.wolfw = M.wolfw;
        m.ucc = M.ucc;
        for (int k = 0; k < 3; k++) {
            m.L[k] = M.L[k];
            m.Li[k] = M.Li[k];
        }
        if (KIND == 1) {
            const double *g = &M.g[0][0];
            for (int k = threadIdx.x; k < m.ni * (MD_P64_DEG + 2); k += blockDim.x) s_g[k] = g[k];
        }
    }
    for (int k = threadIdx.x; k < MD_MAXTYPE * MD_MAXTYPE; k += blockDim.x) {
        const float2 l = ljtab[(size_t)rep * MD_MAXTYPE * MD_MAXTYPE + k];
        lj[k] = make_double2((double)l.x, (double)l.y);
    }
    __syncthreads();
    const int i = i0 + (int)threadIdx.x / P64_TPA, lane = (int)threadIdx.x % P64_TPA;
    const bool active = i < end;
    const int ii = active ? i : i0;
    const size_t P = (size_t)pitch;
    const double xi = x[ii], yi = x[P + ii], zi = x[2 * P + ii];
    const float4 pi = pos4[ii];
    const float bi[3] = {(float)m.Li[0], (float)m.Li[1], (float)m.Li[2]};
    const double qi = m.qfac * (double)pi.w;
    const double2 *ljrow = lj + type[ii] * MD_MAXTYPE;
    const int cnt = active ? nl_n[ii] : 0;
    const int npad = (cnt + P64_TPA - 1) / P64_TPA * P64_TPA;   /* padding past it adds zero */
    /* a warp whose atoms all lie at least rc from every face (positions
     * centred in the box) needs no minimum-image shift for any pair inside
     * rc: the shift is L * 0 there, and a pair beyond L/2 is beyond rc */
    const bool in_i = fabs(xi) + m.rc < 0.499 * m.L[0] && fabs(yi) + m.rc < 0.499 * m.L[1] &&
                      fabs(zi) + m.rc < 0.499 * m.L[2];
    const bool inner = centered && __all_sync(0xffffffffu, !active || in_i);
    double fx = 0.0, fy = 0.0, fz = 0.0, fw = 0.0, fe = 0.0;
    const unsigned *row = nl + (size_t)ii * cap;
    for (int k = lane; k < npad; k += P64_TPA) {
        const unsigned e = __ldg(row + k);
        const int j = (int)(e & MD_INDEX_MASK);
        double dx = xi - x[j], dy = yi - x[P + j], dz = zi - x[2 * P + j];
        const float4 pj = pos4[j];
        if (!inner && centered) {
            /* the shift's multiple of L from the FP32 positions (it differs
             * from the FP64 one only for |d| = L/2 to 1e-5 A, beyond rc);
             * most pairs have none, and then no FP64 operation */
            const float nx = rint_small((pi.x - pj.x) * bi[0]), ny = rint_small((pi.y - pj.y) * bi[1]),
                        nz = rint_small((pi.z - pj.z) * bi[2]);
            if (nx != 0.0f) dx = fma(-m.L[0], (double)nx, dx);
            if (ny != 0.0f) dy = fma(-m.L[1], (double)ny, dy);
            if (nz != 0.0f) dz = fma(-m.L[2], (double)nz, dz);
        } else if (!inner) {
            dx = fma(-m.L[0], rint(__dmul_rn(dx, m.Li[0])), dx);
            dy = fma(-m.L[1], rint(__dmul_rn(dy, m.Li[1])), dy);
            dz = fma(-m.L[2], rint(__dmul_rn(dz, m.Li[2])), dz);
        }
        const double rsq = fma(dz, dz, fma(dy, dy, __dmul_rn(dx, dx)));
        if (rsq <= m.rcsq && (float)rsq > 0.0f) {
            const double2 l = ljrow[e >> MD_TYPE_SHIFT];
            double ff, u = 0.0;
            pair64_eval<KIND, ENERGY>(m, s_g, rsq, __dmul_rn(qi, (double)pj.w), l.x, l.y, ff, u);
            fx = fma(ff, dx, fx);
            fy = fma(ff, dy, fy);
            fz = fma(ff, dz, fz);
            fw = fma(ff, rsq, fw);
            if (ENERGY) fe += 0.5 * u;
        }
    }
    long long ix = __double2ll_rn(fx * FX_SCALE), iy = __double2ll_rn(fy * FX_SCALE),
              iz = __double2ll_rn(fz * FX_SCALE);
#pragma unroll
    for (int off = P64_TPA / 2; off > 0; off >>= 1) {
        ix += __shfl_down_sync(0xffffffffu, ix, off, P64_TPA);
        iy += __shfl_down_sync(0xffffffffu, iy, off, P64_TPA);
        iz += __shfl_down_sync(0xffffffffu, iz, off, P64_TPA);
        fw += __shfl_down_sync(0xffffffffu, fw, off, P64_TPA);
        if (ENERGY) fe += __shfl_down_sync(0xffffffffu, fe, off, P64_TPA);
    }
    if (active && lane == 0) {
        f[i] = ix;
        f[P + i] = iy;
        f[2 * P + i] = iz;
        vir[i] = (float)fw;
        if (ENERGY) epot[i] = (float)fe;
    }
}

/* Harmonic bonds and angles in FP64 on the FP64 positions, one thread per
 * sorted atom (each bond seen from both atoms, each angle from all three),
 * added into the fixed-point forces; the same formulas as k_bonded.  In a
 * batch (reps non-null) the minimum image uses the atom's replica box. */
template <bool ENERGY>
__global__ void k_bonded64(int n, int pitch, const double *__restrict__ boxd,
                           const double *__restrict__ x, const int2 *__restrict__ bl_s,
                           const int *__restrict__ bl_sn, const int4 *__restrict__ al_s,
                           const int *__restrict__ al_sn, const float *__restrict__ par, int has_bonds,
                           int has_angles, const md_rep *__restrict__ reps, const int *__restrict__ arep,
                           long long *f, float *vir, float *epot)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const size_t P = (size_t)pitch;
    const int nb = has_bonds ? bl_sn[s] : 0;
    const int na = has_angles ? al_sn[s] : 0;
    if (nb == 0 && na == 0) return;
    const double *L = reps ? reps[arep[s]].boxd : boxd;
    const double Li[3] = {1.0 / L[0], 1.0 / L[1], 1.0 / L[2]};
    const float *bnd1 = par, *bnd2 = par + MD_MAXTYPE, *ang1 = par + 2 * MD_MAXTYPE,
                *ang2 = par + 3 * MD_MAXTYPE;
    auto pos = [&](int a, double *o) {
        o[0] = x[a];
        o[1] = x[P + a];
        o[2] = x[2 * P + a];
    };
    auto diff = [&](const double *a, const double *b, double *d) {
        for (int k = 0; k < 3; k++) {
            d[k] = a[k] - b[k];
            d[k] -= L[k] * rint(d[k] * Li[k]);
        }
    };
    double p[3];
    pos(s, p);
    double fx = 0.0, fy = 0.0, fz = 0.0, fw = 0.0, fe = 0.0;
    for (int k = 0; k < nb; k++) {
        const int2 b = bl_s[k * P + s];
        double q[3], d[3];
        pos(b.x, q);
        diff(p, q, d);
        const double rsq = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const double r = sqrt(rsq);
        const double kk = bnd1[b.y], r0 = bnd2[b.y];
        const double fa = kk * (r0 / r - 1.0);
        fw += fa * rsq;
        fx += fa * d[0];
        fy += fa * d[1];
        fz += fa * d[2];
        if (ENERGY) {
            const double dr = r - r0;
            fe += 0.25 * kk * dr * dr;
        }
    }
    for (int k = 0; k < na; k++) {
        const int4 a = al_s[k * P + s];
        double qa[3], qb[3], cen[3], va[3], vb[3];
        pos(a.z, qb);
        if (a.x == 1) {   /* this atom is the centre */
            pos(a.y, qa);
            cen[0] = p[0]; cen[1] = p[1]; cen[2] = p[2];
        } else {          /* this atom is an end */
            qa[0] = p[0]; qa[1] = p[1]; qa[2] = p[2];
            pos(a.y, cen);
        }
        diff(qa, cen, va);
        diff(qb, cen, vb);
        const double ai = 1.0 / sqrt(va[0] * va[0] + va[1] * va[1] + va[2] * va[2]);
        const double bi = 1.0 / sqrt(vb[0] * vb[0] + vb[1] * vb[1] + vb[2] * vb[2]);
        const double ab = va[0] * vb[0] + va[1] * vb[1] + va[2] * vb[2];
        double cang = ab * ai * bi;
        cang = fmin(fmax(cang, -0.9999999), 0.9999999);
        const double th = acos(cang);
        const double ff = (double)ang1[a.w] * (th - (double)ang2[a.w]) / sqrt(1.0 - cang * cang) * ai * bi;
        const double aa = ab * ai * ai;
        double g[3] = {vb[0] - aa * va[0], vb[1] - aa * va[1], vb[2] - aa * va[2]};
        if (a.x == 1) {
            const double bb = ab * bi * bi;
            for (int q = 0; q < 3; q++) g[q] = bb * vb[q] - va[q] - g[q];
        }
        fx += ff * g[0];
        fy += ff * g[1];
        fz += ff * g[2];
        if (ENERGY) {
            const double dth = th - (double)ang2[a.w];
            fe += 0.5 * (double)ang1[a.w] * dth * dth * (1.0 / 3.0);
        }
    }
    f[s] += __double2ll_rn(fx * FX_SCALE);
    f[P + s] += __double2ll_rn(fy * FX_SCALE);
    f[2 * P + s] += __double2ll_rn(fz * FX_SCALE);
    vir[s] += (float)fw;
    if (ENERGY) epot[s] += (float)fe;
}

}  // namespace

/* The pieces of G(r) = E(r) + spi r e^{-a^2 r^2} on [0, rc], E(r) = P5(t) t
 * e^{-a^2 r^2}, t = 1 / (1 + p a r): on each the Chebyshev interpolant of
 * degree MD_P64_DEG, written in powers of r - centre and computed in long
 * double, so that its coefficients are as good as FP64 holds them.  Takes the
 * fewest pieces whose deviation at four extrema of the next Chebyshev
 * polynomial, the shape of the error, is at most 1e-16, an ulp of G just below
 * 1 (G as written, evaluated in FP64, is off by 4e-16 to 8e-16; at 4e-15, the
 * line before, the pieces were the larger error); none: m.ni = 0. */
static void fit_coulomb(md_p64 &m)
{
    typedef long double real;
    constexpr int N = MD_P64_DEG + 1, CHK = 4;
    auto G = [&](real r) {
        const real xa = m.alpha * r, t = 1.0L / (1.0L + m.pex * xa);
        const real p = ((((m.a[4] * t + m.a[3]) * t + m.a[2]) * t + m.a[1]) * t + m.a[0]);
        const real ex = expl(-xa * xa);
        return p * t * ex + m.spi * r * ex;
    };
    const real pi = acosl(-1.0L), chk[CHK] = {-1.0L, cosl(5.0L * pi / 8.0L), cosl(3.0L * pi / 8.0L), 1.0L};
    static_assert(MD_P64_DEG == 7, "chk are extrema of T_8");
    /* T_j at the nodes, weighted, and (monomial) T_j's coefficients */
    real node[N], tj[N][N], mono[N][N] = {};
    for (int k = 0; k < N; k++) {
        node[k] = cosl(pi * (k + 0.5L) / N);
        for (int j = 0; j < N; j++) tj[j][k] = cosl(pi * j * (k + 0.5L) / N) * (j == 0 ? 1.0L : 2.0L) / N;
    }
    mono[0][0] = mono[1][1] = 1.0L;
    for (int j = 2; j < N; j++)
        for (int k = 0; k < N; k++) mono[j][k] = (k > 0 ? 2.0L * mono[j - 1][k - 1] : 0.0L) - mono[j - 2][k];
    for (int ni = 16; ni <= MD_P64_MAXI; ni *= 2) {
        const double h = 0.5 * m.rc / ni;   /* half a piece */
        bool ok = true;
        for (int q = 0; q < ni && ok; q++) {
            const double cen = (2 * q + 1) * h;
            real f[N], c[N] = {};
            for (int k = 0; k < N; k++) f[k] = G(cen + h * node[k]);
            for (int j = 0; j < N; j++) {
                real a = 0.0L;
                for (int k = 0; k < N; k++) a += f[k] * tj[j][k];
                for (int k = 0; k <= j; k++) c[k] += a * mono[j][k];
            }
            for (int k = 0; k < CHK && ok; k++) {
                const real y = chk[k];
                real g = 0.0L;
                for (int d = N - 1; d >= 0; d--) g = g * y + c[d];
                ok = fabsl(g - G(cen + h * y)) <= 1e-16L;
            }
            m.g[q][0] = cen;
            real hk = 1.0L;
            for (int k = 0; k < N; k++, hk *= h) m.g[q][k + 1] = (double)(c[k] / hk);
        }
        if (ok) {
            m.ni = ni;
            m.nih = (float)(ni / m.rc);
            return;
        }
    }
    m.ni = 0;
}

/* FP64 model constants of one system (pairmodel of the plain form): rc from
 * the FP32 rc^2 as given, the Wolf shift and energy constants with the A&S
 * erfc in FP64.  The table is that of one of the nmade models made before it
 * with the same rc and alpha, if there is one (a fit takes milliseconds). */
md_p64 md_make_p64(int lkspace, float rcutsq, float reacf, float alfa, const float box[3], const md_p64 *made,
                   int nmade)
{
    md_p64 m;
    memset(&m, 0, sizeof(m));
    m.kind = lkspace;
    m.rcsq = (double)rcutsq;
    m.rc = sqrt(m.rcsq);
    m.rcinv = 1.0 / m.rc;
    const double rc2i = 1.0 / m.rcsq;
    m.rc6i = rc2i * rc2i * rc2i;
    m.reacf = lkspace == 0 ? (double)reacf : 0.0;
    m.alpha = (double)alfa;
    m.spi = 2.0 / sqrt(3.14159265358979323846) * m.alpha;
    m.pex = (double)0.3275911f;
    m.a[0] = (double)A1;
    m.a[1] = (double)A2;
    m.a[2] = (double)A3;
    m.a[3] = (double)A4;
    m.a[4] = (double)A5;
    m.qfac = (double)QFAC;
    for (int k = 0; k < 3; k++) {
        m.L[k] = (double)box[k];
        m.Li[k] = 1.0 / m.L[k];
    }
    if (lkspace == 1) {
        const double xa = m.alpha * m.rc;
        const double t = 1.0 / (1.0 + m.pex * xa);
        const double p = ((((m.a[4] * t + m.a[3]) * t + m.a[2]) * t + m.a[1]) * t + m.a[0]);
        const double ec = p * t * exp(-xa * xa);
        m.wolfw = ec / m.rc + m.spi * exp(-m.alpha * m.alpha * m.rcsq);
        m.ucc = ec / m.rc;
    } else if (lkspace == 0) {
        m.ucc = 1.0 / m.rc + 0.5 * m.reacf * m.rcsq;
    }
    if (lkspace == 0) return m;
    for (int k = 0; k < nmade; k++)
        if (made[k].rcsq == m.rcsq && made[k].alpha == m.alpha) {
            m.ni = made[k].ni;
            m.nih = made[k].nih;
            memcpy(m.g, made[k].g, sizeof(m.g));
            return m;
        }
    fit_coulomb(m);
    return m;
}

void launch_pair64(md_ctx *c, bool energy)
{
    const bool batch = c->batch != 0;
    const int2 *tab = nullptr;
    int dev = 0, nsm = 1, nb;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    /* few atoms: blocks of one warp, so that the SMs' shares of the FP64 work
     * differ less (4082 ions: 255 blocks of four warps leave some SMs with
     * two and some with one, 116 us per launch; 102 us with one warp) */
    const int atoms = c->n / (P64_THREADS / P64_TPA) < 16 * nsm ? 32 / P64_TPA : P64_THREADS / P64_TPA;
    const int threads = atoms * P64_TPA;
    const size_t table = sizeof(double) * (MD_P64_DEG + 2) * (size_t)c->p64_ni;   /* the largest of the replicas' */
    if (batch) {
        const int k = md_grid_index(atoms);
        tab = c->grid_tab + c->grid_off[k];
        nb = c->grid_cnt[k];
    } else {
        nb = (c->n + atoms - 1) / atoms;
    }
    const float2 *lj = batch ? c->ljr_dev : (const float2 *)c->lj_dev;
    const md_rep *reps = batch ? c->reps_dev : nullptr;
#define MD_P64_ARGS                                                                                \
    c->n, c->pitch, c->cap, c->centered, tab, reps, (const md_p64 *)c->p64_dev, lj, (const double *)c->x, \
        (const float4 *)c->pos4, (const int *)c->type, (const unsigned *)c->nl, (const int *)c->nl_n, c->f, \
        c->vir, c->epot
    if (c->lkspace == 0) {
        if (energy) k_pair64<0, true><<<nb, threads, 0, c->stream>>>(MD_P64_ARGS);
        else k_pair64<0, false><<<nb, threads, 0, c->stream>>>(MD_P64_ARGS);
    } else {
        if (energy) k_pair64<1, true><<<nb, threads, table, c->stream>>>(MD_P64_ARGS);
        else k_pair64<1, false><<<nb, threads, table, c->stream>>>(MD_P64_ARGS);
    }
#undef MD_P64_ARGS
}

void launch_bonded64(md_ctx *c, bool energy, int hb, int ha)
{
    const int nb = (c->n + 255) / 256;
    const md_rep *reps = c->batch ? c->reps_dev : nullptr;
    const int *arep = c->batch ? c->arep : nullptr;
    /* a single system: the box of model 0 (a device address; not read here) */
    const double *boxd = (const double *)((const char *)c->p64_dev + offsetof(md_p64, L));
    if (energy)
        k_bonded64<true><<<nb, 256, 0, c->stream>>>(c->n, c->pitch, boxd, c->x, c->bl_s, c->bl_sn, c->al_s,
                                                    c->al_sn, c->bonded_par, hb, ha, reps, arep, c->f,
                                                    c->vir, c->epot);
    else
        k_bonded64<false><<<nb, 256, 0, c->stream>>>(c->n, c->pitch, boxd, c->x, c->bl_s, c->bl_sn, c->al_s,
                                                     c->al_sn, c->bonded_par, hb, ha, reps, arep, c->f,
                                                     c->vir, c->epot);
}
