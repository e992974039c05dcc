/*
 * k_forces.cu -- pair (LJ + Wolf / reaction field) and bonded forces.
 *
 * Pair forces follow pair_forces.cu:34-205: for each listed j inside rc,
 *   Wolf:  ff = qfac qi qj ([2a/sqrt(pi) r + P5(t) t] e^{-a^2 r^2} / r - W) / r^2,
 *          t = 1/(1 + p a r), P5 = A&S 7.1.26 (simulation.h:39-44),
 *   RF:    ff = qfac qi qj (1/r - k_rf r^2) / r^2,
 *   + LJ:  ff += lj1 r^-14 - lj2 r^-8,
 * F_i += ff d, w_i += ff r^2.  Arithmetic is FP32 (contraction allowed);
 * the per-atom sums are taken in FP32 over chunks of a few neighbours and
 * added into int64 fixed point, so the result does not depend on how the
 * list is split across threads.  TPA lanes share one atom (lane l takes list
 * entries l, l+TPA, ...) and combine with shuffles.
 *
 * Bonded forces follow bonded_forces.cu:34-193 as per-atom gathers over
 * per-atom lists (each bond seen from both atoms, each angle from all three);
 * the centre-atom branch uses the role of the entry being processed.
 */
#include "md_bonded.cuh"
#include "md_pair.cuh"

namespace {

/* The pair forces of atom ii (see pair_sum) written to the force arrays. */
template <int KIND, int TPA, int B, bool ENERGY>
__global__ void __launch_bounds__(128) k_pair(md_kparams kp, pair_consts pc,
                                              const float4 *__restrict__ pos4,
                                              const int *__restrict__ type,
                                              const unsigned *__restrict__ nl,
                                              const int *__restrict__ nl_n,
                                              const float2 *__restrict__ ljtab, long long *f,
                                              float *vir, float *epot)
{
    __shared__ float2 lj[MD_MAXTYPE * MD_MAXTYPE];
    pdl_trigger();   /* the integrator may be scheduled; it waits for this grid */
    if (threadIdx.x < MD_MAXTYPE * MD_MAXTYPE) lj[threadIdx.x] = ljtab[threadIdx.x];
    __syncthreads();
    int gt = blockIdx.x * blockDim.x + threadIdx.x;
    int i = gt / TPA, lane = gt % TPA;
    bool active = i < kp.n;
    pair_total t = pair_sum<KIND, TPA, B, ENERGY>(geom_kp{kp, pc}, kp.cap, active ? i : 0, active, lane, pos4, type,
                                                  nl, nl_n, lj);
    const size_t P = (size_t)kp.pitch;
    if (active && lane == 0) {
        f[i] = t.fx;
        f[P + i] = t.fy;
        f[2 * P + i] = t.fz;
        vir[i] = t.fw;
        if (ENERGY) epot[i] = t.fe;
    }
}

/* Bonds and angles (bonded_atom), one thread per sorted atom, added into the
 * fixed-point forces.  Latency bound (one chain of gathers and an arc cosine
 * per atom), so it is launched as a programmatic dependent of the pair kernel:
 * its blocks compute from the positions while that one drains, and wait for it
 * before they add (every block waits, so that what follows this kernel also
 * follows the pair kernel).  98304 water atoms: 164.7 -> 161.2 us per step.
 * In a batch (reps non-null) the minimum image uses the atom's replica box. */
template <bool ENERGY>
__global__ void __launch_bounds__(256) k_bonded(md_kparams kp, const float4 *pos4,
                         const int2 *__restrict__ bl_s, const int *__restrict__ bl_sn,
                         const int4 *__restrict__ al_s, const int *__restrict__ al_sn,
                         const float *__restrict__ par, int has_bonds, int has_angles,
                         const md_rep *__restrict__ reps, const int *__restrict__ arep,
                         long long *f, float *vir, float *epot)
{
    pdl_trigger();   /* the integrator may be scheduled; it waits for this grid */
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int P = kp.pitch;
    const int nb = s < kp.n && has_bonds ? bl_sn[s] : 0;
    const int na = s < kp.n && has_angles ? al_sn[s] : 0;
    const bool any = nb > 0 || na > 0;
    float fx = 0.0f, fy = 0.0f, fz = 0.0f, fw = 0.0f, fe = 0.0f;
    if (any) {
        const float *box = reps ? reps[arep[s]].box : kp.box, *boxi = reps ? reps[arep[s]].boxi : kp.boxi;
        bonded_atom<ENERGY>(s, P, nb, na, box, boxi, pos4, bl_s, al_s, par, fx, fy, fz, fw, fe);
    }
    pdl_wait();   /* the pair forces */
    if (!any) return;
    f[s] += __float2ll_rn(fx * 4294967296.0f);
    f[P + s] += __float2ll_rn(fy * 4294967296.0f);
    f[2 * P + s] += __float2ll_rn(fz * 4294967296.0f);
    vir[s] += fw;
    if (ENERGY) epot[s] += fe;
}

template <int KIND, bool ENERGY>
void pair_dispatch(md_ctx *c, const md_kparams &kp, const pair_consts &pc)
{
    long long threads = (long long)kp.n * c->pair_tpa;
    int nb = (int)((threads + 127) / 128);
    const float2 *lj = (const float2 *)c->lj_dev;
    const int key = c->pair_tpa * 100 + md_pair_depth(c);
    switch (key) {
#define MD_PAIR_CASE(T, BB)                                                                      \
    case T * 100 + BB:                                                                           \
        k_pair<KIND, T, BB, ENERGY><<<nb, 128, 0, c->stream>>>(                                  \
            kp, pc, c->pos4, c->type, c->nl, c->nl_n, lj, c->f, c->vir, c->epot);                \
        break;
        MD_PAIR_CASE(1, 8)
        MD_PAIR_CASE(2, 8)
        MD_PAIR_CASE(4, 4)
        MD_PAIR_CASE(4, 8)
        MD_PAIR_CASE(8, 2)
        MD_PAIR_CASE(8, 4)
        MD_PAIR_CASE(16, 1)
        MD_PAIR_CASE(16, 2)
        MD_PAIR_CASE(32, 1)
#undef MD_PAIR_CASE
    default:
        break;
    }
}

}  // namespace

void launch_forces(md_ctx *c, const md_kparams &kp, bool energy, int terms)
{
    if (c->batch) {
        launch_forces_b(c, kp, energy, terms);
        return;
    }
    pair_consts pc = make_pair_consts(c);
    const bool recip = c->pme.on && (terms & MD_TERM_RECIP);
    if (recip) launch_pme_start(c, kp);
    if ((terms & MD_TERM_PAIR) && c->fp64) {
        launch_pair64(c, energy);
    } else if (terms & MD_TERM_PAIR) {
        if (c->lkspace == 0) {
            if (energy) pair_dispatch<0, true>(c, kp, pc);
            else pair_dispatch<0, false>(c, kp, pc);
        } else {
            if (energy) pair_dispatch<1, true>(c, kp, pc);
            else pair_dispatch<1, false>(c, kp, pc);
        }
    } else {
        cudaMemsetAsync(c->f, 0, sizeof(long long) * 3 * (size_t)c->pitch, c->stream);
        cudaMemsetAsync(c->vir, 0, sizeof(float) * (size_t)c->pitch, c->stream);
        cudaMemsetAsync(c->epot, 0, sizeof(float) * (size_t)c->pitch, c->stream);
    }
    launch_bonded(c, kp, energy, terms);
    if (recip) launch_pme_finish(c, kp, energy);
}

void launch_bonded(md_ctx *c, const md_kparams &kp, bool energy, int terms)
{
    int hb = (terms & MD_TERM_BOND) ? c->has_bonds : 0;
    int ha = (terms & MD_TERM_ANGLE) ? c->has_angles : 0;
    if ((hb || ha) && c->fp64) {
        launch_bonded64(c, energy, hb, ha);
    } else if (hb || ha) {
        int nb = (kp.n + 255) / 256;
        const md_rep *reps = c->batch ? c->reps_dev : nullptr;
        const int *arep = c->batch ? c->arep : nullptr;
        md_launch_pdl(energy ? k_bonded<true> : k_bonded<false>, dim3(nb), dim3(256), c->stream, kp,
                      (const float4 *)c->pos4, (const int2 *)c->bl_s, (const int *)c->bl_sn, (const int4 *)c->al_s,
                      (const int *)c->al_sn, (const float *)c->bonded_par, hb, ha, reps, arep, c->f, c->vir, c->epot);
    }
}
