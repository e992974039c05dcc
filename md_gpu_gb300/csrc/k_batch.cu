/*
 * k_batch.cu -- pair forces and integrators of a batch of independent
 * replicas (md_create_batch), each with its own box, cutoffs, LJ table and
 * charges, advanced together by one launch per stage.
 *
 * The replicas' atoms are concatenated; a replica's atoms stay one
 * contiguous range through every re-sort.  Every launch here runs on a
 * replica-aligned grid (md_rep, grid_tab): a block covers atoms of one
 * replica only, so the replica's geometry and force-field constants are
 * uniform across the block (kept in registers, its LJ table in shared
 * memory), and each block adds its energy sums into its replica's
 * fixed-point accumulators.  The arithmetic per atom is the single-system arithmetic
 * (pair_sum, the leapfrog / velocity-Verlet updates of k_integrate.cu), so a
 * replica advances bit-for-bit as it would alone with the same tuning.
 */
#include "md_pair.cuh"
#include "md_thermo.cuh"

namespace {

/* Pair forces of a batch: block b holds 128/TPA atoms of replica tab[b].x
 * starting at tab[b].y.  Bound by issue slots and by the warps that hide the
 * gathers: at up to two entries per lane, eight blocks per SM at 64
 * registers (seven for the reaction field; one register set with energies).
 * 128 replicas of 512 to 8000 ions: 259 us per launch, 277 us at 72
 * registers, 312 unbounded, 342 before with one register set and 74. */
template <int KIND, int TPA, int B, bool ENERGY>
__global__ void __launch_bounds__(128, B > 2 ? 1 : ENERGY || KIND == 1 ? 8 : 7) k_pair_b(int cap, int pitch, int centered,
                                                const int2 *__restrict__ tab,
                                                const md_rep *__restrict__ reps,
                                                const float2 *__restrict__ ljr,
                                                const float4 *__restrict__ pos4,
                                                const int *__restrict__ type,
                                                const unsigned *__restrict__ nl,
                                                const int *__restrict__ nl_n, long long *f,
                                                float *vir, float *epot)
{
    __shared__ float2 lj[MD_MAXTYPE * MD_MAXTYPE];
    pdl_trigger();   /* the integrator may be scheduled; it waits for this grid */
    const int2 bt = tab[blockIdx.x];
    const md_rep &R = reps[bt.x];
    if (threadIdx.x < MD_MAXTYPE * MD_MAXTYPE)
        lj[threadIdx.x] = ljr[bt.x * MD_MAXTYPE * MD_MAXTYPE + threadIdx.x];
    const geom_reg g = rep_geom(R, centered != 0);
    const int end = R.atom0 + R.natom;
    __syncthreads();
    const int i = bt.y + (int)threadIdx.x / TPA, lane = (int)threadIdx.x % TPA;
    const bool active = i < end;
    pair_total t = pair_sum<KIND, TPA, B, ENERGY, true, (B > 2 ? 3 : ENERGY ? 1 : 2)>(g, cap, active ? i : bt.y, active, lane, pos4,
                                                  type, nl, nl_n, lj);
    const size_t P = (size_t)pitch;
    if (active && lane == 0) {
        f[i] = t.fx;
        f[P + i] = t.fy;
        f[2 * P + i] = t.fz;
        vir[i] = t.fw;
        if (ENERGY) epot[i] = t.fe;
    }
}

/* The end of an integrator block: as block_close, with the sums (nsum > 0)
 * going to the accumulators acc and a moved atom raising the replica's rebuild
 * request *upd too; the block is counted in *counter.  Returns true in every
 * thread of the block that is the last of `blocks`.  Thread 0 alone fences:
 * the other threads' stores are read by later kernels only. */
template <class CNT>
__device__ __forceinline__ bool block_close_b(long long a, long long b, long long c, int nsum, bool moved, int *upd,
                                              unsigned long long *acc, md_devstate *st, CNT *counter, CNT blocks,
                                              long long *sh)
{
    __shared__ bool last;
    if (nsum > 0) {
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            if (nsum > 1) {
                b += __shfl_down_sync(0xffffffffu, b, o);
                c += __shfl_down_sync(0xffffffffu, c, o);
            }
        }
        const int wp = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
        if (l == 0) {
            sh[wp] = a;
            sh[nw + wp] = b;
            sh[2 * nw + wp] = c;
        }
    }
    const int any = __syncthreads_or(moved ? 1 : 0);
    if (threadIdx.x == 0) {
        if (nsum > 0) {
            const int nw = blockDim.x >> 5;
            long long ta = 0, tb = 0, tc = 0;
            for (int k = 0; k < nw; k++) {
                ta += sh[k];
                tb += sh[nw + k];
                tc += sh[2 * nw + k];
            }
            atomicAdd(acc, (unsigned long long)ta);
            if (nsum > 1) {
                atomicAdd(acc + 1, (unsigned long long)tb);
                atomicAdd(acc + 2, (unsigned long long)tc);
            }
        }
        if (any) {
            st->update = 1;
            *upd = 1;
        }
        __threadfence();
        last = atomicAdd(counter, (CNT)1) == blocks - 1;
        __threadfence();
    }
    __syncthreads();
    return last;
}

/* Four sums over the first `count` threads of the block at once, the others'
 * terms being zero (each in the order of a whole block's shuffle tree); valid
 * in thread 0.  Called by every thread of the block. */
__device__ __forceinline__ void block_sum4(double (&v)[4], double (*sh)[4], int count)
{
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int nw = min((count + 31) >> 5, (int)(blockDim.x >> 5));
    if (w < nw) {
        for (int o = 16; o > 0; o >>= 1) {
            if (o >= count) continue;   /* adds zeros only */
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
        }
        if (l == 0)
#pragma unroll
            for (int q = 0; q < 4; q++) sh[w][q] = v[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = 0.0;
        for (int k = 0; k < nw; k++)
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] += sh[k][q];
    }
}

/* NPT: after a leapfrog step, axis d of the replica's box (L before it)
 * scaled by the factor the step applied to its positions, and what the
 * kernels derive from it: the FP32 box and its inverse as the reference
 * rounds it (simulation.cu:290-292), 2/L (twice 1/L, which rounds alike), the
 * wrap limit and the cell side.  The cell grid keeps its cell counts and
 * stencil until the host lays it out again (md_step does between chunks of
 * at most 128 steps, before the grid's 3% margin can be used up at the
 * per-step clamp of mu, 1e-4), so a box whose cells shrink below half the
 * list radius inside a chunk, or whose list radius exceeds half the box, can
 * no longer be listed correctly: that sets the sticky status 2, which the
 * host reports.  Runs in the last block of the replica's leapfrog, when no
 * other block reads its table entry any more. */
__device__ void npt_box_axis(md_rep &R, int d, double L0, double mu, md_devstate *st)
{
    const double L = L0 * mu, inv = 1.0 / L;
    const float box = (float)L, binlen = box / (float)R.ncell[d];
    R.boxd[d] = L;
    R.box[d] = box;
    R.boxi[d] = (float)inv;
    R.box2i[d] = 2.0 * inv;
    R.wlim[d] = 0.4999f * box;
    R.binlen[d] = binlen;
    if ((R.stencil[d] >= 0 && binlen < R.rl_half) || 2.0f * R.rl_half > 0.5f * box) atomicOr(&st->status, 2);
}

/* The end of a step for replica r, by the last of its blocks: thread 0 turns
 * the accumulators into KE, PE and virial (and clears them) and does the
 * replica's thermostat bookkeeping, a second warp the pressure and a third
 * the box (NPT).  FP64 arithmetic on a few values is a chain of latencies on
 * this GPU's narrow FP64 pipe: with every replica in the last block of the
 * batch this end took 24 us of a step of 128 replicas and 12 us of a single
 * NPT replica (one thread each); here replicas overlap with each other and
 * with the blocks still running: 482 -> 473 us per step of 128 replicas of
 * 512 to 8000 ions, 463 -> 457 of 512 replicas, 33.9 -> 28.0 of one NPT
 * system of 7986 ions.  The last replica to come then sums the batch's step
 * record over the replicas in a fixed order.  racc: 3 sums per replica, then
 * its count of finished blocks, then its 4 terms of the record.  Returns true
 * in thread 0 of the batch's last block. */
__device__ bool finalize_b(const md_kparams &kp, const thermo_par &tp, int mode, int nrep, int r, md_rep *reps,
                           md_repstate *repst, unsigned long long *racc, const step_io &io, double (*sh)[4])
{
    __shared__ bool all;
    const int wp = threadIdx.x >> 5, l = threadIdx.x & 31;
    md_devstate *st = io.st;
    md_rep &R = reps[r];
    md_repstate &S = repst[r];
    volatile unsigned long long *acc = racc + 3 * r;
    double *rtot = reinterpret_cast<double *>(racc + 4 * nrep);
    const bool npt = tp.npt && mode == 0;
    /* the step this record belongs to (the batch's last block advances it) */
    const long long step = ((volatile md_devstate *)st)->step;
    const int builds = ((volatile md_devstate *)st)->builds;
    double a = 0.0, b = 0.0, c = 0.0, L0 = 0.0, V = 0.0, mu0 = 1.0;
    if (l == 0 && wp < 2) {
        a = (double)(long long)acc[0] / MD_KFIX;
        b = (double)(long long)acc[1] / MD_EFIX;
        c = (double)(long long)acc[2] / MD_EFIX;
    }
    if (npt && wp == 1) V = R.boxd[0] * R.boxd[1] * R.boxd[2];
    if (npt && wp == 2 && l < 3) L0 = R.boxd[l];
    if (npt) mu0 = S.mu_next;
    __syncthreads();   /* read above, written below */
    double tot[4] = {0.0, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0) {
        acc[0] = acc[1] = acc[2] = 0ull;
        racc[3 * nrep + r] = 0ull;
        if (!tp.energy) b = c = 0.0;
        thermo_par t = tp;
        t.t0 = R.t0;
        t.ndf = R.ndf;
        t.q_nh = R.q_nh;
        t.inv_ndfr = R.inv_ndfr;
        t.inv_q = R.inv_q;
        double xi, eta, lam;
        const double ke = thermo_advance(kp.dt, t, mode, a, b, c, &S, &xi, &eta, &lam);
        const double ex = t.nh ? 0.5 * t.q_nh * xi * xi + t.ndf * RGAS * t.t0 * eta : 0.0;
        tot[0] = ke;
        tot[1] = b;
        tot[2] = c;
        tot[3] = ex;
        if (nrep > 1)
            for (int q = 0; q < 4; q++) rtot[4 * r + q] = tot[q];
        if (io.rep_hist && mode != 2) {
            double *hist = io.rep_hist + ((size_t)(step & (io.rec_cap - 1)) * nrep + r) * 3;
            hist[0] = ke;
            hist[1] = tp.energy ? b : 0.0;
            hist[2] = tp.energy ? ke + b + ex : 0.0;
        }
    } else if (npt && wp == 1 && l == 0) {
        /* P = (2 KE + sum_pairs F.r) / (3 V); c = sum over atoms of ff r^2,
         * every pair counted from both atoms; V of the box the forces saw */
        const double P = (2.0 * a + 0.5 * c) / (3.0 * V);
        double mu = 1.0 - R.mu_k * (R.p0 - P);
        mu = fmin(fmax(mu, 1.0 - R.mu_max), 1.0 + R.mu_max);
        S.pressure = P;
        S.mu_used = mu0;
        S.mu_next = mu;
    } else if (npt && R.npt && wp == 2 && l < 3) {
        npt_box_axis(R, l, L0, mu0, st);
    }
    if (nrep > 1) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            all = atomicAdd(io.counter, 1u) == (unsigned)nrep - 1u;
            __threadfence();
        }
        __syncthreads();
        if (!all) return false;
        for (int q = 0; q < 4; q++) tot[q] = 0.0;
        for (int k = threadIdx.x; k < nrep; k += blockDim.x)
            for (int q = 0; q < 4; q++) tot[q] += __ldcg(rtot + 4 * k + q);
        block_sum4(tot, sh, nrep);
    }
    if (threadIdx.x != 0) return false;
    const double KE = tot[0], PE = tot[1], W = tot[2], EX = tot[3];
    *io.counter = 0;
    st->ke = KE;
    if (tp.energy) {
        st->pe = PE;
        st->virial = W / 6.0;
    }
    if (mode == 2) return true;
    st->temper = 2.0 * KE * tp.inv_ndfr;
    write_record(tp, tp.inv_ndfr, KE, PE, W, EX, 0.0, 1.0, step, builds, st, io.rec, io.rec_cap);
    return true;
}

/* Leapfrog of a batch (k_leapfrog per replica, one thread per (atom, axis)):
 * Berendsen scale, box and skin of the block's replica. */
__global__ void __launch_bounds__(3 * MD_LA) k_leapfrog_b(md_kparams kp, thermo_par tp,
                                                         step_io io, int nrep,
                                                         const int2 *__restrict__ tab,
                                                         md_rep *reps,
                                                         md_repstate *repst, int *rep_upd,
                                                         unsigned long long *racc,
                                                         double *x, double *v,
                                                         const double *__restrict__ mass,
                                                         const double *__restrict__ kick,
                                                         float4 *pos4,
                                                         const long long *__restrict__ f,
                                                         const float *__restrict__ epot,
                                                         const float *__restrict__ vir)
{
    __shared__ double sh[3 * MD_LA / 32][4];
    __shared__ long long shl[3 * (3 * MD_LA / 32)];
    __shared__ float s_x[3][MD_LA];
    pdl_wait();   /* the forces of this step */
    const int2 bt = tab[blockIdx.x];
    const md_rep &R = reps[bt.x];
    const int d = threadIdx.x / MD_LA, a = threadIdx.x - d * MD_LA;
    const int s = bt.y + a;
    const bool act = s < R.atom0 + R.natom;
    const size_t o = (size_t)d * kp.pitch + s;
    long long ke = 0, pe = 0, w = 0;
    if (act) {
        axis_par ax = axis_of(d, R.wlim, R.boxd, R.box2i);
        double vv = v[o] + (double)f[o] * kick[s];
        if (tp.berendsen) vv *= repst[bt.x].lam_next;
        v[o] = vv;
        double xx = x[o] + vv * kp.dt;
        if (tp.npt) {
            /* Berendsen barostat: positions and box scaled by the factor the
             * last step's pressure gave; wrap into the scaled box */
            const double mu = repst[bt.x].mu_next;
            xx *= mu;
            ax.L *= mu;
            ax.lim = 0.4999f * (float)ax.L;
            /* an FP64 division, for the few atoms that wrap (27.1 -> 26.6 us
             * per step of one system of 7986 ions) */
            if (!(fabsf((float)xx) < ax.lim)) ax.two_over_l = 2.0 / ax.L;
        }
        s_x[d][a] = wrap(xx, ax.lim, ax.L, ax.two_over_l);
        x[o] = xx;
        ke = ke_fix(mass[s], vv);
        if (d == 0 && tp.energy) pe = llrint((double)epot[s] * MD_EFIX);
        if (d == 0 && (tp.energy || tp.npt)) w = llrint((double)vir[s] * MD_EFIX);
    }
    __syncthreads();
    bool moved = false;
    if (d == 0 && act) {
        float4 p = make_float4(s_x[0][a], s_x[1][a], s_x[2][a], pos4[s].w);
        pos4[s] = p;
        moved = md_rsq_box(p, io.pos_old[s], R.box, R.boxi) >= R.rmaxdif;
    }
    if (block_close_b(ke, pe, w, tp.energy || tp.npt ? 3 : 1, moved, rep_upd + bt.x, racc + 3 * bt.x, io.st,
                      racc + 3 * nrep + bt.x, (unsigned long long)R.nblk, shl) &&
        finalize_b(kp, tp, 0, nrep, bt.x, reps, repst, racc, io, sh))
        set_condition(io);
}

/* Velocity Verlet first half of a batch (k_vv_first per replica). */
__global__ void __launch_bounds__(3 * MD_LA) k_vv_first_b(md_kparams kp, step_io io,
                                                         const int2 *__restrict__ tab,
                                                         const md_rep *__restrict__ reps,
                                                         const md_repstate *__restrict__ repst,
                                                         int *rep_upd, double *x, double *v,
                                                         const double *__restrict__ kick,
                                                         float4 *pos4,
                                                         const long long *__restrict__ f)
{
    __shared__ float s_x[3][MD_LA];
    const int2 bt = tab[blockIdx.x];
    const md_rep &R = reps[bt.x];
    const int d = threadIdx.x / MD_LA, a = threadIdx.x - d * MD_LA;
    const int s = bt.y + a;
    const bool act = s < R.atom0 + R.natom;
    const size_t o = (size_t)d * kp.pitch + s;
    const double scale = repst[bt.x].kick_scale;
    if (act) {
        const axis_par ax = axis_of(d, R.wlim, R.boxd, R.box2i);
        double vv = v[o];
        if (scale != 1.0) vv *= scale;
        vv += (double)f[o] * (0.5 * kick[s]);
        v[o] = vv;
        double xx = x[o] + vv * kp.dt;
        s_x[d][a] = wrap(xx, ax.lim, ax.L, ax.two_over_l);
        x[o] = xx;
    }
    __syncthreads();
    bool moved = false;
    if (d == 0 && act) {
        float4 p = make_float4(s_x[0][a], s_x[1][a], s_x[2][a], pos4[s].w);
        pos4[s] = p;
        moved = md_rsq_box(p, io.pos_old[s], R.box, R.boxi) >= R.rmaxdif;
    }
    if (!io.has_cond) {   /* nothing to do after the last block */
        if (__syncthreads_or(moved ? 1 : 0) && threadIdx.x == 0) {
            io.st->update = 1;
            rep_upd[bt.x] = 1;
        }
        return;
    }
    if (block_close_b(0, 0, 0, 0, moved, rep_upd + bt.x, nullptr, io.st, io.counter, gridDim.x, nullptr) &&
        threadIdx.x == 0) {
        set_condition(io);
        *io.counter = 0;
    }
}

/* Velocity Verlet second half of a batch (k_vv_second per replica); do_kick
 * = 0 observes the state only. */
__global__ void __launch_bounds__(3 * MD_LA, 4) k_vv_second_b(md_kparams kp, thermo_par tp,
                                                          int do_kick, step_io io, int nrep,
                                                          const int2 *__restrict__ tab,
                                                          md_rep *reps, md_repstate *repst,
                                                          unsigned long long *racc, double *v,
                                                          const double *__restrict__ mass,
                                                          const double *__restrict__ kick,
                                                          const long long *__restrict__ f,
                                                          const float *__restrict__ epot,
                                                          const float *__restrict__ vir)
{
    __shared__ double sh[3 * MD_LA / 32][4];
    __shared__ long long shl[3 * (3 * MD_LA / 32)];
    pdl_wait();   /* the forces of this step */
    const int2 bt = tab[blockIdx.x];
    const md_rep &R = reps[bt.x];
    const int d = threadIdx.x / MD_LA, a = threadIdx.x - d * MD_LA;
    const int s = bt.y + a;
    const size_t o = (size_t)d * kp.pitch + s;
    long long ke = 0, pe = 0, w = 0;
    if (s < R.atom0 + R.natom) {
        double vv = v[o];
        if (do_kick) {
            vv += (double)f[o] * (0.5 * kick[s]);
            v[o] = vv;
        } else {
            vv *= repst[bt.x].vscale;
        }
        ke = ke_fix(mass[s], vv);
        if (d == 0 && tp.energy) {
            pe = llrint((double)epot[s] * MD_EFIX);
            w = llrint((double)vir[s] * MD_EFIX);
        }
    }
    if (block_close_b(ke, pe, w, tp.energy ? 3 : 1, false, nullptr, racc + 3 * bt.x, io.st, racc + 3 * nrep + bt.x,
                      (unsigned long long)R.nblk, shl))
        finalize_b(kp, tp, do_kick ? 1 : 2, nrep, bt.x, reps, repst, racc, io, sh);
}

/* k_vv_second_b and the next step's k_vv_first_b as one kernel (k_vv_mid per
 * replica). */
__global__ void __launch_bounds__(3 * MD_LA, 4) k_vv_mid_b(md_kparams kp, thermo_par tp, step_io io, int nrep,
                                                          const int2 *__restrict__ tab, md_rep *reps,
                                                          md_repstate *repst, int *rep_upd,
                                                          unsigned long long *racc, double *x, double *v,
                                                          const double *__restrict__ mass,
                                                          const double *__restrict__ kick, float4 *pos4,
                                                          const long long *__restrict__ f,
                                                          const float *__restrict__ epot,
                                                          const float *__restrict__ vir)
{
    __shared__ double sh[3 * MD_LA / 32][4];
    __shared__ long long shl[3 * (3 * MD_LA / 32)];
    __shared__ float s_x[3][MD_LA];
    pdl_wait();   /* the forces of this step */
    const int2 bt = tab[blockIdx.x];
    const md_rep &R = reps[bt.x];
    const int d = threadIdx.x / MD_LA, a = threadIdx.x - d * MD_LA;
    const int s = bt.y + a;
    const bool act = s < R.atom0 + R.natom;
    const size_t o = (size_t)d * kp.pitch + s;
    long long ke = 0, pe = 0, w = 0;
    if (act) {
        const axis_par ax = axis_of(d, R.wlim, R.boxd, R.box2i);
        const double fd = (double)f[o], hk = 0.5 * kick[s];
        double vv = fma(fd, hk, v[o]);
        ke = ke_fix(mass[s], vv);
        vv = fma(fd, hk, vv);
        v[o] = vv;
        double xx = x[o] + vv * kp.dt;
        s_x[d][a] = wrap(xx, ax.lim, ax.L, ax.two_over_l);
        x[o] = xx;
        if (d == 0 && tp.energy) {
            pe = llrint((double)epot[s] * MD_EFIX);
            w = llrint((double)vir[s] * MD_EFIX);
        }
    }
    __syncthreads();
    bool moved = false;
    if (d == 0 && act) {
        float4 p = make_float4(s_x[0][a], s_x[1][a], s_x[2][a], pos4[s].w);
        pos4[s] = p;
        moved = md_rsq_box(p, io.pos_old[s], R.box, R.boxi) >= R.rmaxdif;
    }
    if (block_close_b(ke, pe, w, tp.energy ? 3 : 1, moved, rep_upd + bt.x, racc + 3 * bt.x, io.st,
                      racc + 3 * nrep + bt.x, (unsigned long long)R.nblk, shl))
        finalize_b(kp, tp, 1, nrep, bt.x, reps, repst, racc, io, sh);
}

template <int KIND, bool ENERGY>
void pair_dispatch_b(md_ctx *c, const md_kparams &kp)
{
    const int k = md_grid_index(128 / c->pair_tpa);
    const int2 *tab = c->grid_tab + c->grid_off[k];
    const int nb = c->grid_cnt[k];
    switch (c->pair_tpa * 100 + md_pair_depth(c)) {
#define MD_PAIR_B_CASE(T, BB)                                                                    \
    case T * 100 + BB:                                                                           \
        k_pair_b<KIND, T, BB, ENERGY><<<nb, 128, 0, c->stream>>>(                                \
            kp.cap, kp.pitch, kp.centered, tab, c->reps_dev, c->ljr_dev, c->pos4, c->type, c->nl, \
            c->nl_n, c->f, c->vir, c->epot);                                                     \
        break;
        MD_PAIR_B_CASE(1, 8)
        MD_PAIR_B_CASE(2, 8)
        MD_PAIR_B_CASE(4, 4)
        MD_PAIR_B_CASE(4, 8)
        MD_PAIR_B_CASE(8, 2)
        MD_PAIR_B_CASE(8, 4)
        MD_PAIR_B_CASE(16, 1)
        MD_PAIR_B_CASE(16, 2)
        MD_PAIR_B_CASE(32, 1)
#undef MD_PAIR_B_CASE
    default:
        break;
    }
}

inline const int2 *grid_int(const md_ctx *c) { return c->grid_tab + c->grid_off[md_grid_index(MD_LA)]; }
inline int grid_int_blocks(const md_ctx *c) { return c->grid_cnt[md_grid_index(MD_LA)]; }

}  // namespace

void launch_forces_b(md_ctx *c, const md_kparams &kp, bool energy, int terms)
{
    if ((terms & MD_TERM_PAIR) && c->fp64) {
        launch_pair64(c, energy);
    } else if (terms & MD_TERM_PAIR) {
        if (c->lkspace == 0) {
            if (energy) pair_dispatch_b<0, true>(c, kp);
            else pair_dispatch_b<0, false>(c, kp);
        } else {
            if (energy) pair_dispatch_b<1, true>(c, kp);
            else pair_dispatch_b<1, false>(c, kp);
        }
    } else {
        cudaMemsetAsync(c->f, 0, sizeof(long long) * 3 * (size_t)c->pitch, c->stream);
        cudaMemsetAsync(c->vir, 0, sizeof(float) * (size_t)c->pitch, c->stream);
        cudaMemsetAsync(c->epot, 0, sizeof(float) * (size_t)c->pitch, c->stream);
    }
    launch_bonded(c, kp, energy, terms);
}

void launch_leapfrog_b(md_ctx *c, const md_kparams &kp, int energy, unsigned long long cond,
                       int has_cond)
{
    md_launch_pdl(k_leapfrog_b, dim3(grid_int_blocks(c)), dim3(3 * MD_LA), c->stream, kp,
                  make_tp(c, energy), make_io(c, cond, has_cond), c->nrep, grid_int(c),
                  c->reps_dev, c->repst, c->rep_upd, c->racc, c->x, c->v,
                  (const double *)c->mass, (const double *)c->kick, c->pos4,
                  (const long long *)c->f, (const float *)c->epot, (const float *)c->vir);
}

void launch_vv_first_b(md_ctx *c, const md_kparams &kp, unsigned long long cond, int has_cond)
{
    k_vv_first_b<<<grid_int_blocks(c), 3 * MD_LA, 0, c->stream>>>(kp, make_io(c, cond, has_cond),
                                                           grid_int(c), c->reps_dev, c->repst,
                                                           c->rep_upd, c->x, c->v, c->kick, c->pos4,
                                                           c->f);
}

void launch_vv_mid_b(md_ctx *c, const md_kparams &kp, int energy)
{
    md_launch_pdl(k_vv_mid_b, dim3(grid_int_blocks(c)), dim3(3 * MD_LA), c->stream, kp, make_tp(c, energy),
                  make_io(c, 0, 0), c->nrep, grid_int(c), c->reps_dev, c->repst, c->rep_upd, c->racc, c->x, c->v,
                  (const double *)c->mass, (const double *)c->kick, c->pos4, (const long long *)c->f,
                  (const float *)c->epot, (const float *)c->vir);
}

void launch_vv_second_b(md_ctx *c, const md_kparams &kp, int energy, int kick)
{
    md_launch_pdl(k_vv_second_b, dim3(grid_int_blocks(c)), dim3(3 * MD_LA), c->stream, kp,
                  make_tp(c, energy), kick, make_io(c, 0, 0), c->nrep, grid_int(c),
                  c->reps_dev, c->repst, c->racc, c->v, (const double *)c->mass,
                  (const double *)c->kick, (const long long *)c->f, (const float *)c->epot,
                  (const float *)c->vir);
}
