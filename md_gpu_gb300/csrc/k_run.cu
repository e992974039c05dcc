/*
 * k_run.cu -- many steps of a small single system in one cooperative launch.
 *
 * A step of a few thousand atoms is a few microseconds of work, so the
 * ordinary form (a step graph of three or four kernels per step:
 * nve_leapfrog.cu:31-60 and neighborlist.cu:109-146 as separate launches)
 * spends its time on launches and the drain of each grid.  Here every block
 * stays on its SM for the whole run of steps and the phases are separated by
 * one grid barrier per step (two with Nose-Hoover, whose second half needs
 * the total kinetic energy in between):
 *
 *   [rebuild phases, when an atom moved >= skin/2]    md_rebuild.cuh
 *   pair (and bonded) forces of the block's atoms     md_pair.cuh
 *   leapfrog, or second kick of this step and first kick and drift of the
 *   next one; list check; kinetic energy              as k_integrate.cu
 *   barrier
 *
 * Positions are double buffered, so the forces of a step read one buffer
 * while the update writes the other.  A block owns 256 / TPA atoms; their
 * FP64 positions and velocities stay in the registers of its first
 * 3 * 256 / TPA threads, one (atom, axis) each, and go to memory only around
 * a rebuild and at the end.  One block more than the atoms need does the
 * bookkeeping of each step (record, thermostat) while the others compute
 * the next forces.  The arithmetic is the ordinary path's, operation for
 * operation, so a run is bit for bit the same.
 *
 * What bounds it is latency: the chain list entry -> position -> force ->
 * update -> barrier of one step, and the rebuilds (issue slots 18% busy at 982
 * ions and 32 lanes, 30% at 4080 and 16).  Whole md_step calls of
 * 100 steps against the step graphs: 500 LJ atoms 2.48 -> 0.83 ms, 4000 LJ
 * atoms 2.71 -> 1.00 ms, 982 ions 3.30 -> 1.01 ms; 20 steps of 5184 water
 * atoms 1.58 -> 0.74 ms.  Above the resident
 * blocks the step graphs are the only form (7998 ions: 16.4 us per step here,
 * 20.4 with 16 lanes per atom, where they do not fit).  Copying the block's
 * list rows to shared memory at each rebuild was no faster (12.8 against
 * 12.0 us per step for 982 ions at 8 lanes), nor was copying all positions
 * there each step (2048 LJ atoms: 8.5 against 7.6).
 */
#include <algorithm>

#include "md_bonded.cuh"
#include "md_pair.cuh"
#include "md_rebuild.cuh"
#include "md_thermo.cuh"

namespace {

constexpr int RUN_THREADS = CW_WARPS * 32;

/* The thermostat state of the run (the fields of md_devstate that
 * thermo_advance reads and writes), one copy per block. */
struct run_thermo {
    double temper, ke, pe, virial;
    double xi, eta, xi_a, eta_a;
    double vscale, lambda, lam_next, kick_scale;
};

/* f / 2, exactly (f in 2^-32 kJ/mol/A: a half kick's force).  The step is a
 * chain of FP64 latencies: adding a number whose last place is 1/2 converts
 * and halves in one addition (500 LJ atoms at 32 lanes 6.31 -> 6.10 us per
 * step, 4000 at 16 lanes 7.73 -> 7.28).  Where the FP64 pipe's rate binds instead (the integrator
 * kernels of large systems) the addition costs more than the conversion. */
__device__ __forceinline__ double half_of(long long f)
{
    if ((unsigned long long)(f + (1ll << 50)) < (1ull << 51))
        return __longlong_as_double(0x4328000000000000ll + f) - 3377699720527872.0;   /* 1.5 2^51 */
    double r;   /* as written, so that the compiler branches around it */
    asm volatile("cvt.rn.f64.s64 %0, %1;\n\tmul.rn.f64 %0, %0, 0d3FE0000000000000;" : "=&d"(r) : "l"(f));
    return r;
}

struct run_args {
    md_devstate *st;
    md_thermo *rec;
    int rec_cap;
    /* two sets of 64 words, used by alternate launches (each clears the
     * other): word 0 the barrier's arrivals; words 16 (s + 1) and 16 (s + 1)
     * + 1, s = 0, 1, 2, the kinetic energy of steps s modulo 3 and whether
     * an atom moved >= skin/2 in position updates s modulo 3 */
    unsigned long long *ctl;
    int parity;
    int nsteps, vv;
    float4 *buf0, *buf1;   /* positions now, and the other buffer */
    long long *f;
    float *vir;
    const float2 *ljtab;
    const float *bonded_par;
};

template <int KIND, int TPA, int B>
__global__ void __launch_bounds__(RUN_THREADS, 2) k_run_steps(md_kparams kp, pair_consts pc, thermo_par tp,
                                                              run_args a, rb_ptrs p)
{
    constexpr int NA = RUN_THREADS / TPA;   /* atoms per block */
    constexpr int NW = RUN_THREADS / 32;
    __shared__ float2 lj[MD_MAXTYPE * MD_MAXTYPE];
    __shared__ long long s_f[NA][3];
    __shared__ float s_x[NA][3];
    __shared__ long long s_ke[NW];
    __shared__ run_thermo s_ts;
    __shared__ int s_ok, s_flag;
    md_devstate *st = a.st;
    /* the same in every block: written only when a barrier runs out */
    if (*(volatile int *)&st->status != 0) return;
    if ((int)blockIdx.x == p.bar_drop) return;   /* test hook: the others' waits run out */
    const int t = threadIdx.x;
    const int i0 = blockIdx.x * NA;
    const bool book = blockIdx.x == gridDim.x - 1;   /* the bookkeeping block (no atoms) */
    unsigned long long *ctl = a.ctl + 64 * a.parity;
    unsigned long long target = 0;
    if (book && t < 64) a.ctl[64 * (a.parity ^ 1) + t] = 0ull;
    if (t < MD_MAXTYPE * MD_MAXTYPE) lj[t] = a.ljtab[t];
    if (t == 0) {
        s_ts.temper = st->temper;
        s_ts.ke = st->ke;
        s_ts.xi = st->xi;
        s_ts.eta = st->eta;
        s_ts.xi_a = st->xi_a;
        s_ts.eta_a = st->eta_a;
        s_ts.vscale = st->vscale;
        s_ts.lambda = st->lambda;
        s_ts.lam_next = st->lam_next;
        s_ts.kick_scale = st->kick_scale;
    }
    /* pair role: TPA lanes of atom i */
    const int i = i0 + t / TPA, lane = t % TPA;
    const bool active = i < kp.n;
    /* update role: axis d of atom iu; check role: atom i0 + t, t < NA */
    const int d = t / NA, iu = i0 + t % NA;
    const bool upd = d < 3 && iu < kp.n;
    const bool chk = t < NA && iu < kp.n;
    const size_t P = (size_t)kp.pitch, o = (size_t)(d < 3 ? d : 0) * P + iu;
    const axis_par ax = axis_of(d, kp.wlim, kp.boxd, kp.box2i);
    double x = 0.0, v = 0.0, m = 0.0, kick = 0.0;
    float q = 0.0f;
    float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 *pos = a.buf0, *next = a.buf1;   /* positions now, and where the update writes */
    auto load_state = [&]() {
        if (upd) {
            x = p.x[o];
            v = p.v[o];
            m = p.mass[iu];
            kick = p.kick[iu];
        }
        if (chk) {
            q = pos[iu].w;
            old = p.pos_old[iu];
        }
    };
    load_state();
    const unsigned long long bar_ns = p.bar_ns;
    int upd_no = 0;   /* position updates so far */
    /* Grid barrier.  Before it the block adds its kinetic energy to the sum
     * of step kslot modulo 3 (kslot >= 0) and, with moves, its rebuild
     * request to the flag of the current position update; after it s_flag
     * is that request.  A slot is cleared by the bookkeeping block before
     * the barrier of the step (update) that comes before its next use: its
     * last readers read it before they reached the barrier before that. */
    auto barrier = [&](long long ke, int kslot, bool moves, bool moved) -> bool {
        int any = 0;
        if (kslot >= 0) {
            for (int off = 16; off > 0; off >>= 1) ke += __shfl_down_sync(0xffffffffu, ke, off);
            if ((t & 31) == 0) s_ke[t >> 5] = ke;
        }
        if (moves) any = __syncthreads_or(moved ? 1 : 0);
        else __syncthreads();
        target += gridDim.x;
        unsigned long long *mv = ctl + 17 + 16 * (upd_no % 3);
        if (t == 0) {
            if (book) {
                if (kslot >= 0) ctl[16 + 16 * ((kslot + 1) % 3)] = 0ull;
                if (moves) ctl[17 + 16 * ((upd_no + 1) % 3)] = 0ull;
            } else {
                if (kslot >= 0) {
                    long long tot = 0;
                    for (int w = 0; w < NW; w++) tot += s_ke[w];
                    atomicAdd(ctl + 16 + 16 * (kslot % 3), (unsigned long long)tot);
                }
                if (any) *(volatile unsigned long long *)mv = 1ull;
            }
            red_release(ctl);
            s_ok = bar_wait(ctl, target, bar_ns, st);
            if (moves) s_flag = *(volatile unsigned long long *)mv != 0ull;
        }
        if (moves) upd_no++;
        __syncthreads();
        return s_ok != 0;
    };
    /* The bookkeeping of step k, whose kinetic energy is complete: the
     * bookkeeping block writes the record, the others follow only a
     * thermostat. */
    auto advance = [&](int k) {
        if (t != 0 || !(book || tp.berendsen || tp.nh)) return;
        const double ke0 = (double)(long long)*(volatile unsigned long long *)(ctl + 16 + 16 * (k % 3)) / MD_KFIX;
        double xi, eta, lam;
        const double ke = thermo_advance(kp.dt, tp, a.vv ? 1 : 0, ke0, 0.0, 0.0, &s_ts, &xi, &eta, &lam);
        if (!book) return;
        const double extra = tp.nh ? 0.5 * tp.q_nh * xi * xi + tp.ndf * RGAS * tp.t0 * eta : 0.0;
        write_record(tp, tp.inv_ndfr, ke, 0.0, 0.0, extra, xi, lam, *(volatile long long *)&st->step,
                     *(volatile int *)&st->builds, st, a.rec, a.rec_cap);
    };
    /* wrapped FP32 position of the update role, then pos4 and the list check */
    auto drift = [&]() -> bool {
        if (upd) {
            double xx = x + v * kp.dt;
            s_x[t % NA][d] = wrap(xx, ax.lim, ax.L, ax.two_over_l);
            x = xx;
        }
        __syncthreads();
        bool moved = false;
        if (chk) {
            const float4 pn = make_float4(s_x[t][0], s_x[t][1], s_x[t][2], q);
            next[iu] = pn;
            moved = md_rsq_exact(pn, old, kp) >= kp.rmaxdif;
        }
        float4 *tp4 = pos;
        pos = next;
        next = tp4;
        return moved;
    };
    __syncthreads();   /* lj and s_ts are set */
    /* a request left by the step before, or by whoever changed the list
     * since (the same in every block: cleared by a rebuild only, after the
     * first barrier) */
    int flag = *(volatile int *)&st->update;
    if (a.vv) {
        /* first half of the first step, from the forces in memory */
        if (upd) {
            if (s_ts.kick_scale != 1.0) v *= s_ts.kick_scale;
            v = fma(half_of(a.f[o]), kick, v);
        }
        const bool moved = drift();
        if (!barrier(0, -1, true, moved)) return;
        flag |= s_flag;
    }
    for (int k = 0; k < a.nsteps; k++) {
        if (flag) {
            if (upd) {
                p.x[o] = x;
                p.v[o] = v;
            }
            auto bar = [&]() { return barrier(0, -1, false, false); };
            if (!rebuild_phases(kp, st, p, pos, bar) || !bar()) return;
            load_state();
        }
        pair_total r = pair_sum<KIND, TPA, B, false, true, 1, false>(geom_kp{kp, pc}, kp.cap, active ? i : 0, active,
                                                                     lane, pos, p.type, p.nl, p.nl_n, lj);
        if (lane == 0) {
            if (active && (p.has_bonds || p.has_angles)) {
                const int nb = p.has_bonds ? p.bl_sn[i] : 0, na = p.has_angles ? p.al_sn[i] : 0;
                if (nb > 0 || na > 0) {
                    float fx, fy, fz, fw, fe;
                    bonded_atom<false>(i, kp.pitch, nb, na, kp.box, kp.boxi, pos, p.bl_s, p.al_s, a.bonded_par,
                                       fx, fy, fz, fw, fe);
                    r.fx += __float2ll_rn(fx * 4294967296.0f);
                    r.fy += __float2ll_rn(fy * 4294967296.0f);
                    r.fz += __float2ll_rn(fz * 4294967296.0f);
                    r.fw += fw;
                }
            }
            s_f[t / TPA][0] = r.fx;
            s_f[t / TPA][1] = r.fy;
            s_f[t / TPA][2] = r.fz;
            if (active && k == a.nsteps - 1) {
                a.f[i] = r.fx;
                a.f[P + i] = r.fy;
                a.f[2 * P + i] = r.fz;
                a.vir[i] = r.fw;
            }
        }
        __syncthreads();
        const bool last = k == a.nsteps - 1;
        long long ke = 0;
        bool moved = false;
        if (a.vv) {
            const double hf = upd ? half_of(s_f[t % NA][d]) : 0.0;
            if (upd) {
                v = fma(hf, kick, v);
                ke = ke_fix(m, v);
            }
            double scale = 1.0;
            if (tp.nh) {
                if (!barrier(ke, k, false, false)) return;
                advance(k);
                __syncthreads();
                scale = s_ts.kick_scale;
                ke = 0;
            }
            if (last && tp.nh) break;
            if (!last) {
                if (upd) {
                    if (scale != 1.0) v *= scale;
                    v = fma(hf, kick, v);
                }
                moved = drift();
            }
            if (!barrier(ke, tp.nh ? -1 : k, !last, moved)) return;
            if (!tp.nh) advance(k);
        } else {
            if (upd) {
                v += (double)s_f[t % NA][d] * kick;
                if (tp.berendsen) v *= s_ts.lam_next;
                ke = ke_fix(m, v);
            }
            moved = drift();
            if (!barrier(ke, k, true, moved)) return;
            advance(k);
        }
        flag = s_flag;
    }
    if (upd) {
        p.x[o] = x;
        p.v[o] = v;
    }
    if (book && t == 0) {
        if (!a.vv) st->update = flag;   /* the next run's first rebuild */
        st->temper = s_ts.temper;
        st->ke = s_ts.ke;
        st->xi = s_ts.xi;
        st->eta = s_ts.eta;
        st->xi_a = s_ts.xi_a;
        st->eta_a = s_ts.eta_a;
        st->vscale = s_ts.vscale;
        st->lambda = s_ts.lambda;
        st->lam_next = s_ts.lam_next;
        st->kick_scale = s_ts.kick_scale;
    }
}

/* The kernel for the context's lanes and entries per lane, null where there
 * is none.  Four entries per lane go two at a time like two, with the same
 * sums; one (16 lanes) goes one at a time, rounded otherwise. */
template <int KIND>
const void *run_kernel(int tpa, int depth)
{
    switch (tpa * 100 + depth) {
    case 802:
    case 804: return (const void *)k_run_steps<KIND, 8, 2>;
    case 1601: return (const void *)k_run_steps<KIND, 16, 1>;
    case 1602: return (const void *)k_run_steps<KIND, 16, 2>;
    case 3201: return (const void *)k_run_steps<KIND, 32, 1>;
    default: return nullptr;
    }
}

const void *run_kernel(const md_ctx *c)
{
    const int depth = md_pair_depth(c);
    return c->lkspace == 0 ? run_kernel<0>(c->pair_tpa, depth) : run_kernel<1>(c->pair_tpa, depth);
}

}  // namespace

/* Whether k_run_steps can run this system's steps: a single FP32 system
 * without the reciprocal sum whose atoms fit the blocks that are resident at
 * once (two of 256 threads per SM: 9696 atoms at 8 lanes on 152 SMs), rebuilt
 * warp per cell. */
bool md_fits_run(md_ctx *c)
{
    if (c->batch || c->fp64 || c->pme.on) return false;
    const void *k = run_kernel(c);
    if (!k || !md_rebuild_coop(c)) return false;
    const int key = c->pair_tpa * 100 + md_pair_depth(c);
    if (c->run_key != key) {   /* resident blocks, found once per kernel */
        int dev = 0, nsm = 0, occ = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, RUN_THREADS, 0);
        c->run_blocks = nsm * occ;
        c->run_key = key;
    }
    const int na = RUN_THREADS / c->pair_tpa;
    return (c->n + na - 1) / na + 1 <= c->run_blocks;
}

/* Whether md_step runs them there (eager launches, md_set_graphs, do not). */
bool md_can_run_small(md_ctx *c) { return c->use_graphs && md_fits_run(c); }

/* nsteps steps (no energies) in one launch; the positions end in pos4.
 * Returns false when the launch is refused (the caller takes the ordinary
 * path). */
bool launch_run_steps(md_ctx *c, const md_kparams &kp0, int nsteps)
{
    md_kparams kp = kp0;
    pair_consts pc = make_pair_consts(c);
    thermo_par tp = make_tp(c, 0);
    run_args a;
    a.st = c->st;
    a.rec = c->rec;
    a.rec_cap = c->rec_cap;
    a.ctl = c->run_ctl;
    a.parity = c->run_parity;
    a.nsteps = nsteps;
    a.vv = c->integrator != MD_LEAPFROG;
    a.buf0 = c->pos4;
    a.buf1 = c->pos4_alt;
    a.f = c->f;
    a.vir = c->vir;
    a.ljtab = (const float2 *)c->lj_dev;
    a.bonded_par = c->bonded_par;
    const int na = RUN_THREADS / c->pair_tpa, blocks = (c->n + na - 1) / na + 1;
    rb_ptrs p = make_rb_ptrs(c, blocks);
    void *args[] = {&kp, &pc, &tp, &a, &p};
    if (cudaLaunchCooperativeKernel(run_kernel(c), dim3(blocks), dim3(RUN_THREADS), args, 0, c->stream) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    c->run_parity ^= 1;
    if (nsteps & 1) std::swap(c->pos4, c->pos4_alt);
    return true;
}
