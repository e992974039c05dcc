/*
 * k_cells.cu -- neighbour-list maintenance: displacement check, cell binning,
 * Hilbert-order atom sort and the list build.
 *
 * Semantics follow neighborlist.cu: the list of atom i holds every j != i,
 * not excluded, with FP32 min-image r^2 < rskinsq evaluated exactly as the
 * reference writes it (neighborlist.cu:268-283; each operation rounded on its
 * own, so the set is bit-identical to the O(N^2) kernel's); it is rebuilt when
 * any atom moved >= skin/2 since the last build (neighborlist.cu:157-176).
 * Unlike the reference the candidates come from the 27..125 cells around i
 * (cells of side >= rl/2), the atoms are re-sorted along a Hilbert curve of
 * cells at every build, and the rebuild decision never leaves the device.
 */
#include <algorithm>

#include "md_rebuild.cuh"

namespace {

__global__ void k_check(md_kparams kp, const float4 *__restrict__ pos4,
                        const float4 *__restrict__ pos_old, md_devstate *st)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    if (md_rsq_exact(pos4[i], pos_old[i], kp) >= kp.rmaxdif) st->update = 1;
}

/* Cell rank (Hilbert order) of every atom and the per-cell counts. */
__global__ void k_cell_key(md_kparams kp, const md_devstate *st, int always,
                           const float4 *__restrict__ pos4, const int *__restrict__ cell_rank,
                           int *key, int *cell_count)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    key_one(kp, i, pos4, cell_rank, key, cell_count);
}

/* The same for a batch: each atom is tested with its replica's box and skin. */
__global__ void k_check_b(int n, const md_rep *__restrict__ reps, const int *__restrict__ arep,
                          const float4 *__restrict__ pos4, const float4 *__restrict__ pos_old,
                          md_devstate *st, int *rep_upd)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = arep[i];
    const md_rep &R = reps[r];
    if (md_rsq_box(pos4[i], pos_old[i], R.box, R.boxi) >= R.rmaxdif) {
        st->update = 1;
        rep_upd[r] = 1;
    }
}

/* Cell keys of a batch: the replica's cell grid, ranks offset by its first
 * cell, so every replica's cells (and atoms) stay one contiguous range.
 * Only replicas with a rebuild request are re-binned; every other replica
 * keeps its order, cell ranges and list rows untouched by all build passes. */
__global__ void k_cell_key_b(int n, int centered, const md_rep *__restrict__ reps,
                             const int *__restrict__ arep,
                             const md_devstate *st, int always, const int *__restrict__ rep_upd,
                             const float4 *__restrict__ pos4, const int *__restrict__ cell_rank,
                             int *key, int *cell_count)
{
    if (!always && !st->update) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int rep = arep[i];
    if (!rep_upd[rep]) return;
    const md_rep &R = reps[rep];
    float4 p = pos4[i];
    int cx = cell_of(cell_coord(p.x, R.box[0], R.boxi[0], centered), R.box[0], R.binlen[0], R.ncell[0]);
    int cy = cell_of(cell_coord(p.y, R.box[1], R.boxi[1], centered), R.box[1], R.binlen[1], R.ncell[1]);
    int cz = cell_of(cell_coord(p.z, R.box[2], R.boxi[2], centered), R.box[2], R.binlen[2], R.ncell[2]);
    int r = cell_rank[R.cell0 + cx + R.ncell[0] * (cy + R.ncell[1] * cz)];
    key[i] = r;
    atomicAdd(&cell_count[r], 1);
}

/* Per-replica exclusive scan of the cell counts, one warp per replica being
 * rebuilt: its cells start at its first atom.  Counters are zeroed for the
 * next build. */
__global__ void k_cell_scan_b(const md_devstate *st, int always, int nrep,
                              const md_rep *__restrict__ reps, const int *__restrict__ rep_upd,
                              int *cell_count, int *cell_start, int *cell_fill)
{
    if (!always && !st->update) return;
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= nrep || !rep_upd[r]) return;
    const md_rep &R = reps[r];
    int run = R.atom0;
    for (int k0 = 0; k0 < R.ncells; k0 += 32) {
        const int k = k0 + lane;
        const int c = R.cell0 + k;
        int cnt = k < R.ncells ? cell_count[c] : 0;
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (k < R.ncells) {
            cell_start[c] = run + incl - cnt;
            cell_count[c] = 0;
            cell_fill[c] = 0;
        }
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) cell_start[R.cell0 + R.ncells] = run;   /* = the next replica's first atom */
}

/* Rebuild every replica of a batch (forced builds). */
__global__ void k_flag_all(int *rep_upd, int nrep)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < nrep) rep_upd[r] = 1;
}

/* Ends a rebuild of a batch: counts the build and the rebuilt replicas'
 * builds and clears the requests. */
__global__ void k_clear_update_b(md_devstate *st, int always, int *rep_upd, md_repstate *repst,
                                 int nrep)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) {
        if (always || st->update) st->builds += 1;
        st->update = 0;
        st->cell_next = 0;
    }
    if (r < nrep && rep_upd[r]) {
        repst[r].builds += 1;
        rep_upd[r] = 0;
    }
}

/* The scan as its own pass (one block of 1024 threads); cell_start has
 * ncells + 1 entries. */
__global__ void __launch_bounds__(1024) k_cell_scan(md_kparams kp, md_devstate *st, int always,
                                                    int ncells, int *cell_count, int *cell_start,
                                                    int *cell_fill)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    const int total = scan_cells<1024>(ncells, cell_count, cell_start, cell_fill);
    if (threadIdx.x == 0) {
        cell_start[ncells] = total;
        st->builds += 1;
    }
}

/* In a batch (arep, rep_upd non-null) the passes below touch only the atoms
 * and cells of replicas being rebuilt. */
__global__ void k_cell_scatter(md_kparams kp, const md_devstate *st, int always,
                               const int *__restrict__ key, const int *__restrict__ cell_start,
                               int *cell_fill, int *src, const int *__restrict__ arep,
                               const int *__restrict__ rep_upd)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp.n) return;
    if (arep && !rep_upd[arep[i]]) return;
    int r = key[i];
    src[cell_start[r] + atomicAdd(&cell_fill[r], 1)] = i;
}

__global__ void k_cell_order(md_kparams kp, const md_devstate *st, int always, int ncells,
                             const int *__restrict__ cell_start, const int *__restrict__ perm,
                             int *src, const int *__restrict__ crep, const int *__restrict__ rep_upd)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    const int lane = threadIdx.x & 31, nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < ncells; c += nw) {
        order_cell(c, cell_start, perm, src, crep, rep_upd, lane);
        __syncwarp();
    }
}

__global__ void k_permute(md_kparams kp, const md_devstate *st, int always,
                          const int *__restrict__ src, const double *__restrict__ x,
                          const double *__restrict__ v, const double *__restrict__ mass,
                          const double *__restrict__ kick,
                          const float4 *__restrict__ pos4, const int *__restrict__ perm,
                          const int *__restrict__ type, double *tmp_d, float4 *tmp4, int *tmp_i,
                          const int *__restrict__ arep, const int *__restrict__ rep_upd)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= kp.n) return;
    if (arep && !rep_upd[arep[s]]) return;   /* atoms stay inside their replica's range */
    permute_one(kp, s, src[s], x, v, mass, kick, pos4, perm, type, tmp_d, tmp4, tmp_i);
}

__global__ void k_copyback(md_kparams kp, const md_devstate *st, int always,
                           const double *__restrict__ tmp_d, const float4 *__restrict__ tmp4,
                           const int *__restrict__ tmp_i, double *x, double *v, double *mass,
                           double *kick, float4 *pos4, int *perm, int *iperm, int *type,
                           const int *__restrict__ arep, const int *__restrict__ rep_upd)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= kp.n) return;
    if (arep && !rep_upd[arep[s]]) return;
    copyback_one(kp, s, tmp_d, tmp4, tmp_i, x, v, mass, kick, pos4, perm, iperm, type);
}

/* Exclusions and bonded lists re-expressed in the new sorted indices. */
__global__ void k_remap(md_kparams kp, const md_devstate *st, int always,
                        const int *__restrict__ perm, const int *__restrict__ iperm,
                        const uint4 *__restrict__ excl_orig, uint4 *excl_s,
                        const int2 *__restrict__ bl_o, const int *__restrict__ bl_on, int2 *bl_s,
                        int *bl_sn, const int4 *__restrict__ al_o, const int *__restrict__ al_on,
                        int4 *al_s, int *al_sn, int has_bonds, int has_angles)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= kp.n) return;
    remap_one(kp, s, perm, iperm, excl_orig, excl_s, bl_o, bl_on, bl_s, bl_sn, al_o, al_on, al_s, al_sn,
              has_bonds, has_angles);
}

/* Ends a rebuild (or a step without one): the next step's check sets the
 * request again. */
__global__ void k_clear_update(md_devstate *st)
{
    pdl_wait();
    st->update = 0;
    st->cell_next = 0;
}

/* First node of a captured step graph: the rebuild condition of its first
 * step comes from the check done by the step before the graph. */
__global__ void k_set_condition(cudaGraphConditionalHandle h, const md_devstate *st)
{
    cudaGraphSetConditional(h, st->update ? 1u : 0u);
}

/* List build: TPA lanes per atom scan the stencil cells; lane l tests the
 * candidates l, l+TPA, ... of each cell and the lanes append their hits in
 * candidate order with a ballot, so the list order is fixed by the cell
 * traversal order alone. */
template <int TPA>
__global__ void __launch_bounds__(256) k_build_list(
    md_kparams kp, md_devstate *st, int always, const float4 *__restrict__ pos4,
    const int *__restrict__ type, const uint4 *__restrict__ excl_s,
    const int *__restrict__ cell_rank, const int *__restrict__ cell_start,
    const unsigned *__restrict__ type_mask, unsigned *nl, int *nl_n, float4 *pos_old)
{
    pdl_wait();      /* launched after the previous pass (programmatic launch) */
    pdl_trigger();
    if (!always && !st->update) return;
    int gt = blockIdx.x * blockDim.x + threadIdx.x;
    int i = gt / TPA, lane = gt % TPA;
    int lane_w = threadIdx.x & 31;
    unsigned gmask = (TPA == 32) ? 0xffffffffu : (((1u << TPA) - 1u) << (lane_w & ~(TPA - 1)));
    bool active = i < kp.n;
    int ii = active ? i : 0;
    float4 p = pos4[ii];
    int ti = type[ii];
    uint4 ex = excl_s[ii];
    unsigned tmask = type_mask[ti];
    int c3[3];
    for (int d = 0; d < 3; d++)
        c3[d] = cell_of(cell_coord(d == 0 ? p.x : (d == 1 ? p.y : p.z), kp.box[d], kp.boxi[d], kp.centered),
                        kp.box[d], kp.binlen[d], kp.ncell[d]);
    int lo[3], hi[3];
    for (int d = 0; d < 3; d++) {
        if (kp.stencil[d] < 0) { lo[d] = 0; hi[d] = kp.ncell[d] - 1; }
        else { lo[d] = c3[d] - kp.stencil[d]; hi[d] = c3[d] + kp.stencil[d]; }
    }
    int cnt = 0;
    for (int zz = lo[2]; zz <= hi[2]; zz++) {
        int cz = zz < 0 ? zz + kp.ncell[2] : (zz >= kp.ncell[2] ? zz - kp.ncell[2] : zz);
        for (int yy = lo[1]; yy <= hi[1]; yy++) {
            int cy = yy < 0 ? yy + kp.ncell[1] : (yy >= kp.ncell[1] ? yy - kp.ncell[1] : yy);
            for (int xx = lo[0]; xx <= hi[0]; xx++) {
                int cx = xx < 0 ? xx + kp.ncell[0] : (xx >= kp.ncell[0] ? xx - kp.ncell[0] : xx);
                int r = cell_rank[cx + kp.ncell[0] * (cy + kp.ncell[1] * cz)];
                int b = cell_start[r], e = cell_start[r + 1];
                for (int j0 = b; j0 < e; j0 += TPA) {
                    int j = j0 + lane;
                    bool ok = false;
                    unsigned entry = 0;
                    if (active && j < e) {
                        float4 q = pos4[j];
                        unsigned uj = (unsigned)j;
                        int tj = type[j];
                        ok = md_rsq_exact(p, q, kp) < kp.rskinsq && j != i && uj != ex.x &&
                             uj != ex.y && uj != ex.z && uj != ex.w && !((tmask >> tj) & 1u);
                        entry = uj | ((unsigned)tj << MD_TYPE_SHIFT);
                    }
                    unsigned bal = __ballot_sync(gmask, ok);
                    if (ok) {
                        int slot = cnt + __popc(bal & ((1u << lane_w) - 1u));
                        if (slot < kp.cap) nl[(size_t)i * kp.cap + slot] = entry;
                    }
                    cnt += __popc(bal);
                }
            }
        }
    }
    if (active) {
        /* pad the row to the next multiple of 32 with the atom itself */
        int lim = min(kp.cap, (cnt + MD_LIST_QUANTUM - 1) / MD_LIST_QUANTUM * MD_LIST_QUANTUM);
        unsigned self = (unsigned)i | ((unsigned)ti << MD_TYPE_SHIFT);
        for (int k = cnt + lane; k < lim; k += TPA) nl[(size_t)i * kp.cap + k] = self;
    }
    if (active && lane == 0) {
        nl_n[i] = cnt < kp.cap ? cnt : kp.cap;
        pos_old[i] = p;
        if (cnt > kp.cap) atomicMax(&st->list_overflow, cnt);
    }
}

/* The warp-per-cell list builder.  A persistent grid (the blocks that fit
 * on the GPU at once): each warp takes the next cell from a counter in the
 * device state until none is left, so cells of uneven work balance, and a
 * launch without a rebuild due starts only that many blocks.  The counter
 * is reset by the pass that ends the rebuild. */
/* In a batch the warps take work items over the cells of the replicas that
 * rebuild only (a replica's cells are the contiguous ranks [cell0, cell0 +
 * ncells)): each block first scans, in shared memory, the cell counts of
 * those replicas, and maps a work item to its replica by binary search.  A
 * step in which a few replicas rebuild then costs one counter increment per
 * cell of those replicas, not one per cell of the batch (2.2 M atoms in
 * 230 k cells).  Batches of more than CW_MAXREP replicas take every cell and
 * skip the ones of replicas that keep their lists. */
constexpr int CW_MAXREP = 4 * CW_WARPS * 32;

/* Exclusive prefix sums of of(r), r < nrep <= CW_MAXREP, in s_pre[0 .. nrep]
 * by a block of CW_WARPS warps; returns the total. */
template <class F>
__device__ __forceinline__ int replica_prefix(int nrep, int *s_pre, F &&of)
{
    constexpr int K = CW_MAXREP / (CW_WARPS * 32);   /* replicas per thread */
    __shared__ int s_wsum[CW_WARPS];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int v[K], sum = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int rr = t * K + k;
        v[k] = rr < nrep ? of(rr) : 0;
        sum += v[k];
    }
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();   /* s_wsum may still be read by an earlier call */
    if (lane == 31) s_wsum[w] = incl;
    __syncthreads();
    int before = incl - sum, total = 0;
    for (int u = 0; u < CW_WARPS; u++) {
        if (u < w) before += s_wsum[u];
        total += s_wsum[u];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int rr = t * K + k;
        if (rr <= nrep) s_pre[rr] = before;   /* s_pre[nrep] = total */
        before += v[k];
    }
    __syncthreads();
    return total;
}

/* The replica whose range of a prefix holds k: the largest r with pre[r] <= k. */
__device__ __forceinline__ int replica_of(const int *pre, int nrep, int k)
{
    int lo = 0, hi = nrep;
    while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (pre[m] <= k) lo = m; else hi = m;
    }
    return lo;
}

template <bool BATCH>
__global__ void __launch_bounds__(CW_WARPS * 32, 2) k_build_cells(
    md_kparams kp, md_devstate *st, int always, int ncells, int parts, int any_excl, int nrep,
    const float4 *__restrict__ pos4, const int *__restrict__ type, const uint4 *__restrict__ excl_s,
    const int *__restrict__ cell_rank, const int *__restrict__ cell_lin,
    const int *__restrict__ cell_start, const unsigned *__restrict__ type_mask, unsigned *nl,
    int *nl_n, float4 *pos_old, const md_rep *__restrict__ reps, const int *__restrict__ crep,
    const int *__restrict__ rep_upd)
{
    pdl_wait();
    pdl_trigger();
    if (!always && !st->update) return;
    __shared__ build_shm sm;
    const excl_src ex = {excl_s, nullptr, nullptr, nullptr, any_excl};
    const int lane = threadIdx.x & 31;
    if (BATCH && nrep <= CW_MAXREP) {
        __shared__ int s_pre[CW_MAXREP + 1];
        const int items =
            replica_prefix(nrep, s_pre, [&](int r) { return rep_upd[r] ? reps[r].ncells : 0; }) * parts;
        for (;;) {
            int wi = 0;
            if (lane == 0) wi = atomicAdd(&st->cell_next, 1);
            wi = __shfl_sync(0xffffffffu, wi, 0);
            if (wi >= items) break;
            const int cell = wi / parts, lo = replica_of(s_pre, nrep, cell);
            build_part<BATCH>(sm, reps[lo].cell0 + (cell - s_pre[lo]), wi - cell * parts, parts, kp, st, pos4, type, ex,
                              cell_rank, cell_lin, cell_start, type_mask, nl, nl_n, pos_old, reps, crep, rep_upd);
        }
        return;
    }
    for (;;) {
        int r = 0;
        if (lane == 0) r = atomicAdd(&st->cell_next, 1);
        r = __shfl_sync(0xffffffffu, r, 0);
        if (r >= ncells * parts) break;
        build_part<BATCH>(sm, r / parts, r % parts, parts, kp, st, pos4, type, ex, cell_rank, cell_lin, cell_start,
                          type_mask, nl, nl_n, pos_old, reps, crep, rep_upd);
    }
}

/* The whole rebuild of a single system as one cooperative kernel (the phases
 * of md_rebuild.cuh separated by grid barriers); a launch without a rebuild
 * due returns at once. */
__global__ void __launch_bounds__(CW_WARPS * 32, 2) k_rebuild_coop(md_kparams kp, md_devstate *st, int always,
                                                                rb_ptrs p)
{
    /* the same in every block: the request is cleared after the first
     * barrier, which every block reaches only after reading it, and the status
     * written only when a wait runs out; one left by an earlier launch (a
     * barrier that timed out, whose arrival count is then stale) stops every
     * later rebuild */
    if (!always && !st->update) return;
    if (*(volatile int *)&st->status != 0) return;
    grid_bar bar = {st, gridDim.x, p.bar_ns, 0ull};
    if (rebuild_phases(kp, st, p, p.pos4, bar)) bar.arrive_last();
}

/* The rebuild of a batch as one cooperative kernel: the phases of
 * rebuild_phases over the atoms and cells of the replicas that asked for it
 * (all: every replica), each replica in its own range of atoms and cells.
 * Atoms are taken in chunks of 32 of those replicas only.  A launch with no
 * rebuild due returns at once, so step graphs hold it inline: a conditional
 * node with the chain of nine passes cost ~10 us a step idle and 80 us per
 * rebuild of one 7986-ion replica, this kernel 3 and 51 (55 -> 37 us per NPT
 * step; 607 -> 485 us per step of 128 replicas, 35 of them from here). */
__global__ void __launch_bounds__(CW_WARPS * 32, 2) k_rebuild_coop_b(
    md_kparams kp, md_devstate *st, int always, int all, int nrep, rb_ptrs p, const md_rep *__restrict__ reps,
    const int *__restrict__ crep, int *rep_upd, md_repstate *repst)
{
    if (!always && !st->update) return;
    if (*(volatile int *)&st->status != 0) return;
    __shared__ build_shm sm;
    __shared__ int s_pre[CW_MAXREP + 1];   /* cells of the replicas to rebuild before replica r */
    static_assert(sizeof(build_shm) >= sizeof(int) * (CW_MAXREP + 32 + SCAN_LOCAL + SCAN_LOCAL / SCAN_K),
                  "chunk prefix and scan buffer");
    int *chunk = reinterpret_cast<int *>(&sm), *buf = chunk + CW_MAXREP + 32;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = tid >> 5, P = kp.pitch;
    const int cells = replica_prefix(nrep, s_pre, [&](int r) { return all || rep_upd[r] ? reps[r].ncells : 0; });
    const int nch =
        replica_prefix(nrep, chunk, [&](int r) { return all || rep_upd[r] ? (reps[r].natom + 31) / 32 : 0; });
    /* as many blocks as the work fills, at two atoms or more a warp; the
     * others leave (the same decision in every block) */
    const int blocks = min((int)gridDim.x, max(1, nch * 16 / CW_WARPS)), warps = blocks * CW_WARPS;
    if ((int)blockIdx.x >= blocks) return;
    const int parts = max(1, min(warps / max(1, cells), (nch * 32 + cells - 1) / max(1, cells)));
    const int nth = warps * 32;
    grid_bar bar = {st, (unsigned)blocks, p.bar_ns, 0ull};
    /* every atom of the replicas to rebuild, with its replica */
    auto for_atoms = [&](auto &&f) {
        for (int c = warp; c < nch; c += warps) {
            const int r = replica_of(chunk, nrep, c), a0 = reps[r].atom0;
            const int i = a0 + (c - chunk[r]) * 32 + lane;
            if (i < a0 + reps[r].natom) f(i, r);
        }
    };
    int *slot = p.tmp_i + 2 * (size_t)P;
    for_atoms([&](int i, int r) {
        const md_rep &R = reps[r];
        const float4 q = p.pos4[i];
        const int cx = cell_of(cell_coord(q.x, R.box[0], R.boxi[0], kp.centered), R.box[0], R.binlen[0], R.ncell[0]);
        const int cy = cell_of(cell_coord(q.y, R.box[1], R.boxi[1], kp.centered), R.box[1], R.binlen[1], R.ncell[1]);
        const int cz = cell_of(cell_coord(q.z, R.box[2], R.boxi[2], kp.centered), R.box[2], R.binlen[2], R.ncell[2]);
        const int k = p.cell_rank[R.cell0 + cx + R.ncell[0] * (cy + R.ncell[1] * cz)];
        p.key[i] = k;
        slot[i] = atomicAdd(&p.cell_count[k], 1);
    });
    if ((int)blockIdx.x == p.bar_drop) return;
    if (!bar()) return;
    if (tid == 0) {
        st->builds += 1;
        st->cell_next = 0;
    }
    /* a block per replica scans its cell counts from its first atom on */
    for (int r = blockIdx.x; r < nrep; r += blocks) {
        if (!(all || rep_upd[r])) continue;
        const int cell0 = reps[r].cell0, nc = reps[r].ncells;
        int base = reps[r].atom0;
        for (int c0 = 0; c0 < nc; c0 += SCAN_LOCAL) {
            const int m = min(SCAN_LOCAL, nc - c0), g0 = cell0 + c0;
            scan_local(m, p.cell_count + g0, buf);
            for (int c = threadIdx.x; c < m; c += blockDim.x) p.cell_start[g0 + c] = base + buf[scan_pad(c)];
            base += buf[scan_pad(m - 1)] + p.cell_count[g0 + m - 1];
            __syncthreads();
        }
        if (threadIdx.x == 0) p.cell_start[cell0 + nc] = base;   /* = the next replica's first atom */
    }
    if (!bar()) return;
    for_atoms([&](int i, int) { p.src[p.cell_start[p.key[i]] + slot[i]] = i; });
    if (!bar()) return;
    for_atoms([&](int s, int) {
        const int o = p.src[s], c = p.key[o], mine = p.perm[o];
        const int b = p.cell_start[c], e = p.cell_start[c + 1];
        int to = b;
#pragma unroll 4
        for (int k = b; k < e; k++) to += p.perm[p.src[k]] < mine ? 1 : 0;
        permute_one(kp, to, o, p.x, p.v, p.mass, p.kick, p.pos4, p.perm, p.type, p.tmp_d, p.tmp4, p.tmp_i);
        p.iperm[mine] = to;
    });
    for (int k = tid; k < cells; k += nth) {   /* for the next build */
        const int r = replica_of(s_pre, nrep, k);
        p.cell_count[reps[r].cell0 + k - s_pre[r]] = 0;
    }
    if (!bar()) return;
    const bool remap = p.has_bonds || p.has_angles;   /* the same in every block */
    for_atoms([&](int s, int) {
        copyback_one(kp, s, p.tmp_d, p.tmp4, p.tmp_i, p.x, p.v, p.mass, p.kick, p.pos4, p.perm, nullptr, p.type);
        if (remap)
            remap_one(kp, s, p.tmp_i, p.iperm, p.excl_orig, p.excl_s, p.bl_o, p.bl_on, p.bl_s, p.bl_sn, p.al_o,
                      p.al_on, p.al_s, p.al_sn, p.has_bonds, p.has_angles);
    });
    __syncthreads();   /* chunk is overwritten by the list build */
    const excl_src ex = {p.excl_s, remap ? p.excl_orig : nullptr, p.tmp_i, p.iperm, remap ? 1 : 0};
    const int items = cells * parts;
    for (int it = warp; it < items;) {
        const int cell = it / parts, r = replica_of(s_pre, nrep, cell);
        build_part<true>(sm, reps[r].cell0 + cell - s_pre[r], it - cell * parts, parts, kp, st, p.tmp4, p.tmp_i + P,
                         ex, p.cell_rank, p.cell_lin, p.cell_start, p.type_mask, p.nl, p.nl_n, p.pos_old, reps, crep,
                         nullptr);
        if (items <= warps) break;   /* one item a warp */
        if (lane == 0) it = warps + atomicAdd(&st->cell_next, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
    }
    if (!bar.arrive_last()) return;
    /* the last block to finish clears the requests */
    for (int r = threadIdx.x; r < nrep; r += blockDim.x)
        if (all || rep_upd[r]) {
            repst[r].builds += 1;
            rep_upd[r] = 0;
        }
    if (threadIdx.x == 0) st->update = 0;
}

}  // namespace

void launch_check(md_ctx *c, const md_kparams &kp)
{
    int nb = (kp.n + 255) / 256;
    if (c->batch) {
        k_check_b<<<nb, 256, 0, c->stream>>>(kp.n, c->reps_dev, c->arep, c->pos4, c->pos_old, c->st,
                                             c->rep_upd);
        return;
    }
    k_check<<<nb, 256, 0, c->stream>>>(kp, c->pos4, c->pos_old, c->st);
}

/* A pass of the rebuild: a plain launch, or (pdl) a programmatic dependent
 * launch whose blocks may be scheduled while the previous pass finishes;
 * every pass waits for its predecessor (pdl_wait) before it reads anything. */
template <typename... KArgs, typename... Args>
static void rb_launch(bool pdl, void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t s,
                      Args... args)
{
    if (pdl) md_launch_pdl(k, grid, block, s, args...);
    else k<<<grid, block, 0, s>>>(args...);
}

/* Blocks of the persistent warp-per-cell builder: as many as are resident
 * at once (found once per context, on its first, uncaptured, build), at
 * most one warp per part of a cell (*parts, md_build_parts). */
static int cw_blocks(md_ctx *c, bool batch, int *parts)
{
    int &g = c->cw_grid[batch ? 1 : 0];
    if (g == 0) {
        int dev = 0, nsm = 0, occ = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        c->nsm = std::max(1, nsm);
        if (batch) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_build_cells<true>, CW_WARPS * 32, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_build_cells<false>, CW_WARPS * 32, 0);
        g = std::max(1, nsm) * std::max(1, occ);
    }
    *parts = md_build_parts(c, g * CW_WARPS);
    return std::max(1, std::min(g, (c->ncells * *parts + CW_WARPS - 1) / CW_WARPS));
}

/* Whether the context rebuilds with one cooperative kernel: the warp-per-part
 * builder with its stencil in shared memory, in a batch at most CW_MAXREP
 * replicas, and enough resident blocks found for a cooperative launch. */
bool md_rebuild_coop(md_ctx *c)
{
    if (c->list_tpa != 0 || !c->rebuild_coop || (c->batch && c->nrep > CW_MAXREP)) return false;
    int nst = 1;   /* a batch's stencils have at most 125 cells */
    for (int d = 0; d < 3; d++) nst *= c->stencil[d] < 0 ? c->ncell[d] : 2 * c->stencil[d] + 1;
    if (nst > CW_MAXST) return false;
    if (c->coop_grid == 0) {   /* found once, on the context's first, uncaptured, build */
        int dev = 0, nsm = 0, occ = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (c->batch) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_rebuild_coop_b, CW_WARPS * 32, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_rebuild_coop, CW_WARPS * 32, 0);
        c->coop_grid = occ > 0 ? nsm * occ : -1;
    }
    return c->coop_grid > 0;
}

void launch_rebuild(md_ctx *c, const md_kparams &kp, bool unconditional, bool all_replicas, bool pdl)
{
    int always = unconditional ? 1 : 0;
    if (c->batch) pdl = false;
    if (md_rebuild_coop(c)) {
        const rb_ptrs p = make_rb_ptrs(c, c->coop_grid);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c->coop_grid);
        cfg.blockDim = dim3(CW_WARPS * 32);
        cfg.stream = c->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const cudaError_t e =
            c->batch ? cudaLaunchKernelEx(&cfg, k_rebuild_coop_b, kp, c->st, always, all_replicas ? 1 : 0, c->nrep, p,
                                          (const md_rep *)c->reps_dev, (const int *)c->crep, c->rep_upd, c->repst)
                     : cudaLaunchKernelEx(&cfg, k_rebuild_coop, kp, c->st, always, p);
        if (e == cudaSuccess) return;
        /* a refused cooperative launch (fewer resident blocks than found
         * when the context was set up) falls back to the chain of passes,
         * for good when not capturing (during a capture the error stays
         * sticky in the capture, which then fails and is reported) */
        (void)cudaGetLastError();
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(c->stream, &cs);
        if (cs != cudaStreamCaptureStatusNone) return;
        c->coop_grid = -1;
    }
    int parts = 1;
    const int cwb = cw_blocks(c, c->batch, &parts);   /* also finds the SM count */
    int nb = (kp.n + 255) / 256;
    cudaStream_t s = c->stream;
    const bool batch = c->batch;
    const int rb = (c->nrep + 255) / 256;
    const int *arep = batch ? c->arep : nullptr;
    const int *crep = batch ? c->crep : nullptr;
    if (batch) {
        if (all_replicas) k_flag_all<<<rb, 256, 0, s>>>(c->rep_upd, c->nrep);
        k_cell_key_b<<<nb, 256, 0, s>>>(kp.n, kp.centered, c->reps_dev, c->arep, c->st, always, c->rep_upd,
                                        c->pos4, c->cell_rank, c->key, c->cell_count);
        k_cell_scan_b<<<(c->nrep + 7) / 8, 256, 0, s>>>(c->st, always, c->nrep, c->reps_dev,
                                                        c->rep_upd, c->cell_count, c->cell_start,
                                                        c->cell_fill);
    } else {
        rb_launch(pdl, k_cell_key, dim3(nb), dim3(256), s, kp, c->st, always, (const float4 *)c->pos4,
                  (const int *)c->cell_rank, c->key, c->cell_count);
        rb_launch(pdl, k_cell_scan, dim3(1), dim3(1024), s, kp, c->st, always, c->ncells, c->cell_count,
                  c->cell_start, c->cell_fill);
    }
    rb_launch(pdl, k_cell_scatter, dim3(nb), dim3(256), s, kp, (const md_devstate *)c->st, always,
              (const int *)c->key, (const int *)c->cell_start, c->cell_fill, c->src, arep,
              (const int *)c->rep_upd);
    /* a warp per cell, at most two blocks of 8 warps per SM (a loop over cells) */
    rb_launch(pdl, k_cell_order, dim3(std::min((c->ncells + 7) / 8, 2 * c->nsm)), dim3(256), s, kp,
              (const md_devstate *)c->st, always, c->ncells, (const int *)c->cell_start,
              (const int *)c->perm, c->src, crep, (const int *)c->rep_upd);
    rb_launch(pdl, k_permute, dim3(nb), dim3(256), s, kp, (const md_devstate *)c->st, always,
              (const int *)c->src, (const double *)c->x, (const double *)c->v,
              (const double *)c->mass, (const double *)c->kick, (const float4 *)c->pos4,
              (const int *)c->perm, (const int *)c->type, c->tmp_d, c->tmp4, c->tmp_i, arep,
              (const int *)c->rep_upd);
    rb_launch(pdl, k_copyback, dim3(nb), dim3(256), s, kp, (const md_devstate *)c->st, always,
              (const double *)c->tmp_d, (const float4 *)c->tmp4, (const int *)c->tmp_i, c->x, c->v,
              c->mass, c->kick, c->pos4, c->perm, c->iperm, c->type, arep, (const int *)c->rep_upd);
    /* exclusions and bonded lists to re-express only with bonds or angles
     * (in a batch every atom: a replica that kept its order maps to the
     * same lists) */
    if (c->has_bonds || c->has_angles)
        rb_launch(pdl, k_remap, dim3(nb), dim3(256), s, kp, (const md_devstate *)c->st, always,
                  (const int *)c->perm, (const int *)c->iperm, (const uint4 *)c->excl_orig, c->excl_s,
                  (const int2 *)c->bl_o, (const int *)c->bl_on, c->bl_s, c->bl_sn,
                  (const int4 *)c->al_o, (const int *)c->al_on, c->al_s, c->al_sn, c->has_bonds,
                  c->has_angles);
    if (batch) {
        /* at most 5 stencil cells per axis (cells of side >= rl/2): <= 125 */
        k_build_cells<true><<<cwb, CW_WARPS * 32, 0, s>>>(
            kp, c->st, always, c->ncells, parts, c->has_bonds, c->nrep, c->pos4, c->type, c->excl_s, c->cell_rank,
            c->cell_lin, c->cell_start, c->type_mask_dev, c->nl, c->nl_n, c->pos_old, c->reps_dev, c->crep,
            c->rep_upd);
        k_clear_update_b<<<rb, 256, 0, s>>>(c->st, always, c->rep_upd, c->repst, c->nrep);
        return;
    }
    int ltpa = c->list_tpa;
    if (ltpa == 0) {   /* the warp-per-cell builder keeps up to 128 stencil cells in shared memory */
        int nst = 1;
        for (int d = 0; d < 3; d++) nst *= c->stencil[d] < 0 ? c->ncell[d] : 2 * c->stencil[d] + 1;
        if (nst > CW_MAXST) ltpa = 8;
    }
    long long threads = (long long)kp.n * (ltpa > 0 ? ltpa : 1);
    int lb = (int)((threads + 255) / 256);
    switch (ltpa) {
    case 0:
        rb_launch(pdl, k_build_cells<false>, dim3(cwb),
                  dim3(CW_WARPS * 32), s, kp, c->st, always, c->ncells, parts, c->has_bonds, 0,
                  (const float4 *)c->pos4,
                  (const int *)c->type, (const uint4 *)c->excl_s, (const int *)c->cell_rank,
                  (const int *)c->cell_lin, (const int *)c->cell_start,
                  (const unsigned *)c->type_mask_dev, c->nl, c->nl_n, c->pos_old,
                  (const md_rep *)nullptr, (const int *)nullptr, (const int *)nullptr);
        break;
#define MD_LIST_CASE(T)                                                                            \
    case T:                                                                                        \
        rb_launch(pdl, k_build_list<T>, dim3(lb), dim3(256), s, kp, c->st, always,                 \
                  (const float4 *)c->pos4, (const int *)c->type, (const uint4 *)c->excl_s,         \
                  (const int *)c->cell_rank, (const int *)c->cell_start,                           \
                  (const unsigned *)c->type_mask_dev, c->nl, c->nl_n, c->pos_old);                 \
        break;
        MD_LIST_CASE(1)
        MD_LIST_CASE(2)
        MD_LIST_CASE(4)
        MD_LIST_CASE(8)
        MD_LIST_CASE(16)
        MD_LIST_CASE(32)
#undef MD_LIST_CASE
    default:
        break;
    }
    rb_launch(pdl, k_clear_update, dim3(1), dim3(1), s, c->st);
}

void launch_set_condition(md_ctx *c, unsigned long long handle)
{
    k_set_condition<<<1, 1, 0, c->stream>>>((cudaGraphConditionalHandle)handle, c->st);
}
