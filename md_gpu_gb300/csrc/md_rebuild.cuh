/*
 * md_rebuild.cuh -- the neighbour-list rebuild of a single system as phases
 * of one kernel: binning, scan, scatter, permute, then copy-back, remap and
 * the list build, separated by a grid barrier that the kernel brings.  k_rebuild_coop (k_cells.cu) is these
 * phases alone; k_run_steps (k_run.cu) runs them between its steps.
 */
#ifndef MD_REBUILD_CUH
#define MD_REBUILD_CUH

#include <algorithm>

#include "md_device.cuh"

namespace {

/* Cell rank (Hilbert order) of atom i, counted in its cell; returns its
 * arrival number there. */
__device__ __forceinline__ int key_one(const md_kparams &kp, int i, const float4 *__restrict__ pos4,
                                        const int *__restrict__ cell_rank, int *key, int *cell_count)
{
    float4 p = pos4[i];
    int cx = cell_of(cell_coord(p.x, kp.box[0], kp.boxi[0], kp.centered), kp.box[0], kp.binlen[0], kp.ncell[0]);
    int cy = cell_of(cell_coord(p.y, kp.box[1], kp.boxi[1], kp.centered), kp.box[1], kp.binlen[1], kp.ncell[1]);
    int cz = cell_of(cell_coord(p.z, kp.box[2], kp.boxi[2], kp.centered), kp.box[2], kp.binlen[2], kp.ncell[2]);
    int r = cell_rank[cx + kp.ncell[0] * (cy + kp.ncell[1] * cz)];
    key[i] = r;
    return atomicAdd(&cell_count[r], 1);
}

/* Exclusive scan of the cell counts by one block of NT threads, then the
 * counters are zeroed for the next build; returns the total in thread 0.  In
 * rounds of NT x SCAN_K cells: the counts pass through shared memory, so
 * that global loads and stores are coalesced (one SM issues them all) while
 * each thread scans SCAN_K consecutive counts; warps scan their threads'
 * sums with shuffles and warp 0 the warp totals.  Shared index i is stored
 * at i + i / SCAN_K, so the per-thread reads hit distinct banks. */
constexpr int SCAN_K = 8;
__device__ __forceinline__ int scan_pad(int i) { return i + i / SCAN_K; }

template <int NT>
__device__ __forceinline__ int scan_cells(int ncells, int *cell_count, int *cell_start, int *cell_fill)
{
    constexpr int N = NT * SCAN_K;
    __shared__ int buf[N + N / SCAN_K];
    __shared__ int wsum[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int carry = 0;
    for (int base = 0; base < ncells; base += N) {
#pragma unroll
        for (int k = 0; k < SCAN_K; k++) {
            const int i = k * NT + t, g = base + i;
            buf[scan_pad(i)] = g < ncells ? cell_count[g] : 0;
        }
        __syncthreads();
        int v[SCAN_K], s = 0;
#pragma unroll
        for (int k = 0; k < SCAN_K; k++) {
            v[k] = buf[scan_pad(t * SCAN_K + k)];
            s += v[k];
        }
        int incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        if (w == 0) {
            int x = lane < NT / 32 ? wsum[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            wsum[lane] = x;   /* inclusive over warps */
        }
        __syncthreads();
        int run = carry + (w > 0 ? wsum[w - 1] : 0) + incl - s;
#pragma unroll
        for (int k = 0; k < SCAN_K; k++) {
            buf[scan_pad(t * SCAN_K + k)] = run;
            run += v[k];
        }
        carry += wsum[NT / 32 - 1];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SCAN_K; k++) {
            const int i = k * NT + t, g = base + i;
            if (g < ncells) {
                cell_start[g] = buf[scan_pad(i)];
                cell_count[g] = 0;
                cell_fill[g] = 0;
            }
        }
        __syncthreads();   /* buf and wsum are rewritten by the next round */
    }
    return carry;
}

/* Within each cell, order atoms by original index: the sorted order is then a
 * function of the positions alone.  One warp per cell: each atom's place is
 * the number of the cell's atoms with a smaller original index (indices are
 * distinct), counted with shuffles; cells of more than 4 x 32 atoms (far
 * denser than any liquid at these cell sizes) are sorted by one lane. */
constexpr int ORD_MAX = 4;
/* The rank sort of one cell's atoms (one warp). */
__device__ __forceinline__ void order_cell(int c, const int *__restrict__ cell_start,
                                           const int *__restrict__ perm, int *src,
                                           const int *__restrict__ crep,
                                           const int *__restrict__ rep_upd, int lane)
{
    if (crep && !rep_upd[crep[c]]) return;
    const int b = cell_start[c], n = cell_start[c + 1] - b;
    if (n <= 1) return;
    if (n <= 32 * ORD_MAX) {
        int a[ORD_MAX], key[ORD_MAX], rank[ORD_MAX];
#pragma unroll
        for (int q = 0; q < ORD_MAX; q++) {
            const int k = q * 32 + lane;
            a[q] = k < n ? src[b + k] : 0;
            key[q] = k < n ? perm[a[q]] : 0x7fffffff;
            rank[q] = 0;
        }
#pragma unroll
        for (int q2 = 0; q2 < ORD_MAX; q2++) {
            if (q2 * 32 >= n) break;
            const int m = min(32, n - q2 * 32);
            for (int j = 0; j < m; j++) {
                const int kj = __shfl_sync(0xffffffffu, key[q2], j);
#pragma unroll
                for (int q = 0; q < ORD_MAX; q++) rank[q] += kj < key[q] ? 1 : 0;
            }
        }
        __syncwarp();   /* every read of src above precedes the writes below */
#pragma unroll
        for (int q = 0; q < ORD_MAX; q++)
            if (q * 32 + lane < n) src[b + rank[q]] = a[q];
        return;
    }
    if (lane != 0) return;
    for (int k = b + 1; k < b + n; k++) {
        int a = src[k], ka = perm[a];
        int m = k - 1;
        while (m >= b && perm[src[m]] > ka) {
            src[m + 1] = src[m];
            m--;
        }
        src[m + 1] = a;
    }
}

/* Sorted slot s takes the state of atom o (into the staging arrays). */
__device__ __forceinline__ void permute_one(const md_kparams &kp, int s, int o,
                                            const double *__restrict__ x, const double *__restrict__ v,
                                            const double *__restrict__ mass, const double *__restrict__ kick,
                                            const float4 *__restrict__ pos4, const int *__restrict__ perm,
                                            const int *__restrict__ type, double *tmp_d, float4 *tmp4,
                                            int *tmp_i)
{
    int P = kp.pitch;
    for (int d = 0; d < 3; d++) {
        tmp_d[d * P + s] = x[d * P + o];
        tmp_d[(3 + d) * P + s] = v[d * P + o];
    }
    tmp_d[6 * P + s] = mass[o];
    tmp_d[7 * P + s] = kick[o];
    tmp4[s] = pos4[o];
    tmp_i[s] = perm[o];
    tmp_i[P + s] = type[o];
}

/* The staged state back into the per-atom arrays, and (iperm non-null) the
 * inverse order. */
__device__ __forceinline__ void copyback_one(const md_kparams &kp, int s, const double *__restrict__ tmp_d,
                                             const float4 *__restrict__ tmp4, const int *__restrict__ tmp_i,
                                             double *x, double *v, double *mass, double *kick, float4 *pos4,
                                             int *perm, int *iperm, int *type)
{
    int P = kp.pitch;
    for (int d = 0; d < 3; d++) {
        x[d * P + s] = tmp_d[d * P + s];
        v[d * P + s] = tmp_d[(3 + d) * P + s];
    }
    mass[s] = tmp_d[6 * P + s];
    kick[s] = tmp_d[7 * P + s];
    pos4[s] = tmp4[s];
    int o = tmp_i[s];
    perm[s] = o;
    if (iperm) iperm[o] = s;
    type[s] = tmp_i[P + s];
}

/* Exclusions and bonded lists of sorted slot s in the new sorted indices. */
__device__ __forceinline__ void remap_one(const md_kparams &kp, int s, const int *__restrict__ perm,
                                          const int *__restrict__ iperm, const uint4 *__restrict__ excl_orig,
                                          uint4 *excl_s, const int2 *__restrict__ bl_o,
                                          const int *__restrict__ bl_on, int2 *bl_s, int *bl_sn,
                                          const int4 *__restrict__ al_o, const int *__restrict__ al_on,
                                          int4 *al_s, int *al_sn, int has_bonds, int has_angles)
{
    int o = perm[s], P = kp.pitch;
    uint4 e = excl_orig[o];
    uint4 m;
    m.x = e.x == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)iperm[e.x];
    m.y = e.y == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)iperm[e.y];
    m.z = e.z == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)iperm[e.z];
    m.w = e.w == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)iperm[e.w];
    excl_s[s] = m;
    if (has_bonds) {
        int nb = bl_on[o];
        for (int k = 0; k < nb; k++) {
            int2 b = bl_o[4 * o + k];
            bl_s[k * P + s] = make_int2(iperm[b.x], b.y);
        }
        bl_sn[s] = nb;
    }
    if (has_angles) {
        int na = al_on[o];
        for (int k = 0; k < na; k++) {
            int4 a = al_o[4 * o + k];
            al_s[k * P + s] = make_int4(a.x, iperm[a.y], iperm[a.z], a.w);
        }
        al_sn[s] = na;
    }
}

/* List build, a warp per part of a cell: every atom of a cell shares the
 * cell's stencil.  A cell's atoms are split evenly over `parts` warps, which
 * take them in even groups of up to CW_GA.  The warp first gathers the stencil
 * cells' atom ranges into shared memory (in traversal order) with their
 * prefix sums, then streams the concatenated candidates 32 at a time (lane =
 * candidate; a bit map of the places where a cell's candidates begin gives
 * its stencil cell with a population count).  A conservative test against
 * the bounding box of the group drops the candidates that no atom of it can
 * reach; the rest enter a per-warp queue in candidate order, and each full
 * queue of 64 is tested exactly against the group's atoms, two ballots per
 * atom appending the hits to its row.
 * Where a stencil cell's periodic image does not fix the shift (boxes of a
 * few cells), every candidate is tested with the per-pair shift.  Entries
 * land in the same order as in k_build_list (stencil cells in traversal order, ascending
 * j) whatever the parts, so all builders produce identical lists.
 *
 * At 16 warps per SM it is bound by their chains of ballots, shuffles and
 * loads (issue slots 46% busy, stalls per issue long scoreboard 1.9, wait 1.8,
 * barrier 1.3), so fewer instructions per candidate count.  Per build against
 * one warp per cell with a 32-wide queue: 64000 ions 149 -> 122 us (102 M -> 66 M warp instructions;
 * the whole rebuild kernel), 982 ions (64 cells, split in parts) 106 -> 39
 * us, 5184 water atoms (exclusions) 476 -> 91 us, 128 replicas of 512 to
 * 8000 ions 834 -> 762 us.  Two blocks of 8 warps per SM at 128 registers:
 * three at 80 measured 134 us (83 M instructions, rematerialised addresses).
 *
 * Exclusions are rare, so a 1024-bit map of the group's excluded indices
 * (modulo 1024) decides per round whether any candidate can be one; only
 * then are the exact comparisons made. */
constexpr int CW_WARPS = 8;   /* warps per block (fewer blocks: fewer grid-barrier arrivals) */
constexpr int CW_GA = 32;     /* atoms of a group, at most (a lane each) */
constexpr int CW_MAXST = 128;
constexpr int CW_CHUNK = 1024;   /* candidates whose stencil cells are marked at a time */
constexpr int CW_CODES = 43;     /* image codes: 2 bits an axis, each 0, 1 or 2 */

/* Shared memory of a list-building warp: one base address, everything else
 * an immediate offset from it. */
struct warp_shm {
    /* ring of near candidates: position and (w) list entry, image code */
    float4 fq[128];
    unsigned char fc[128];
    /* the group's coordinates by axis, so that two atoms' x (y, z) are one
     * load of a register pair; slots past the group hold a far point */
    float hx[CW_GA], hy[CW_GA], hz[CW_GA];
    uint4 ex[CW_GA];
    unsigned tm[CW_GA];
    unsigned map[32];               /* excluded indices modulo 1024 */
    float4 u[CW_CODES];              /* L rint(d / L) by image code */
    /* the stencil's cells that hold atoms, in traversal order: the place of
     * their first candidate, its index less that place, their image code */
    int pre[CW_MAXST];
    int jb[CW_MAXST];
    unsigned char sh[CW_MAXST];
    unsigned first[CW_CHUNK / 32];  /* a bit where a cell's candidates begin */
};
struct build_shm {
    warp_shm warp[CW_WARPS];
};

/* Cell geometry seen by one warp: the system's, or in a batch the replica's
 * that owns the cell. */
struct cell_geom {
    float L[3], Li[3], rskinsq;
    int nc[3], sten[3], shift, lin0;
};

/* Where the exclusions of a group come from: the sorted lists (excl_s), or
 * (orig non-null) the original ones through the new order. */
struct excl_src {
    const uint4 *excl_s;
    const uint4 *orig;
    const int *perm, *iperm;
    int any;   /* 0: the system has none */
};

__device__ __forceinline__ uint4 excl_of(const excl_src &x, int i)
{
    if (!x.orig) return x.excl_s[i];
    const uint4 e = x.orig[x.perm[i]];
    uint4 m;
    m.x = e.x == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)x.iperm[e.x];
    m.y = e.y == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)x.iperm[e.y];
    m.z = e.z == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)x.iperm[e.z];
    m.w = e.w == MD_EXCL_NONE ? MD_EXCL_NONE : (unsigned)x.iperm[e.w];
    return m;
}

/* The periodic image of a stencil cell on one axis from two bits of its
 * code: 0 none, 1 wrapped from below (the reference's rint(d/L) = -1), 2
 * from above (+1); u = L rint(d / L). */
__device__ __forceinline__ float image_of(int code, float L)
{
    return (code & 1) ? -L : ((code & 2) ? L : 0.0f);
}

/* The list rows of part `part` of `parts` of the atoms of cell r (sorted
 * rank), built by one warp. */
template <bool BATCH>
__device__ __forceinline__ void build_part(
    build_shm &sm, int r, int part, int parts, const md_kparams &kp, md_devstate *st, const float4 *pos4, const int *type,
    const excl_src &ex_src, const int *cell_rank, const int *cell_lin, const int *cell_start,
    const unsigned *type_mask, unsigned *nl, int *nl_n, float4 *pos_old, const md_rep *reps, const int *crep,
    const int *rep_upd)
{
    const int lane = threadIdx.x & 31;
    warp_shm &ws = sm.warp[threadIdx.x >> 5];
    const int c0 = cell_start[r], cn = cell_start[r + 1] - c0;
    const int ib = c0 + cn * part / parts, ie = c0 + cn * (part + 1) / parts;
    if (ib == ie) return;
    cell_geom G;
    if (BATCH) {
        const int rr = crep[r];
        if (rep_upd && !rep_upd[rr]) return;   /* this replica keeps its list */
        const md_rep &R = reps[rr];
        for (int d = 0; d < 3; d++) {
            G.L[d] = R.box[d]; G.Li[d] = R.boxi[d]; G.nc[d] = R.ncell[d]; G.sten[d] = R.stencil[d];
        }
        G.rskinsq = R.rskinsq; G.shift = R.cell_shift && kp.centered; G.lin0 = R.cell0;
    } else {
        for (int d = 0; d < 3; d++) {
            G.L[d] = kp.box[d]; G.Li[d] = kp.boxi[d]; G.nc[d] = kp.ncell[d]; G.sten[d] = kp.stencil[d];
        }
        G.rskinsq = kp.rskinsq; G.shift = kp.cell_shift; G.lin0 = 0;
    }
    const int lin = cell_lin[r];
    const int nx = G.nc[0], ny = G.nc[1], nz = G.nc[2];
    const int c3[3] = {lin % nx, (lin / nx) % ny, lin / (nx * ny)};
    int lo[3], len[3];
    for (int d = 0; d < 3; d++) {
        if (G.sten[d] < 0) { lo[d] = 0; len[d] = G.nc[d]; }
        else { lo[d] = c3[d] - G.sten[d]; len[d] = 2 * G.sten[d] + 1; }
    }
    const int nst = len[0] * len[1] * len[2];   /* <= 125 with cells of side >= rl/2 */
    const unsigned lt = (1u << lane) - 1u;
    /* stencil ranges in traversal order (z outer, x inner); lane k takes k,
     * k + 32, ...; every range is loaded before the first is needed */
    int total = 0, nne = 0;
    {
        int jb[CW_MAXST / 32], cnt[CW_MAXST / 32], code[CW_MAXST / 32];
#pragma unroll
        for (int u = 0; u < CW_MAXST / 32; u++) {
            const int k = u * 32 + lane;
            jb[u] = cnt[u] = code[u] = 0;
            if (k < nst) {
                const int dx = k % len[0], dy = (k / len[0]) % len[1], dz = k / (len[0] * len[1]);
                const int xx = lo[0] + dx, yy = lo[1] + dy, zz = lo[2] + dz;
                code[u] = (xx < 0 ? 1 : (xx >= nx ? 2 : 0)) | ((yy < 0 ? 1 : (yy >= ny ? 2 : 0)) << 2) |
                          ((zz < 0 ? 1 : (zz >= nz ? 2 : 0)) << 4);
                const int cx = xx < 0 ? xx + nx : (xx >= nx ? xx - nx : xx);
                const int cy = yy < 0 ? yy + ny : (yy >= ny ? yy - ny : yy);
                const int cz = zz < 0 ? zz + nz : (zz >= nz ? zz - nz : zz);
                const int r2 = cell_rank[G.lin0 + cx + nx * (cy + ny * cz)];
                jb[u] = cell_start[r2];
                cnt[u] = cell_start[r2 + 1] - jb[u];
            }
        }
#pragma unroll
        for (int u = 0; u < CW_MAXST / 32; u++) {
            if (u * 32 < nst) {
                int incl = cnt[u];
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                const unsigned ne = __ballot_sync(0xffffffffu, cnt[u] > 0);
                if (cnt[u] > 0) {
                    const int at = nne + __popc(ne & lt), pre = total + incl - cnt[u];
                    ws.pre[at] = pre;
                    ws.jb[at] = jb[u] - pre;   /* j of candidate g is s_jb + g */
                    ws.sh[at] = (unsigned char)code[u];
                }
                nne += __popc(ne);
                total += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
    }
    for (int k = lane; k < CW_CODES; k += 32)
        ws.u[k] = make_float4(image_of(k, G.L[0]), image_of(k >> 2, G.L[1]), image_of(k >> 4, G.L[2]), 0.0f);
    typedef v2<true> V;
    __syncwarp();
    const int ng = (ie - ib + CW_GA - 1) / CW_GA;
    for (int gr = 0; gr < ng; gr++) {
        const int i0 = ib + (ie - ib) * gr / ng, ni = ib + (ie - ib) * (gr + 1) / ng - i0;
        const float4 own = pos4[i0 + (lane < ni ? lane : 0)];
        const int own_type = type[i0 + (lane < ni ? lane : 0)];
        ws.hx[lane] = lane < ni ? own.x : 1e30f;
        ws.hy[lane] = lane < ni ? own.y : 1e30f;
        ws.hz[lane] = lane < ni ? own.z : 1e30f;
        const unsigned tmask = lane < ni ? type_mask[own_type] : 0u;
        const bool any_tm = __any_sync(0xffffffffu, tmask != 0u);
        bool any_ex = false;
        if (ex_src.any || any_tm) {
            ws.map[lane] = 0u;
            __syncwarp();
            if (lane < ni) {
                const uint4 ex = excl_of(ex_src, i0 + lane);
                ws.ex[lane] = ex;
                ws.tm[lane] = tmask;
                const unsigned e4[4] = {ex.x, ex.y, ex.z, ex.w};
                for (int k = 0; k < 4; k++)
                    if (e4[k] != MD_EXCL_NONE) {
                        atomicOr(&ws.map[(e4[k] >> 5) & 31], 1u << (e4[k] & 31));
                        any_ex = true;
                    }
            }
            any_ex = __any_sync(0xffffffffu, any_ex);
        }
        __syncwarp();
        unsigned *rows = nl + (size_t)i0 * kp.cap;
        unsigned rowoff = (unsigned)(lane * kp.cap);   /* lane a: where row a's next entry goes, from rows */
        int mycnt = 0;                                  /* its length */
        /* The exact test of 64 queued candidates (two a lane, 32 apart; cnt of
         * them from slot `head` on) against the group; two ballots per atom
         * append the hits to its row in candidate order.  A row's offset
         * changes only in its own iteration, so each iteration takes it from
         * the offsets at the start of the batch and the iterations are
         * independent; lane a keeps row a's ballots and counts them after
         * the loop.  Two atoms at once: the differences and squares in
         * packed f32x2 instructions, the two sums in scalar adds with
         * explicit rounding (a packed multiply followed by a packed add may
         * be contracted into a packed FMA by the code generator, which would
         * change the rounding of r^2); fl(fl(px - qx) - u) is the reference's
         * fl(d - fl(L rint(d/L))).  The comparisons that can matter only in
         * some batches (a possible exclusion, a row near its capacity) have
         * a loop of their own. */
        auto process = [&](int head, int cnt) {
            const bool v0 = lane < cnt, v1 = lane + 32 < cnt;
            const int a0 = (head + lane) & 127, a1 = (head + 32 + lane) & 127;
            const float4 q0 = ws.fq[a0], q1 = ws.fq[a1];
            const float4 u0 = ws.u[v0 ? ws.fc[a0] : 0], u1 = ws.u[v1 ? ws.fc[a1] : 0];
            const unsigned e0 = __float_as_uint(q0.w), e1 = __float_as_uint(q1.w);
            const unsigned j0 = e0 & MD_INDEX_MASK, j1 = e1 & MD_INDEX_MASK;
            /* the group member a candidate is, if < ni */
            const unsigned s0 = j0 - (unsigned)i0, s1 = j1 - (unsigned)i0;
            const float far0 = v0 ? G.rskinsq : -1.0f, far1 = v1 ? G.rskinsq : -1.0f;   /* no hit in an empty slot */
            bool slow = any_tm || !(G.shift || kp.centered) || (lane < ni && mycnt + 64 > kp.cap);
            if (any_ex)
                slow = slow || (v0 && ((ws.map[(j0 >> 5) & 31] >> (j0 & 31)) & 1u)) ||
                       (v1 && ((ws.map[(j1 >> 5) & 31] >> (j1 & 31)) & 1u));
            unsigned k0 = 0u, k1 = 0u;   /* lane a: the ballots of atom a */
            auto append = [&](int a, bool ok0, bool ok1, unsigned end) {
                const unsigned b0 = __ballot_sync(0xffffffffu, ok0), b1 = __ballot_sync(0xffffffffu, ok1);
                const unsigned at = __shfl_sync(0xffffffffu, rowoff, a);
                const unsigned o0 = at + __popc(b0 & lt), o1 = at + __popc(b0) + __popc(b1 & lt);
                if (ok0 && o0 < end) rows[o0] = e0;
                if (ok1 && o1 < end) rows[o1] = e1;
                if (lane == a) {
                    k0 = b0;
                    k1 = b1;
                }
            };
            if (__any_sync(0xffffffffu, slow)) {
                for (int a = 0; a < ni; a++) {
                    const float4 p = make_float4(ws.hx[a], ws.hy[a], ws.hz[a], 0.0f);
                    uint4 ex = make_uint4(MD_EXCL_NONE, MD_EXCL_NONE, MD_EXCL_NONE, MD_EXCL_NONE);
                    unsigned tm = 0u;
                    if (any_ex || any_tm) {
                        ex = ws.ex[a];
                        tm = ws.tm[a];
                    }
                    auto test = [&](float4 q, float4 u, unsigned e, unsigned j, unsigned self, float far) {
                        float rsq;
                        if (G.shift) {
                            const float dx = __fsub_rn(__fsub_rn(p.x, q.x), u.x);
                            const float dy = __fsub_rn(__fsub_rn(p.y, q.y), u.y);
                            const float dz = __fsub_rn(__fsub_rn(p.z, q.z), u.z);
                            rsq = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                        } else {
                            rsq = md_rsq_box(p, q, G.L, G.Li);
                        }
                        return rsq < far && (unsigned)a != self && j != ex.x && j != ex.y && j != ex.z && j != ex.w &&
                               !((tm >> (e >> MD_TYPE_SHIFT)) & 1u);
                    };
                    const bool ok0 = test(q0, u0, e0, j0, s0, far0), ok1 = test(q1, u1, e1, j1, s1, far1);
                    append(a, ok0, ok1, (unsigned)((a + 1) * kp.cap));
                }
            } else if (G.shift) {
                const V QX0 = V::make(q0.x, q0.x), QY0 = V::make(q0.y, q0.y), QZ0 = V::make(q0.z, q0.z);
                const V QX1 = V::make(q1.x, q1.x), QY1 = V::make(q1.y, q1.y), QZ1 = V::make(q1.z, q1.z);
                const V UX0 = V::make(u0.x, u0.x), UY0 = V::make(u0.y, u0.y), UZ0 = V::make(u0.z, u0.z);
                const V UX1 = V::make(u1.x, u1.x), UY1 = V::make(u1.y, u1.y), UZ1 = V::make(u1.z, u1.z);
#pragma unroll 2
                for (int a = 0; a < ni; a += 2) {
                    const float2 px = *reinterpret_cast<const float2 *>(&ws.hx[a]);
                    const float2 py = *reinterpret_cast<const float2 *>(&ws.hy[a]);
                    const float2 pz = *reinterpret_cast<const float2 *>(&ws.hz[a]);
                    const V PX = V::make(px.x, px.y), PY = V::make(py.x, py.y), PZ = V::make(pz.x, pz.y);
                    auto dist = [&](V QX, V QY, V QZ, V UX, V UY, V UZ, float &ra, float &rb) {
                        const V dx = (PX - QX) - UX, dy = (PY - QY) - UY, dz = (PZ - QZ) - UZ;
                        float x0, x1, y0, y1, z0, z1;
                        (dx * dx).get(x0, x1);
                        (dy * dy).get(y0, y1);
                        (dz * dz).get(z0, z1);
                        ra = __fadd_rn(__fadd_rn(x0, y0), z0);
                        rb = __fadd_rn(__fadd_rn(x1, y1), z1);
                    };
                    float ra0, rb0, ra1, rb1;
                    dist(QX0, QY0, QZ0, UX0, UY0, UZ0, ra0, rb0);
                    dist(QX1, QY1, QZ1, UX1, UY1, UZ1, ra1, rb1);
                    append(a, ra0 < far0 && s0 != (unsigned)a, ra1 < far1 && s1 != (unsigned)a, 0xffffffffu);
                    append(a + 1, rb0 < far0 && s0 != (unsigned)a + 1u, rb1 < far1 && s1 != (unsigned)a + 1u, 0xffffffffu);
                }
            } else {
                /* per-pair shift (boxes of a few cells), every position in the
                 * box: rint(d / L) of |d / L| <= 1 by adding and subtracting
                 * 1.5 * 2^23 (the same value as rintf) */
#pragma unroll 2
                for (int a = 0; a < ni; a++) {
                    const float px = ws.hx[a], py = ws.hy[a], pz = ws.hz[a];
                    auto axis = [&](float p, float q, float L, float Li) {
                        const float d = __fsub_rn(p, q);
                        return __fsub_rn(d, __fmul_rn(L, __fsub_rn(__fadd_rn(__fmul_rn(d, Li), 12582912.0f), 12582912.0f)));
                    };
                    auto dist = [&](float4 q) {
                        const float dx = axis(px, q.x, G.L[0], G.Li[0]), dy = axis(py, q.y, G.L[1], G.Li[1]),
                                    dz = axis(pz, q.z, G.L[2], G.Li[2]);
                        return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                    };
                    append(a, dist(q0) < far0 && s0 != (unsigned)a, dist(q1) < far1 && s1 != (unsigned)a, 0xffffffffu);
                }
            }
            const int inc = __popc(k0) + __popc(k1);
            mycnt += inc;
            rowoff += inc;
        };
        /* Bounding box of the group: candidates farther than rl from it
         * cannot pass the exact test for any member and are dropped before
         * it (a conservative FP32 test; the exact test decides the rest). */
        float bx0 = lane < ni ? own.x : 3.4e38f, by0 = lane < ni ? own.y : 3.4e38f, bz0 = lane < ni ? own.z : 3.4e38f;
        float bx1 = lane < ni ? own.x : -3.4e38f, by1 = lane < ni ? own.y : -3.4e38f,
              bz1 = lane < ni ? own.z : -3.4e38f;
        for (int o = 16; o > 0; o >>= 1) {
            bx0 = fminf(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
            by0 = fminf(by0, __shfl_xor_sync(0xffffffffu, by0, o));
            bz0 = fminf(bz0, __shfl_xor_sync(0xffffffffu, bz0, o));
            bx1 = fmaxf(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
            by1 = fmaxf(by1, __shfl_xor_sync(0xffffffffu, by1, o));
            bz1 = fmaxf(bz1, __shfl_xor_sync(0xffffffffu, bz1, o));
        }
        const float near_sq = G.shift ? G.rskinsq * 1.001f + 1e-4f : 3.4e38f;
        int fill = 0, head = 0;   /* queued candidates (in candidate order), the first one's slot */
        int kbase = -1;           /* the occupied stencil cells that begin before the round, less one */
        for (int cb = 0; cb < total; cb += CW_CHUNK) {
            const int ce = min(total, cb + CW_CHUNK);
            for (int k = lane; k < CW_CHUNK / 32; k += 32) ws.first[k] = 0u;
            __syncwarp();
            for (int k = lane; k < nne; k += 32) {
                const int pre = ws.pre[k] - cb;
                if (pre >= 0 && pre < CW_CHUNK) atomicOr(&ws.first[pre >> 5], 1u << (pre & 31));
            }
            __syncwarp();
            /* candidate g0 + lane: its stencil cell from the count of cells
             * that begin up to it, its position and type */
            auto fetch = [&](int g0, int &j, int &code, float4 &q, int &t) {
                if (g0 >= ce) return;
                const unsigned word = ws.first[(g0 - cb) >> 5];
                const int k = kbase + __popc(word & (lt * 2u + 1u)), g = g0 + lane;
                kbase += __popc(word);
                if (g < ce) {
                    j = ws.jb[k] + g;
                    code = ws.sh[k];
                    q = pos4[j];
                    t = type[j];
                }
            };
            auto near = [&](float4 q, int code) {
                const float4 u = ws.u[code];
                const float qx = q.x + u.x, qy = q.y + u.y, qz = q.z + u.z;
                const float ex = fmaxf(fmaxf(bx0 - qx, qx - bx1), 0.0f);
                const float ey = fmaxf(fmaxf(by0 - qy, qy - by1), 0.0f);
                const float ez = fmaxf(fmaxf(bz0 - qz, qz - bz1), 0.0f);
                return ex * ex + ey * ey + ez * ez < near_sq;
            };
            /* rounds of 64 candidates, software pipelined: the next round's
             * are located and loaded while this round's are filtered and a
             * queue is tested */
            int ja = 0, ca = 0, ta = 0, jc = 0, cc = 0, tc = 0;
            float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), qc = qa;
            fetch(cb, ja, ca, qa, ta);
            fetch(cb + 32, jc, cc, qc, tc);
            for (int g0 = cb; g0 < ce; g0 += 64) {
                const bool n0 = g0 + lane < ce && near(qa, ca), n1 = g0 + 32 + lane < ce && near(qc, cc);
                const unsigned nb0 = __ballot_sync(0xffffffffu, n0), nb1 = __ballot_sync(0xffffffffu, n1);
                if (n0) {
                    const int at = (head + fill + __popc(nb0 & lt)) & 127;
                    ws.fq[at] = make_float4(qa.x, qa.y, qa.z,
                                               __uint_as_float((unsigned)ja | ((unsigned)ta << MD_TYPE_SHIFT)));
                    ws.fc[at] = (unsigned char)ca;
                }
                fill += __popc(nb0);
                if (n1) {
                    const int at = (head + fill + __popc(nb1 & lt)) & 127;
                    ws.fq[at] = make_float4(qc.x, qc.y, qc.z,
                                               __uint_as_float((unsigned)jc | ((unsigned)tc << MD_TYPE_SHIFT)));
                    ws.fc[at] = (unsigned char)cc;
                }
                fill += __popc(nb1);
                fetch(g0 + 64, ja, ca, qa, ta);
                fetch(g0 + 96, jc, cc, qc, tc);
                __syncwarp();
                const bool end = g0 + 64 >= total;
                while (fill >= 64 || (end && fill > 0)) {
                    process(head, min(fill, 64));
                    head = (head + 64) & 127;
                    fill = max(fill - 64, 0);
                    __syncwarp();
                }
            }
        }
        /* pad every row to a multiple of 32 with the atom itself */
        for (int a = 0; a < ni; a++) {
            const int c = __shfl_sync(0xffffffffu, mycnt, a), ta = __shfl_sync(0xffffffffu, own_type, a);
            const int lim = min(kp.cap, (c + MD_LIST_QUANTUM - 1) / MD_LIST_QUANTUM * MD_LIST_QUANTUM);
            if (c + lane < lim)
                rows[(size_t)a * kp.cap + c + lane] = (unsigned)(i0 + a) | ((unsigned)ta << MD_TYPE_SHIFT);
        }
        if (lane < ni) {
            const int i = i0 + lane;
            nl_n[i] = mycnt < kp.cap ? mycnt : kp.cap;
            pos_old[i] = own;
            if (mycnt > kp.cap) atomicMax(&st->list_overflow, mycnt);
        }
        __syncwarp();
    }
}

/* ---- The whole rebuild as one cooperative kernel ---- */

constexpr unsigned long long MD_BAR_NS = 50000000ull;   /* 50 ms */

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void red_release(unsigned long long *p)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(1ull) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* One thread's wait until *count reaches target: at most bar_ns of global
 * time, after which it records the timeout in st->status and returns false.
 * The clock is read now and then. */
__device__ __forceinline__ bool bar_wait(const unsigned long long *count, unsigned long long target,
                                         unsigned long long bar_ns, md_devstate *st)
{
    int it = 0;
    unsigned long long t0 = 0;
    while (ld_acquire(count) < target) {
        if ((++it & 127) == 0) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > bar_ns) {
                atomicOr(&st->status, 1);
                return false;
            }
        }
    }
    return true;
}

/* Grid-wide barrier of `blocks` blocks that are all resident (a cooperative
 * launch): each adds one to a count and waits for it to reach the barrier's
 * multiple of blocks (MD_BAR_NS at most unless a test shortens it).  Returns
 * false in every thread of the block when its wait timed out: the caller
 * then returns at once.  A block passes a barrier only when every block has
 * reached it, i.e. after every block finished the phase before it, so no
 * phase runs on counts or prefix sums a barrier did not complete; blocks
 * that passed while another one gave up find that one absent at the next
 * barrier and leave there.  At the end arrive_last() adds the block without
 * a wait and returns true in the last one's threads, which then owns what
 * the kernel leaves for the next launch, the count's reset included.  (A
 * count and a generation on two lines, with a backoff in the polls, measured
 * 2 to 3 us more per rebuild.) */
struct grid_bar {
    md_devstate *st;
    unsigned blocks;
    unsigned long long bar_ns, target;
    __device__ __forceinline__ bool operator()()
    {
        __shared__ int s_ok;
        __syncthreads();
        target += blocks;
        if (threadIdx.x == 0) {
            red_release(&st->bar_count);
            s_ok = bar_wait(&st->bar_count, target, bar_ns, st);
        }
        __syncthreads();
        return s_ok != 0;
    }
    __device__ __forceinline__ bool arrive_last()
    {
        __shared__ int s_last;
        __syncthreads();
        target += blocks;
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicAdd(&st->bar_count, 1ull) + 1ull == target;
            if (s_last) {
                st->bar_count = 0ull;
                __threadfence();
            }
        }
        __syncthreads();
        return s_last != 0;
    }
};

/* The arrays the rebuild passes touch. */
struct rb_ptrs {
    const int *cell_rank, *cell_lin;
    int *key, *cell_count, *cell_start, *src;
    double *x, *v, *mass, *kick, *tmp_d;
    float4 *pos4, *tmp4, *pos_old;
    int *perm, *iperm, *type, *tmp_i;
    const uint4 *excl_orig;
    uint4 *excl_s;
    const int2 *bl_o;
    const int *bl_on;
    int2 *bl_s;
    int *bl_sn;
    const int4 *al_o;
    const int *al_on;
    int4 *al_s;
    int *al_sn;
    const unsigned *type_mask;
    unsigned *nl;
    int *nl_n;
    int ncells, has_bonds, has_angles;
    int parts;                   /* warps per cell of the list build (md_build_parts) */
    unsigned long long bar_ns;   /* limit of each barrier wait */
    int bar_drop;                /* test hook: this block leaves before the first barrier (-1: none) */
};

/* Warps per cell of the list build on a grid of `warps` warps: as many as
 * keep all of them busy once, at most one per atom of an average cell (each
 * part scans the stencil again, so cells are not split when there are more
 * of them than warps: halving the last round's measured 147 against 131 us
 * per build of 64000 ions). */
inline int md_build_parts(const md_ctx *c, int warps)
{
    const int per_cell = std::max(1, (c->n + c->ncells - 1) / c->ncells);
    return std::max(1, std::min(warps / std::max(1, c->ncells), per_cell));
}

inline rb_ptrs make_rb_ptrs(const md_ctx *c, int blocks)
{
    rb_ptrs p;
    p.parts = md_build_parts(c, blocks * CW_WARPS);
    p.cell_rank = c->cell_rank;
    p.cell_lin = c->cell_lin;
    p.key = c->key;
    p.cell_count = c->cell_count;
    p.cell_start = c->cell_start;
    p.src = c->src;
    p.x = c->x;
    p.v = c->v;
    p.mass = c->mass;
    p.kick = c->kick;
    p.tmp_d = c->tmp_d;
    p.pos4 = c->pos4;
    p.tmp4 = c->tmp4;
    p.pos_old = c->pos_old;
    p.perm = c->perm;
    p.iperm = c->iperm;
    p.type = c->type;
    p.tmp_i = c->tmp_i;
    p.excl_orig = c->excl_orig;
    p.excl_s = c->excl_s;
    p.bl_o = c->bl_o;
    p.bl_on = c->bl_on;
    p.bl_s = c->bl_s;
    p.bl_sn = c->bl_sn;
    p.al_o = c->al_o;
    p.al_on = c->al_on;
    p.al_s = c->al_s;
    p.al_sn = c->al_sn;
    p.type_mask = c->type_mask_dev;
    p.nl = c->nl;
    p.nl_n = c->nl_n;
    p.ncells = c->ncells;
    p.has_bonds = c->has_bonds;
    p.has_angles = c->has_angles;
    p.bar_ns = c->dbg_bar_ns > 0 ? c->dbg_bar_ns : MD_BAR_NS;
    p.bar_drop = c->dbg_bar_drop;
    return p;
}

/* Exclusive scan of up to SCAN_LOCAL cell counts by one block of CW_WARPS
 * warps into shared memory (buf); entry c of the result is at scan_pad(c). */
constexpr int SCAN_LOCAL = CW_WARPS * 32 * SCAN_K;
static_assert(sizeof(build_shm) >= sizeof(int) * (SCAN_LOCAL + SCAN_LOCAL / SCAN_K), "the scan's buffer");
__device__ __forceinline__ void scan_local(int ncells, const int *cell_count, int *buf)
{
    __shared__ int wsum[CW_WARPS];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int k = 0; k < SCAN_K; k++) {
        const int i = k * CW_WARPS * 32 + t;
        buf[scan_pad(i)] = i < ncells ? cell_count[i] : 0;
    }
    __syncthreads();
    int v[SCAN_K], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_K; k++) {
        v[k] = buf[scan_pad(t * SCAN_K + k)];
        sum += v[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int u = 0; u < w; u++) run += wsum[u];
#pragma unroll
    for (int k = 0; k < SCAN_K; k++) {
        buf[scan_pad(t * SCAN_K + k)] = run;
        run += v[k];
    }
    __syncthreads();
}

/* The block's share of the exclusive scan of many cell counts: it sums every
 * count before its share of the cells, then scans the share itself. */
__device__ __forceinline__ void scan_share(int ncells, const int *cell_count, int *cell_start)
{
    __shared__ int wsum[CW_WARPS];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int c0 = (int)((long long)ncells * blockIdx.x / gridDim.x),
              c1 = (int)((long long)ncells * (blockIdx.x + 1) / gridDim.x);
    int sum = 0;
#pragma unroll 4
    for (int c = t; c < c0; c += CW_WARPS * 32) sum += cell_count[c];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) wsum[w] = sum;
    __syncthreads();
    if (w == 0) {
        int run = 0;
        for (int u = 0; u < CW_WARPS; u++) run += wsum[u];
        for (int k = c0; k < c1; k += 32) {
            const int cnt = k + lane < c1 ? cell_count[k + lane] : 0;
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (k + lane < c1) cell_start[k + lane] = run + incl - cnt;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

/* The rebuild by blocks of CW_WARPS warps (stencils of up to CW_MAXST
 * cells), its phases separated by bar(), a barrier over every block of the
 * grid that returns false when its wait ran out; returns false then.  The
 * list and the new order are visible to every block after the caller's next
 * barrier.
 *
 *   bin       key and arrival number of every atom in its cell
 *   scan      up to SCAN_LOCAL cells: by every block for itself, with no
 *             barrier before the scatter; more: each block a share
 *   scatter   atoms into their cell's range in arrival order
 *   permute   every atom to its place: the cell's start plus the number of
 *             the cell's atoms with a smaller original index
 *   build     copy-back, remap and list build, all from the staged order
 *
 * Few barriers (3 with few cells, 4 with many; ~1.3 us each) and parts of
 * cells: a rebuild of a few thousand atoms is bound by latency. */
template <class Bar>
__device__ __forceinline__ bool rebuild_phases(const md_kparams &kp, md_devstate *st, const rb_ptrs &p, float4 *pos4,
                                               Bar &&bar)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    __shared__ build_shm sm;
    const int n = kp.n, P = kp.pitch;
    int *slot = p.tmp_i + 2 * (size_t)P;
    for (int i = tid; i < n; i += nth) slot[i] = key_one(kp, i, pos4, p.cell_rank, p.key, p.cell_count);
    if ((int)blockIdx.x == p.bar_drop) return false;
    if (!bar()) return false;
    /* every block has read the request by now, so it is cleared here */
    if (tid == 0) {
        st->update = 0;
        st->builds += 1;
        st->cell_next = 0;
    }
    if (p.ncells <= SCAN_LOCAL) {
        int *start = reinterpret_cast<int *>(&sm);
        scan_local(p.ncells, p.cell_count, start);
        if (blockIdx.x == 0) {
            for (int c = threadIdx.x; c < p.ncells; c += blockDim.x) p.cell_start[c] = start[scan_pad(c)];
            if (threadIdx.x == 0) p.cell_start[p.ncells] = n;
        }
        for (int i = tid; i < n; i += nth) p.src[start[scan_pad(p.key[i])] + slot[i]] = i;
    } else {
        scan_share(p.ncells, p.cell_count, p.cell_start);
        if (tid == 0) p.cell_start[p.ncells] = n;
        if (!bar()) return false;
        for (int i = tid; i < n; i += nth) p.src[p.cell_start[p.key[i]] + slot[i]] = i;
    }
    if (!bar()) return false;
    for (int s = tid; s < n; s += nth) {
        const int o = p.src[s], c = p.key[o], mine = p.perm[o];
        const int b = p.cell_start[c], e = p.cell_start[c + 1];
        int to = b;
#pragma unroll 4
        for (int k = b; k < e; k++) to += p.perm[p.src[k]] < mine ? 1 : 0;
        permute_one(kp, to, o, p.x, p.v, p.mass, p.kick, pos4, p.perm, p.type, p.tmp_d, p.tmp4, p.tmp_i);
        p.iperm[mine] = to;
    }
    for (int c = tid; c < p.ncells; c += nth) p.cell_count[c] = 0;   /* for the next build */
    if (!bar()) return false;
    const bool remap = p.has_bonds || p.has_angles;   /* the same in every block */
    for (int s = tid; s < n; s += nth) {
        copyback_one(kp, s, p.tmp_d, p.tmp4, p.tmp_i, p.x, p.v, p.mass, p.kick, pos4, p.perm, nullptr, p.type);
        if (remap)
            remap_one(kp, s, p.tmp_i, p.iperm, p.excl_orig, p.excl_s, p.bl_o, p.bl_on, p.bl_s, p.bl_sn, p.al_o,
                      p.al_on, p.al_s, p.al_sn, p.has_bonds, p.has_angles);
    }
    /* the list from the staged positions and types while the copy-back of
     * other blocks runs (it writes nothing the build reads) */
    const excl_src ex = {p.excl_s, remap ? p.excl_orig : nullptr, p.tmp_i, p.iperm, remap ? 1 : 0};
    const int lane = threadIdx.x & 31, items = p.ncells * p.parts;
    for (int it = tid >> 5; it < items;) {
        const int c = it / p.parts;
        build_part<false>(sm, c, it - c * p.parts, p.parts, kp, st, p.tmp4, p.tmp_i + P, ex, p.cell_rank, p.cell_lin,
                          p.cell_start, p.type_mask, p.nl, p.nl_n, p.pos_old, nullptr, nullptr, nullptr);
        if (items <= nth >> 5) break;   /* one item a warp */
        if (lane == 0) it = (nth >> 5) + atomicAdd(&st->cell_next, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
    }
    return true;
}

}  // namespace

#endif
