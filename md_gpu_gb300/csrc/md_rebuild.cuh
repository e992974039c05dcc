/*
 * md_rebuild.cuh -- the neighbour-list rebuild of a single system as phases
 * of one kernel: binning, one-block scan, scatter, in-cell order, permute,
 * copy-back, remap and the warp-per-cell list build, separated by a grid
 * barrier that the kernel brings.  k_rebuild_coop (k_cells.cu) is these
 * phases alone; k_run_steps (k_run.cu) runs them between its steps.
 */
#ifndef MD_REBUILD_CUH
#define MD_REBUILD_CUH

#include <type_traits>

#include "md_device.cuh"

namespace {

/* Cell rank (Hilbert order) of atom i and its count in the cell. */
__device__ __forceinline__ void key_one(const md_kparams &kp, int i, const float4 *__restrict__ pos4,
                                        const int *__restrict__ cell_rank, int *key, int *cell_count)
{
    float4 p = pos4[i];
    int cx = cell_of(cell_coord(p.x, kp.box[0], kp.boxi[0], kp.centered), kp.box[0], kp.binlen[0], kp.ncell[0]);
    int cy = cell_of(cell_coord(p.y, kp.box[1], kp.boxi[1], kp.centered), kp.box[1], kp.binlen[1], kp.ncell[1]);
    int cz = cell_of(cell_coord(p.z, kp.box[2], kp.boxi[2], kp.centered), kp.box[2], kp.binlen[2], kp.ncell[2]);
    int r = cell_rank[cx + kp.ncell[0] * (cy + kp.ncell[1] * cz)];
    key[i] = r;
    atomicAdd(&cell_count[r], 1);
}

/* Exclusive scan of the cell counts by one block of NT threads, then (ZERO)
 * zero the counters for the next build; returns the total in thread 0.
 * Without ZERO, cell_start may be cell_count itself (each round loads its
 * counts before it writes their starts).  In
 * rounds of NT x SCAN_K cells: the counts pass through shared memory, so
 * that global loads and stores are coalesced (one SM issues them all) while
 * each thread scans SCAN_K consecutive counts; warps scan their threads'
 * sums with shuffles and warp 0 the warp totals.  Shared index i is stored
 * at i + i / SCAN_K, so the per-thread reads hit distinct banks. */
constexpr int SCAN_K = 8;
__device__ __forceinline__ int scan_pad(int i) { return i + i / SCAN_K; }

template <int NT, bool ZERO = true>
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
                if (ZERO) {
                    cell_count[g] = 0;
                    cell_fill[g] = 0;
                }
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

/* Sorted slot s takes the state of atom src[s] (into the staging arrays). */
__device__ __forceinline__ void permute_one(const md_kparams &kp, int s, const int *__restrict__ src,
                                            const double *__restrict__ x, const double *__restrict__ v,
                                            const double *__restrict__ mass, const double *__restrict__ kick,
                                            const float4 *__restrict__ pos4, const int *__restrict__ perm,
                                            const int *__restrict__ type, double *tmp_d, float4 *tmp4,
                                            int *tmp_i)
{
    int o = src[s], P = kp.pitch;
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

/* The staged state back into the per-atom arrays, and the inverse order. */
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
    iperm[o] = s;
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

/* List build, one warp per cell: every atom of a cell shares the cell's
 * stencil.  The warp first gathers the stencil cells' atom ranges into
 * shared memory (in traversal order) with their prefix sums, then streams the
 * concatenated candidates 32 at a time (lane = candidate, its stencil cell
 * found by stepping forward through the prefix sums).  A conservative test
 * against the bounding box of the cell's atoms drops the candidates (about a
 * third) that no atom of the cell can reach; the rest enter a per-warp queue
 * in candidate order, and each full queue of 32 is tested exactly against
 * the cell's atoms, two at a time, a ballot per atom appending the hits to
 * its list.  Entries land in the
 * same order as in k_build_list (stencil cells in traversal order, ascending
 * j), so both builders produce identical lists. */
constexpr int CW_WARPS = 8;   /* warps per block (fewer blocks: fewer grid-barrier arrivals) */
constexpr int CW_MAXI = 32;
constexpr int CW_MAXST = 128;

/* Cell geometry seen by one warp: the system's, or in a batch the replica's
 * that owns the cell. */
struct cell_geom {
    float L[3], Li[3], rskinsq;
    int nc[3], sten[3], shift, lin0;
};

/* The list rows of the atoms of cell r (sorted rank), built by one warp. */
template <bool BATCH>
__device__ __forceinline__ void build_cell(
    int r, const md_kparams &kp, md_devstate *st, const float4 *__restrict__ pos4,
    const int *__restrict__ type, const uint4 *__restrict__ excl_s,
    const int *__restrict__ cell_rank, const int *__restrict__ cell_lin,
    const int *__restrict__ cell_start, const unsigned *__restrict__ type_mask, unsigned *nl,
    int *nl_n, float4 *pos_old, const md_rep *__restrict__ reps, const int *__restrict__ crep,
    const int *__restrict__ rep_upd)
{
    __shared__ float4 s_p[CW_WARPS][CW_MAXI];
    /* the group's coordinates once more by axis, so that two atoms' x (y, z)
     * are one aligned 8-byte load; slots past the group hold a far point */
    __shared__ __align__(16) float s_h[CW_WARPS][3][CW_MAXI];
    __shared__ uint4 s_ex[CW_WARPS][CW_MAXI];
    __shared__ unsigned s_tm[CW_WARPS][CW_MAXI];
    __shared__ int s_jb[CW_WARPS][CW_MAXST];
    __shared__ int s_pre[CW_WARPS][CW_MAXST + 1];
    __shared__ unsigned char s_sh[CW_WARPS][CW_MAXST];   /* image code per stencil cell */
    __shared__ float4 s_fq[CW_WARPS][64];                 /* queue of near candidates: position, */
    __shared__ unsigned s_fe[CW_WARPS][64];               /* list entry (j | type << 29) */
    __shared__ unsigned char s_fc[CW_WARPS][64];          /* and image code */
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ib = cell_start[r], ie = cell_start[r + 1];
    if (ib == ie) return;
    cell_geom G;
    if (BATCH) {
        const int rr = crep[r];
        if (!rep_upd[rr]) return;   /* this replica keeps its list */
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
    /* stencil ranges in traversal order (z outer, x inner); lane k takes k, k+32, ... */
    int run = 0;
    for (int k0 = 0; k0 < nst; k0 += 32) {
        int k = k0 + lane;
        int cnt = 0, jb = 0, code = 0;
        if (k < nst) {
            int dx = k % len[0], dy = (k / len[0]) % len[1], dz = k / (len[0] * len[1]);
            int xx = lo[0] + dx, yy = lo[1] + dy, zz = lo[2] + dz;
            /* code per axis: 0 no image, 1 the cell wrapped from below (the
             * reference's rint(d/L) = -1), 2 from above (+1) */
            code = (xx < 0 ? 1 : (xx >= nx ? 2 : 0)) | ((yy < 0 ? 1 : (yy >= ny ? 2 : 0)) << 2) |
                   ((zz < 0 ? 1 : (zz >= nz ? 2 : 0)) << 4);
            int cx = xx < 0 ? xx + nx : (xx >= nx ? xx - nx : xx);
            int cy = yy < 0 ? yy + ny : (yy >= ny ? yy - ny : yy);
            int cz = zz < 0 ? zz + nz : (zz >= nz ? zz - nz : zz);
            int r2 = cell_rank[G.lin0 + cx + nx * (cy + ny * cz)];
            jb = cell_start[r2];
            cnt = cell_start[r2 + 1] - jb;
        }
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (k < nst) {
            s_jb[w][k] = jb;
            s_pre[w][k] = run + incl - cnt;
            s_sh[w][k] = (unsigned char)code;
        }
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_pre[w][nst] = run;
    const int total = run;
    const unsigned lt = (1u << lane) - 1u;
    const float L0 = G.L[0], L1 = G.L[1], L2 = G.L[2];
    __syncwarp();
    for (int i0 = ib; i0 < ie; i0 += CW_MAXI) {
        const int ni = min(CW_MAXI, ie - i0);
        bool any_excl = false;
        {
            const float4 p = lane < ni ? pos4[i0 + lane] : make_float4(1e30f, 1e30f, 1e30f, 0.0f);
            s_h[w][0][lane] = p.x;
            s_h[w][1][lane] = p.y;
            s_h[w][2][lane] = p.z;
        }
        if (lane < ni) {
            int i = i0 + lane;
            s_p[w][lane] = pos4[i];
            uint4 ex = excl_s[i];
            s_ex[w][lane] = ex;
            unsigned tm = type_mask[type[i]];
            s_tm[w][lane] = tm;
            any_excl = ex.x != MD_EXCL_NONE || ex.y != MD_EXCL_NONE || ex.z != MD_EXCL_NONE ||
                       ex.w != MD_EXCL_NONE || tm != 0u;
        }
        const unsigned excl_bits = __ballot_sync(0xffffffffu, any_excl);
        __syncwarp();
        int mycnt = 0;   /* list length of atom i0 + lane */
        /* The exact test of 32 queued candidates against every atom of the
         * group; a ballot appends the hits to each atom's row in candidate
         * order.  An atom's row offset changes only in its own iteration, so
         * each iteration takes it from the counts at the start of the batch
         * and the iterations are independent (unrolled by 4: 156 against 168
         * us per build of 64000 ions with the count as a loop-carried
         * register). */
        auto process = [&](int cnt) {
            const bool vj = lane < cnt;
            const float4 q = vj ? s_fq[w][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            const unsigned entry = vj ? s_fe[w][lane] : 0u;
            const int code = vj ? s_fc[w][lane] : 0;
            const unsigned uj = entry & MD_INDEX_MASK;
            const int tj = (int)(entry >> MD_TYPE_SHIFT);
            /* exact images: u = L * rint(d / L) is -L, 0 or +L by stencil cell */
            const float ux = (code & 3) == 1 ? -L0 : ((code & 3) == 2 ? L0 : 0.0f);
            const float uy = ((code >> 2) & 3) == 1 ? -L1 : (((code >> 2) & 3) == 2 ? L1 : 0.0f);
            const float uz = ((code >> 4) & 3) == 1 ? -L2 : (((code >> 4) & 3) == 2 ? L2 : 0.0f);
            /* the group member this candidate is, if any (never its own neighbour) */
            const int selfa = (vj && (int)uj >= i0 && (int)uj < i0 + ni) ? (int)uj - i0 : -1;
            /* two copies of the loop: with and without the exclusion tests */
            auto loop = [&](auto with_excl) {
                unsigned *rowp = nl + (size_t)i0 * kp.cap;
                const int cnt0 = mycnt;
                int inc = 0;
#pragma unroll 4
                for (int a = 0; a < ni; a++, rowp += kp.cap) {
                    const float4 p = s_p[w][a];
                    float rsq;
                    if (G.shift) {
                        /* fl(fl(px - qx) - u) is the reference's fl(d - fl(L rint(d/L))) */
                        float dx = __fsub_rn(__fsub_rn(p.x, q.x), ux);
                        float dy = __fsub_rn(__fsub_rn(p.y, q.y), uy);
                        float dz = __fsub_rn(__fsub_rn(p.z, q.z), uz);
                        rsq = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                    } else {
                        rsq = md_rsq_box(p, q, G.L, G.Li);
                    }
                    bool ok = vj && rsq < G.rskinsq && a != selfa;
                    if (decltype(with_excl)::value && ((excl_bits >> a) & 1u)) {
                        uint4 ex = s_ex[w][a];
                        ok = ok && uj != ex.x && uj != ex.y && uj != ex.z && uj != ex.w &&
                             !((s_tm[w][a] >> tj) & 1u);
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, ok);
                    const int base = __shfl_sync(0xffffffffu, cnt0, a);
                    if (ok) {
                        const int slot = base + __popc(bal & lt);
                        if (slot < kp.cap) rowp[slot] = entry;
                    }
                    if (lane == a) inc += __popc(bal);
                }
                mycnt = cnt0 + inc;
            };
            if (excl_bits) {
                loop(std::true_type());
            } else if (G.shift) {
                /* two group atoms per iteration: the differences and squares
                 * in packed f32x2 instructions, the two sums in scalar adds
                 * with explicit rounding (a packed multiply followed by a
                 * packed add may be contracted into a packed FMA by the code
                 * generator, which would change the rounding of r^2) */
                typedef v2<true> V;
                const V QX = V::make(q.x, q.x), QY = V::make(q.y, q.y), QZ = V::make(q.z, q.z);
                const V UX = V::make(ux, ux), UY = V::make(uy, uy), UZ = V::make(uz, uz);
                const float far = vj ? G.rskinsq : -1.0f;   /* no hit in an empty slot */
                const int cnt0 = mycnt;
                int inc = 0;
#pragma unroll 4
                for (int a = 0; a < ni; a += 2) {
                    const float2 hx = *reinterpret_cast<const float2 *>(&s_h[w][0][a]);
                    const float2 hy = *reinterpret_cast<const float2 *>(&s_h[w][1][a]);
                    const float2 hz = *reinterpret_cast<const float2 *>(&s_h[w][2][a]);
                    const V dx = (V::make(hx.x, hx.y) - QX) - UX;
                    const V dy = (V::make(hy.x, hy.y) - QY) - UY;
                    const V dz = (V::make(hz.x, hz.y) - QZ) - UZ;
                    float x0, x1, y0, y1, z0, z1;
                    (dx * dx).get(x0, x1);
                    (dy * dy).get(y0, y1);
                    (dz * dz).get(z0, z1);
                    const float r0 = __fadd_rn(__fadd_rn(x0, y0), z0);
                    const float r1 = __fadd_rn(__fadd_rn(x1, y1), z1);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const bool ok = (h ? r1 : r0) < far && a + h != selfa;
                        const unsigned bal = __ballot_sync(0xffffffffu, ok);
                        const int base = __shfl_sync(0xffffffffu, cnt0, a + h);
                        const int slot = base + __popc(bal & lt);
                        if (ok && slot < kp.cap) nl[(size_t)(i0 + a + h) * kp.cap + slot] = entry;
                        inc += lane == a + h ? __popc(bal) : 0;
                    }
                }
                mycnt = cnt0 + inc;
            } else {
                loop(std::false_type());
            }
        };
        /* Bounding box of the group: candidates farther than rl from it
         * cannot pass the exact test for any member and are dropped before
         * it (a conservative FP32 test; the exact test decides the rest). */
        float bx0 = 3.4e38f, by0 = 3.4e38f, bz0 = 3.4e38f, bx1 = -3.4e38f, by1 = -3.4e38f, bz1 = -3.4e38f;
        if (lane < ni) {
            const float4 p = s_p[w][lane];
            bx0 = bx1 = p.x;
            by0 = by1 = p.y;
            bz0 = bz1 = p.z;
        }
        for (int o = 16; o > 0; o >>= 1) {
            bx0 = fminf(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
            by0 = fminf(by0, __shfl_xor_sync(0xffffffffu, by0, o));
            bz0 = fminf(bz0, __shfl_xor_sync(0xffffffffu, bz0, o));
            bx1 = fmaxf(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
            by1 = fmaxf(by1, __shfl_xor_sync(0xffffffffu, by1, o));
            bz1 = fmaxf(bz1, __shfl_xor_sync(0xffffffffu, bz1, o));
        }
        const float near_sq = G.rskinsq * 1.001f + 1e-4f;
        int fill = 0;   /* queued candidates (in candidate order) */
        int kc = 0;     /* this lane's stencil cell: the largest k with s_pre[k] <= g */
        /* software pipelined: the next round's candidate (its stencil cell,
         * position and type) is located and loaded while this round's are
         * filtered (144 against 156 us per build of 64000 ions) */
        int jn = 0, cn = 0, tn = 0;
        bool vn = lane < total;
        float4 qn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vn) {
            while (s_pre[w][kc + 1] <= lane) kc++;
            jn = s_jb[w][kc] + (lane - s_pre[w][kc]);
            cn = s_sh[w][kc];
            qn = pos4[jn];
            tn = type[jn];
        }
        for (int g0 = 0; g0 < total; g0 += 32) {
            const int j = jn, code = cn, tj = tn;
            const bool vj = vn;
            const float4 q = qn;
            {
                const int g = g0 + 32 + lane;
                vn = g < total;
                if (vn) {
                    while (s_pre[w][kc + 1] <= g) kc++;
                    jn = s_jb[w][kc] + (g - s_pre[w][kc]);
                    cn = s_sh[w][kc];
                    qn = pos4[jn];
                    tn = type[jn];
                }
            }
            bool near = vj;
            if (vj && G.shift) {
                const float qx = q.x + ((code & 3) == 1 ? -L0 : ((code & 3) == 2 ? L0 : 0.0f));
                const float qy = q.y + (((code >> 2) & 3) == 1 ? -L1 : (((code >> 2) & 3) == 2 ? L1 : 0.0f));
                const float qz = q.z + (((code >> 4) & 3) == 1 ? -L2 : (((code >> 4) & 3) == 2 ? L2 : 0.0f));
                const float ex = fmaxf(fmaxf(bx0 - qx, qx - bx1), 0.0f);
                const float ey = fmaxf(fmaxf(by0 - qy, qy - by1), 0.0f);
                const float ez = fmaxf(fmaxf(bz0 - qz, qz - bz1), 0.0f);
                near = ex * ex + ey * ey + ez * ez < near_sq;
            }
            const unsigned nb = __ballot_sync(0xffffffffu, near);
            if (near) {
                const int pos = fill + __popc(nb & lt);
                s_fq[w][pos] = q;
                s_fe[w][pos] = (unsigned)j | ((unsigned)tj << MD_TYPE_SHIFT);
                s_fc[w][pos] = (unsigned char)code;
            }
            fill += __popc(nb);
            __syncwarp();
            if (fill >= 32) {
                process(32);
                /* move the overflow to the front of the queue */
                float4 tq;
                unsigned te = 0;
                unsigned char tc = 0;
                const bool mv = lane < fill - 32;
                if (mv) {
                    tq = s_fq[w][32 + lane];
                    te = s_fe[w][32 + lane];
                    tc = s_fc[w][32 + lane];
                }
                __syncwarp();
                if (mv) {
                    s_fq[w][lane] = tq;
                    s_fe[w][lane] = te;
                    s_fc[w][lane] = tc;
                }
                fill -= 32;
                __syncwarp();
            }
        }
        if (fill > 0) process(fill);
        /* pad every row to a multiple of 32 with the atom itself */
        for (int a = 0; a < ni; a++) {
            int c = __shfl_sync(0xffffffffu, mycnt, a);
            int lim = min(kp.cap, (c + MD_LIST_QUANTUM - 1) / MD_LIST_QUANTUM * MD_LIST_QUANTUM);
            int k = c + lane;
            if (k < lim) {
                int ta = type[i0 + a];
                nl[(size_t)(i0 + a) * kp.cap + k] = (unsigned)(i0 + a) | ((unsigned)ta << MD_TYPE_SHIFT);
            }
        }
        if (lane < ni) {
            int i = i0 + lane;
            nl_n[i] = mycnt < kp.cap ? mycnt : kp.cap;
            pos_old[i] = s_p[w][lane];
            if (mycnt > kp.cap) atomicMax(&st->list_overflow, mycnt);
        }
        __syncwarp();
    }
}

/* ---- The whole rebuild of a single system as one cooperative kernel ---- */

/* Grid-wide barrier of the cooperative rebuild (every block is resident:
 * the kernel is launched cooperatively).  The last block to arrive resets
 * the count and advances the generation; the others wait for the
 * generation to change for at most bar_ns of global time (MD_BAR_NS unless
 * a test shortens it), after which they record the timeout in st->status.
 * Returns false in every thread of the block when its wait timed out: the
 * caller then returns at once.  A block passes a barrier only when every
 * block has reached it, i.e. after every block finished the phase before
 * it, so no phase runs on counts or prefix sums a barrier did not complete;
 * blocks that passed while another one gave up find that one absent at the
 * next barrier and leave there.  The waiting
 * blocks poll the generation, which lies on another cache line than the
 * arrival counter, so the polls do not slow the arrivals' atomics (the two
 * on one line cost ~12 us per rebuild of 64000 ions with 1216 blocks of 4
 * warps, ~1 us with the 608 blocks of 8 warps used now; a two-level barrier
 * measured no faster). */
constexpr unsigned long long MD_BAR_NS = 50000000ull;   /* 50 ms */

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool grid_barrier(md_devstate *st, unsigned long long bar_ns)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *gen = &st->bar_gen;
        const unsigned g = *gen;
        __threadfence();
        int ok = 1;
        if (atomicAdd(&st->bar_count, 1u) == gridDim.x - 1) {
            atomicExch(&st->bar_count, 0u);
            __threadfence();
            atomicAdd(&st->bar_gen, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            while (*gen == g) {
                if (global_ns() - t0 > bar_ns) {
                    atomicOr(&st->status, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(20);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

/* The order in which the list-building warps take the cells: most atoms
 * first (a counting sort of the cell ranks by atom count, counts above 63
 * together), so that the last cells handed out are the cheapest and the
 * warps finish close together.  Which warp builds a cell does not change
 * the cell's rows, so the order within a count may vary.  One block. */
__device__ __forceinline__ void work_order(int ncells, const int *cell_start, int *cell_work)
{
    __shared__ int s_at[64];
    if (threadIdx.x < 64) s_at[threadIdx.x] = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < ncells; c += blockDim.x)
        atomicAdd(&s_at[min(cell_start[c + 1] - cell_start[c], 63)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int m = 63; m >= 0; m--) {
            const int h = s_at[m];
            s_at[m] = run;
            run += h;
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < ncells; c += blockDim.x)
        cell_work[atomicAdd(&s_at[min(cell_start[c + 1] - cell_start[c], 63)], 1)] = c;
}

/* The arrays the rebuild passes touch. */
struct rb_ptrs {
    const int *cell_rank, *cell_lin;
    int *key, *cell_count, *cell_start, *cell_fill, *cell_work, *src;
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
    unsigned long long bar_ns;   /* limit of each barrier wait */
    int bar_drop;                /* test hook: this block leaves before the first barrier (-1: none) */
};

inline rb_ptrs make_rb_ptrs(const md_ctx *c)
{
    rb_ptrs p;
    p.cell_rank = c->cell_rank;
    p.cell_lin = c->cell_lin;
    p.key = c->key;
    p.cell_count = c->cell_count;
    p.cell_start = c->cell_start;
    p.cell_fill = c->cell_fill;
    p.cell_work = c->cell_work;
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

/* Binning, scan, scatter, in-cell order, permutation, remap and list build
 * of blocks of CW_WARPS warps (stencils of up to CW_MAXST cells), separated
 * by bar(), a barrier over every block of the grid that returns false when
 * its wait ran out; returns false then.  Ends with a barrier, so the list
 * and the new order are visible to every block. */
template <class Bar>
__device__ __forceinline__ bool rebuild_phases(const md_kparams &kp, md_devstate *st, const rb_ptrs &p, float4 *pos4,
                                               Bar &&bar)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const int n = kp.n;
    for (int i = tid; i < n; i += nth) key_one(kp, i, pos4, p.cell_rank, p.key, p.cell_count);
    if ((int)blockIdx.x == p.bar_drop) return false;
    if (!bar()) return false;
    /* one block scans (one barrier is dearer than its few rounds); every
     * block has read the request by now, so it is cleared here */
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) st->update = 0;
        const int total = scan_cells<CW_WARPS * 32>(p.ncells, p.cell_count, p.cell_start, p.cell_fill);
        if (threadIdx.x == 0) {
            p.cell_start[p.ncells] = total;
            st->builds += 1;
        }
        work_order(p.ncells, p.cell_start, p.cell_work);
    }
    if (!bar()) return false;
    for (int i = tid; i < n; i += nth) {
        const int r = p.key[i];
        p.src[p.cell_start[r] + atomicAdd(&p.cell_fill[r], 1)] = i;
    }
    if (!bar()) return false;
    {
        const int lane = threadIdx.x & 31, nw = nth >> 5;
        for (int c = tid >> 5; c < p.ncells; c += nw) {
            order_cell(c, p.cell_start, p.perm, p.src, nullptr, nullptr, lane);
            __syncwarp();
        }
    }
    if (!bar()) return false;
    for (int s = tid; s < n; s += nth)
        permute_one(kp, s, p.src, p.x, p.v, p.mass, p.kick, pos4, p.perm, p.type, p.tmp_d, p.tmp4, p.tmp_i);
    if (!bar()) return false;
    for (int s = tid; s < n; s += nth)
        copyback_one(kp, s, p.tmp_d, p.tmp4, p.tmp_i, p.x, p.v, p.mass, p.kick, pos4, p.perm, p.iperm, p.type);
    /* with bonds or angles the exclusions need the new order first; without,
     * the list build reads the sorted positions and types from the staging
     * arrays while the copy-back runs (it writes nothing the build reads) */
    const bool remap = p.has_bonds || p.has_angles;   /* the same in every block */
    if (remap) {
        if (!bar()) return false;
        for (int s = tid; s < n; s += nth)
            remap_one(kp, s, p.perm, p.iperm, p.excl_orig, p.excl_s, p.bl_o, p.bl_on, p.bl_s, p.bl_sn, p.al_o,
                      p.al_on, p.al_s, p.al_sn, p.has_bonds, p.has_angles);
        if (!bar()) return false;
    }
    {
        const float4 *bpos = remap ? pos4 : p.tmp4;
        const int *btype = remap ? p.type : p.tmp_i + kp.pitch;
        const int lane = threadIdx.x & 31;
        for (;;) {
            int r = 0;
            if (lane == 0) r = atomicAdd(&st->cell_next, 1);
            r = __shfl_sync(0xffffffffu, r, 0);
            if (r >= p.ncells) break;
            r = p.cell_work[r];
            build_cell<false>(r, kp, st, bpos, btype, p.excl_s, p.cell_rank, p.cell_lin, p.cell_start,
                              p.type_mask, p.nl, p.nl_n, p.pos_old, nullptr, nullptr, nullptr);
        }
    }
    if (!bar()) return false;
    if (tid == 0) st->cell_next = 0;
    return true;
}

}  // namespace

#endif
