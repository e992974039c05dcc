/*
 * md_bonded.cuh -- harmonic bonds and angles of one atom (bonded_forces.cu:
 * 34-193 as a per-atom gather), shared by the bonded kernel and the
 * many-step kernel of small systems.
 */
#ifndef MD_BONDED_CUH
#define MD_BONDED_CUH

#include "md_device.cuh"

namespace {

__device__ __forceinline__ void min_image(float &dx, float &dy, float &dz, const float *box, const float *boxi)
{
    dx -= box[0] * rintf(dx * boxi[0]);
    dy -= box[1] * rintf(dy * boxi[1]);
    dz -= box[2] * rintf(dz * boxi[2]);
}

/* Harmonic bonds (U = k (r - r0)^2, bnd1 = 2k) and angles (U = k (th - th0)^2,
 * ang1 = 2k) seen from sorted atom s with nb bonds and na angles: its force,
 * sum fa r^2 of the bonds and (ENERGY) its share of the energy, in FP32. */
template <bool ENERGY>
__device__ __forceinline__ void bonded_atom(int s, int P, int nb, int na, const float *box, const float *boxi,
                                            const float4 *pos4, const int2 *bl_s, const int4 *al_s,
                                            const float *par, float &fx, float &fy, float &fz, float &fw, float &fe)
{
    const float *bnd1 = par, *bnd2 = par + MD_MAXTYPE, *ang1 = par + 2 * MD_MAXTYPE,
                *ang2 = par + 3 * MD_MAXTYPE;
    float4 p = pos4[s];
    fx = fy = fz = fw = fe = 0.0f;
    for (int k = 0; k < nb; k++) {
        int2 b = bl_s[k * P + s];
        float4 q = pos4[b.x];
        float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        min_image(dx, dy, dz, box, boxi);
        float rsq = dx * dx + dy * dy + dz * dz;
        float ri = rsqrtf(rsq);
        float kk = bnd1[b.y], r0 = bnd2[b.y];
        float fa = kk * (r0 * ri - 1.0f);
        fw += fa * rsq;
        fx += fa * dx; fy += fa * dy; fz += fa * dz;
        if (ENERGY) { float dr = rsq * ri - r0; fe += 0.25f * kk * dr * dr; }
    }
    for (int k = 0; k < na; k++) {
        int4 a = al_s[k * P + s];
        float4 qa, qb = pos4[a.z];
        float4 cen;
        if (a.x == 1) { qa = pos4[a.y]; cen = p; }   /* this atom is the centre */
        else { qa = p; cen = pos4[a.y]; }           /* this atom is an end */
        float ax = qa.x - cen.x, ay = qa.y - cen.y, az = qa.z - cen.z;
        min_image(ax, ay, az, box, boxi);
        float bx = qb.x - cen.x, by = qb.y - cen.y, bz = qb.z - cen.z;
        min_image(bx, by, bz, box, boxi);
        float ai = rsqrtf(ax * ax + ay * ay + az * az);
        float bi = rsqrtf(bx * bx + by * by + bz * bz);
        float ab = ax * bx + ay * by + az * bz;
        float cang = ab * ai * bi;
        cang = fminf(fmaxf(cang, -0.9999999f), 0.9999999f);
        float th = acosf(cang);
        float ff = ang1[a.w] * (th - ang2[a.w]) * rsqrtf(1.0f - cang * cang) * ai * bi;
        float aa = ab * ai * ai;
        float gx = bx - aa * ax, gy = by - aa * ay, gz = bz - aa * az;
        if (a.x == 1) {
            float bb = ab * bi * bi;
            gx = bb * bx - ax - gx;
            gy = bb * by - ay - gy;
            gz = bb * bz - az - gz;
        }
        fx += ff * gx; fy += ff * gy; fz += ff * gz;
        if (ENERGY) { float dth = th - ang2[a.w]; fe += 0.5f * ang1[a.w] * dth * dth * (1.0f / 3.0f); }
    }
}

}  // namespace

#endif
