// Triangles near a sphere, in FP32.  Plain arithmetic, on the host as well
// (tests/cpp/triangle_near.cpp).
#pragma once

#ifdef __CUDACC__
#define XD_TRI __host__ __device__ __forceinline__
#define XD_TRI_COLD static __host__ __device__ __noinline__
#else
#include <cmath>
#define XD_TRI inline
#define XD_TRI_COLD inline
#endif

namespace xd {

// Squared distance from the origin to triangle abc in FP32 (the closest-point
// regions of Ericson, Real-Time Collision Detection 5.1.5, with the query
// point at the origin).  The distance is continuous across the regions, so a
// region misjudged by rounding moves it by rounding only, but the barycentric
// coordinates of a needle cancel: their error grows with the fourth power of
// length over width (tri_near).  face: the closest point is inside the face
// with every barycentric coordinate above 1e-5, beyond the FP32 rounding of
// all but needles, so the FP64 region test of the reference takes its face
// branch as well.
XD_TRI float tri_dist2_f(float ax, float ay, float az, float bx, float by, float bz, float cx, float cy, float cz,
                         bool& face)
{
    face = false;
    const float abx = bx - ax, aby = by - ay, abz = bz - az;
    const float acx = cx - ax, acy = cy - ay, acz = cz - az;
    const float d1 = -(abx * ax + aby * ay + abz * az), d2 = -(acx * ax + acy * ay + acz * az);
    if (d1 <= 0.f && d2 <= 0.f) return ax * ax + ay * ay + az * az;
    const float d3 = -(abx * bx + aby * by + abz * bz), d4 = -(acx * bx + acy * by + acz * bz);
    if (d3 >= 0.f && d4 <= d3) return bx * bx + by * by + bz * bz;
    const float vc = d1 * d4 - d3 * d2;
    float qx, qy, qz;
    if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
        const float v = d1 / (d1 - d3);
        qx = ax + v * abx;
        qy = ay + v * aby;
        qz = az + v * abz;
        return qx * qx + qy * qy + qz * qz;
    }
    const float d5 = -(abx * cx + aby * cy + abz * cz), d6 = -(acx * cx + acy * cy + acz * cz);
    if (d6 >= 0.f && d5 <= d6) return cx * cx + cy * cy + cz * cz;
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
        const float w = d2 / (d2 - d6);
        qx = ax + w * acx;
        qy = ay + w * acy;
        qz = az + w * acz;
        return qx * qx + qy * qy + qz * qz;
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        qx = bx + w * (cx - bx);
        qy = by + w * (cy - by);
        qz = bz + w * (cz - bz);
        return qx * qx + qy * qy + qz * qz;
    }
    const float den = 1.f / (va + vb + vc);
    const float v = vb * den, w = vc * den;
    face = va * den > 1e-5f && v > 1e-5f && w > 1e-5f;
    qx = ax + v * abx + w * acx;
    qy = ay + v * aby + w * acy;
    qz = az + v * abz + w * acz;
    return qx * qx + qy * qy + qz * qz;
}

// Whether a triangle with edges u and v is a needle for the mixed form's walls:
// (2 area)^2 below 1e-3 of the longest edge's fourth power, a width of some
// 1/30 of its length.  Their FP32 tests allow 5e-6 of |ab| + |ac| at least;
// above the line tri_dist2_f stays within 4e-6, and no contact of spheres from
// 0.03 to 15 mm is lost down to a tenth of it.  (Below it 2 to 5 % of the
// touches over the face of a strip of 300 by 0.3 mm were, with 1 mm spheres.)
XD_TRI bool tri_needle(float ux, float uy, float uz, float vx, float vy, float vz)
{
    const float uu = ux * ux + uy * uy + uz * uz, vv = vx * vx + vy * vy + vz * vz;
    const float uv = ux * vx + uy * vy + uz * vz, ll = fmaxf(fmaxf(uu, vv), uu + vv - 2.f * uv);
    return !(uu * vv - uv * uv > 1e-3f * ll * ll);
}

// tri_near's distance test of a triangle (edges u and v from vertex a) too thin
// for barycentric coordinates: the distance to its longest edge less its
// height.  d: the centre from a.  Out of line, as it is rare: a hopper of
// 17,159 spheres, which has no such triangle, takes 363.5 us, 365.2 with this
// in the search's loop (362.6 without it).
XD_TRI_COLD bool tri_edge_near(float dx, float dy, float dz, float reach, float ux, float uy, float uz, float vx,
                               float vy, float vz)
{
    const float uu = ux * ux + uy * uy + uz * uz, vv = vx * vx + vy * vy + vz * vz;
    const float wx = vx - ux, wy = vy - uy, wz = vz - uz, ww = wx * wx + wy * wy + wz * wz;
    const float nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    const float nn = nx * nx + ny * ny + nz * nz, ee = fmaxf(uu, fmaxf(vv, ww));
    if (!(ee > 1e-14f && ee < 1e30f)) return true;
    const bool bc = ww >= uu && ww >= vv, ab = !bc && uu >= vv;
    const float ex = bc ? wx : (ab ? ux : vx), ey = bc ? wy : (ab ? uy : vy), ez = bc ? wz : (ab ? uz : vz);
    if (bc) {
        dx -= ux;
        dy -= uy;
        dz -= uz;
    }
    const float t = fminf(fmaxf((dx * ex + dy * ey + dz * ez) / ee, 0.f), 1.f);
    dx -= t * ex;
    dy -= t * ey;
    dz -= t * ez;
    const float lim = reach + sqrtf(nn / ee) + 1e-4f * sqrtf(ee);
    return !(dx * dx + dy * dy + dz * dz > lim * lim);
}

// Whether a sphere (centre px, py, pz and radius r) may touch triangle abc:
// never false for one that does.  size: the sum of the sizes of the centre's
// coordinates.  All are FP32 values of FP64 ones, within 2^-23 of each.
//
// The triangle's box first, against the radius with a margin above the
// rounding of the coordinates, then its distance.  With N2 = (2 area)^2 and L
// the longest edge, tri_dist2_f is off by at most 3e-7 of |ab| + |ac| while
// N2 > 1e-2 L^2 max(L^2, r^2) (60,000,000 triangles of 0.01 to 1,000 radii;
// 1e-4 of it for N2 a hundred times smaller, 1e-2 for ten thousand times: a
// needle of 1 m by 10 um lost 0.4 % of its contacts), so the margin there is
// 1e-4.  A thinner triangle lies within its height N/L of the longest edge,
// whose distance has no such cancellation (tri_edge_near).  What is not finite, or too small
// for its squares, counts as near.
XD_TRI bool tri_near(float px, float py, float pz, float r, float size, float ax, float ay, float az, float bx,
                     float by, float bz, float cx, float cy, float cz)
{
    size += fabsf(ax) + fabsf(ay) + fabsf(az) + fabsf(bx) + fabsf(by) + fabsf(bz) + fabsf(cx) + fabsf(cy) + fabsf(cz);
    const float reach = r * 1.00001f + size * 1e-6f + 1e-15f;
    if (fminf(ax, fminf(bx, cx)) - px > reach || px - fmaxf(ax, fmaxf(bx, cx)) > reach) return false;
    if (fminf(ay, fminf(by, cy)) - py > reach || py - fmaxf(ay, fmaxf(by, cy)) > reach) return false;
    if (fminf(az, fminf(bz, cz)) - pz > reach || pz - fmaxf(az, fmaxf(bz, cz)) > reach) return false;
    const float ux = bx - ax, uy = by - ay, uz = bz - az, vx = cx - ax, vy = cy - ay, vz = cz - az;
    const float uu = ux * ux + uy * uy + uz * uz, vv = vx * vx + vy * vy + vz * vz;
    const float uv = ux * vx + uy * vy + uz * vz;
    // N2 and L^2, each within a few 1e-7 L^4 and L^2
    const float n2 = uu * vv - uv * uv, ll = fmaxf(fmaxf(uu, vv), uu + vv - 2.f * uv);
    if (n2 > 1e-2f * ll * fmaxf(ll, r * r) && n2 > 1e-30f) {
        bool face;
        const float d2 = tri_dist2_f(ax - px, ay - py, az - pz, bx - px, by - py, bz - pz, cx - px, cy - py, cz - pz,
                                     face);
        const float lim = reach + 1e-4f * (sqrtf(uu) + sqrtf(vv));
        return !(d2 > lim * lim);
    }
    return tri_edge_near(px - ax, py - ay, pz - az, reach, ux, uy, uz, vx, vy, vz);
}

}  // namespace xd
