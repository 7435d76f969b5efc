// FP64 contact forces with the reference's semantics (the "plain" form):
// particle-particle (calculate_p2p_kernel<1>, mphysics_cuda_impl.cuh:403-485),
// particle-plane (plane_contact_force_kernel<1>, impl:572-621), particle-
// triangle (particle_polygonObject_collision_kernel<1>, impl:923-1021), the
// mesh update (impl:1911-1956), reductionD3 (def.cu:223-242) and a pair-list
// diagnostic.
//
// Compiled with --fmad=false.  Differences from the reference's arithmetic,
// all inside the stated FP64 tolerance:
//   * pow(cdist, 1.5) is evaluated as cdist * sqrt(cdist) (both within a few
//     ulp of the exact value; the FP64 pow is far more expensive on GB300);
//   * the pair-independent parts of getConstant (Eeq, beta = pi / ln e,
//     1 + beta^2, (4/3) Eeq) are computed once per thread from the contact
//     property instead of once per pair -- same expressions, same bits.
// Reference behaviour that is kept on purpose:
//   * Ft and M live across the pairs of one particle and are only assigned
//     when |e| != 0 (impl:390-400), so a pair with zero tangential slip adds
//     the previous pair's Ft and M again;
//   * planes and triangles are evaluated with ir = 0 in DHSModel, so they
//     apply no moment to the particle (impl:613-615, 1000-1002);
//   * corner contacts of a plane use u = (x - corner)/|x - corner|
//     (impl:506-529) and the third edge test can never pass (impl:549).
#include <cuda_runtime.h>

#include "xd_grid.cuh"
#include "xd_internal.cuh"
#include "xd_physics64.cuh"
#include "xd_scan.cuh"

namespace xd {

// ------------------------------------------------------- particle-particle

// Results of contacts in the block's ScanBuf (9 values): T = Fn + Ft (the
// normal force alone when the slip is zero), Ft, M.
enum { kContact = 1u, kSlip = 2u };

template <unsigned L>
__device__ __forceinline__ void put3(double (*res)[L], int a, unsigned lane, d3 v)
{
    res[a][lane] = v.x;
    res[a + 1][lane] = v.y;
    res[a + 2][lane] = v.z;
}
template <unsigned L>
__device__ __forceinline__ d3 get3(const double (*res)[L], int a, unsigned lane)
{
    return mk(res[a][lane], res[a + 1][lane], res[a + 2][lane]);
}

// A position and radius in FP32 for the search's near tests, and the sum of
// its coordinates' sizes, which bounds their rounding.
struct Near4 {
    float x, y, z, r, size;
};
__device__ __forceinline__ Near4 near_of(const d4& p)
{
    Near4 n{ f32_of(p.x), f32_of(p.y), f32_of(p.z), f32_of(p.w), 0.f };
    n.size = fabsf(n.x) + fabsf(n.y) + fabsf(n.z);
    return n;
}

// Whether two spheres may touch: the FP32 distance against the radii with a
// margin above the rounding of both (2^-23 of every coordinate, and of the
// sums).  A value that is not finite, and any distance below 1e-15 m (where
// squares leave the FP32 range), counts as near.
__device__ __forceinline__ bool spheres_near(const Near4& a, const Near4& b)
{
    const float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    const float lim = (a.r + b.r) * 1.000001f + (a.size + b.size) * 2e-7f;
    return !(d2 > lim * lim * 1.000002f && d2 > 1e-30f);
}

// calculate_p2p_kernel<1> (impl:403-485), a warp for 32 / LP particles.
//
// Bound by the FP64 pipe: some 250 operations a contact.  The candidates (65
// a particle on cells of one diameter, a thousand on the coarse cells of a
// mesh) are tested in FP32 from integer-cut coordinates, and the FP64 law
// runs on contacts alone, one per lane (xd_scan.cuh).  Every operation on a
// contact and the order of every sum are the thread-per-particle form's, so
// the results are the same bits.  A bed of 120,989 spheres: 327 us, 3.5 ms
// with the law evaluated where a thread found a contact; 8,000 spheres 37.5 us
// (438), 17,159 on a mesh's cells of 2.5 cm 213 us (2,527).
template <int LP, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW) k_p2p(Params P, const double* __restrict__ pos,
                                               const double* __restrict__ vel, const double* __restrict__ omega,
                                               double* __restrict__ force, double* __restrict__ moment,
                                               const double* __restrict__ mass, const unsigned* __restrict__ sorted,
                                               const unsigned* __restrict__ cstart, const unsigned* __restrict__ cend,
                                               const xd_contact_property* __restrict__ cp, unsigned np,
                                               unsigned each)
{
    using Buf = ScanBuf<LP, NW, double, 9>;
    __shared__ Buf B;
    __shared__ PairConst pc;
    if (threadIdx.x == 0) pc = load_pair_const(cp);   // (scan_contacts' barriers before the first use)
    constexpr unsigned NP = 32 / LP;
    const unsigned lane = threadIdx.x & 31u;
    for (unsigned b0 = blockIdx.x * each; b0 < np; b0 += gridDim.x * each) {
        const unsigned id0 = b0 + threadIdx.x / 32u * NP, id = id0 + lane / LP, end = min(np, b0 + each);
        const bool valid = id < end;
        d4 ip = d4{ 0, 0, 0, 0 };
        int3 gp = make_int3(0, 0, 0);
        if (valid) {
            ip = ld4(pos, id);
            gp = grid_pos_fast(P, ip.x, ip.y, ip.z);
        }
        const Near4 mine = near_of(ip);
        const unsigned runs = stage_runs<LP>(B, valid, gp, cstart, cend,
                                             [&](int x, int y, int z) { return grid_hash(P, x, y, z); });
        d3 Ft = mk(0, 0, 0), M = mk(0, 0, 0), sumF = mk(0, 0, 0), sumM = mk(0, 0, 0);
        scan_contacts<LP>(
            B, runs, sorted,
            [&](unsigned k, unsigned) { return k != id && k < np && spheres_near(mine, near_of(ld4(pos, k))); },
            [&](unsigned o, unsigned k, unsigned l) {
                const unsigned i = b0 + o;
                const d4 a = ld4(pos, i), b = ld4(pos, k);
                const d3 rp = mk(b.x - a.x, b.y - a.y, b.z - a.z);
                const double dist = length(rp);
                const double cdist = (a.w + b.w) - dist;
                if (!(cdist > 0)) return 0u;
                const d3 ivel = ld3(vel, i), jvel = ld3(vel, k), iomega = ld3(omega, i), jomega = ld3(omega, k);
                const d3 unit = rp / dist;
                const d3 rv = P.rolling ? (jvel + cross(jomega, -b.w * unit)) - (ivel + cross(iomega, a.w * unit))
                                        : (jvel - ivel);
                const Fc c = get_constant(pc, a.w, b.w, __ldg(mass + i), __ldg(mass + k));
                d3 Fn, t = mk(0, 0, 0), m = mk(0, 0, 0);
                const bool slip = dhs(c, a.w, b.w, pc.Ei, pc.Ej, pc.pri, pc.prj, pc.coh, cdist, rv, unit, P.dt, t,
                                      Fn, m);
                if (!slip) {
                    put3(B.res, 0, l, Fn);
                    return (unsigned)kContact;
                }
                put3(B.res, 0, l, Fn + t);
                put3(B.res, 3, l, t);
                put3(B.res, 6, l, m);
                return (unsigned)(kContact | kSlip);
            },
            [&](unsigned code, unsigned l) {
                d3 t = get3(B.res, 0, l);
                if (code & kSlip) {
                    Ft = get3(B.res, 3, l);
                    M = get3(B.res, 6, l);
                } else {   // the tangential force and moment of the contact before stay (impl:390-400)
                    t = t + Ft;
                }
                sumF += t;
                sumM += M;
            });
        const unsigned me = id0 + lane;
        if (lane < NP && me < end) {
            st3(force, me, ld3rw(force, me) + sumF);
            st3(moment, me, ld3rw(moment, me) + sumM);
        }
    }
}

// With tangential history: a thread per particle (the tables are read and
// written contact by contact in search order).
__global__ void __launch_bounds__(128) k_p2p_hist(Params P, const double* __restrict__ pos,
                                             const double* __restrict__ vel,
                                             const double* __restrict__ omega,
                                             double* __restrict__ force, double* __restrict__ moment,
                                             const double* __restrict__ mass,
                                             const unsigned* __restrict__ sorted,
                                             const unsigned* __restrict__ cstart,
                                             const unsigned* __restrict__ cend,
                                             const xd_contact_property* __restrict__ cp, unsigned np,
                                             HistTable ht)
{
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= np) return;
    HistState hs;
    hist_begin(ht, id, hs);
    const PairConst pc = load_pair_const(cp);
    d4 ip = ld4(pos, id);
    d3 ipos = xyz(ip);
    d3 ivel = ld3(vel, id);
    d3 iomega = ld3(omega, id);
    int3 gp = grid_pos(P, ip.x, ip.y, ip.z);
    double ir = ip.w;
    double im = __ldg(mass + id);
    d3 Ft = mk(0, 0, 0), Fn = mk(0, 0, 0), M = mk(0, 0, 0);
    d3 sumF = mk(0, 0, 0), sumM = mk(0, 0, 0);
    for (int z = -1; z <= 1; z++) {
        for (int y = -1; y <= 1; y++) {
            for (int x = -1; x <= 1; x++) {
                unsigned h = grid_hash(P, gp.x + x, gp.y + y, gp.z + z);
                unsigned st = __ldg(cstart + h);
                if (st == 0xffffffffu) continue;
                unsigned en = __ldg(cend + h);
                for (unsigned j = st; j < en; j++) {
                    unsigned k = __ldg(sorted + j);
                    if (id == k || k >= np) continue;
                    d4 jp = ld4(pos, k);
                    double jr = jp.w;
                    d3 rp = mk(jp.x - ipos.x, jp.y - ipos.y, jp.z - ipos.z);
                    double dist = length(rp);
                    double cdist = (ir + jr) - dist;
                    if (cdist > 0) {
                        d3 jvel = ld3(vel, k);
                        d3 jomega = ld3(omega, k);
                        double jm = __ldg(mass + k);
                        d3 unit = rp / dist;
                        d3 rv = P.rolling ? (jvel + cross(jomega, -jr * unit)) - (ivel + cross(iomega, ir * unit))
                                          : (jvel - ivel);
                        Fc c = get_constant(pc, ir, jr, im, jm);
                        Fn = normal_force(c, ir, jr, pc.Ei, pc.Ej, pc.pri, pc.prj, pc.coh, cdist, rv, unit);
                        d3 d;
                        int sl = hist_slot(ht, hs, id, k, d);
                        hist_tangential(c, ir, rv, unit, P.dt, Fn, d, Ft, M);
                        hist_store(ht, sl, id, d);
                        sumF += Fn + Ft;
                        sumM += M;
                    }
                }
            }
        }
    }
    hist_end(ht, hs, id, 0u);
    double* f = force + 3 * (size_t)id;
    double* m = moment + 3 * (size_t)id;
    f[0] += sumF.x; f[1] += sumF.y; f[2] += sumF.z;
    m[0] += sumM.x; m[1] += sumM.y; m[2] += sumM.z;
}

// ------------------------------------------------------------------ planes

// Planes applied in order; each adds Fn + Ft to the running force exactly
// like one plane_contact_force_kernel launch per plane.  cp_stride = 0
// shares one property (cube), 1 gives one per plane.
//
// Every region of plane_detection needs |wp.z| < r (wp.z the offset along
// uw), so a particle whose FP32 offset exceeds r by more than its rounding
// has no contact and adds zero.  The few that remain are gathered by block
// and run the FP64 code side by side: one warp of a block's eight instead of
// every warp that holds a particle near the wall.  8,000 spheres: 14 us a plane
// (30 to 45 before), 17 for all five in one launch.
__global__ void __launch_bounds__(256) k_planes(Params P, const xd_plane_info* __restrict__ planes,
                                                const xd_contact_property* __restrict__ cps, unsigned cp_stride,
                                                unsigned nplanes, const double* __restrict__ pos,
                                                const double* __restrict__ vel, const double* __restrict__ omega,
                                                double* __restrict__ force, double* __restrict__ moment,
                                                const double* __restrict__ mass, unsigned np)
{
    __shared__ unsigned near_of_block[256], who[256];
    __shared__ unsigned count;
    const unsigned mine = blockIdx.x * blockDim.x + threadIdx.x;
    Near4 p{};
    if (mine < np) p = near_of(ld4(pos, mine));
    for (unsigned w0 = 0; w0 < nplanes; w0 += 32u) {
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        unsigned near = 0;
        for (unsigned w = w0; w < min(nplanes, w0 + 32u); ++w) {
            const xd_plane_info* q = planes + w;
            const float ux = f32_of(__ldg(q->uw)), uy = f32_of(__ldg(q->uw + 1)), uz = f32_of(__ldg(q->uw + 2));
            const float x0 = f32_of(__ldg(q->xw)), y0 = f32_of(__ldg(q->xw + 1)), z0 = f32_of(__ldg(q->xw + 2));
            const float h = (p.x - x0) * ux + (p.y - y0) * uy + (p.z - z0) * uz;
            const float err = (fabsf(p.x) + fabsf(x0)) * fabsf(ux) + (fabsf(p.y) + fabsf(y0)) * fabsf(uy) +
                              (fabsf(p.z) + fabsf(z0)) * fabsf(uz);
            if (!(fabsf(h) > p.r * 1.000001f + err * 1e-6f + 1e-30f)) near |= 1u << (w - w0);
        }
        if (mine < np && near) {
            const unsigned t = atomicAdd(&count, 1u);
            near_of_block[t] = near;
            who[t] = mine;
        }
        __syncthreads();
        if (threadIdx.x < count) {
            const unsigned id = who[threadIdx.x];
            const double m = __ldg(mass + id);
            const d4 ip = ld4(pos, id);
            const d3 ipos3 = xyz(ip);
            const double r = ip.w;
            const d3 ivel = ld3(vel, id);
            const d3 iomega = ld3(omega, id);
            d3 f = ld3rw(force, id);
            d3 mo = ld3rw(moment, id);
            for (unsigned left = near_of_block[threadIdx.x]; left; left &= left - 1u) {
                const unsigned w = w0 + (unsigned)(__ffs(left) - 1);
                const PlaneD pe = load_plane(planes + w);
                d3 Fn = mk(0, 0, 0), Ft = mk(0, 0, 0), M = mk(0, 0, 0);
                const d3 dp = ipos3 - pe.xw;
                d3 unit = mk(0, 0, 0);
                const d3 wp = mk(dot(dp, pe.u1), dot(dp, pe.u2), dot(dp, pe.uw));
                const double cdist = plane_detection(pe, ipos3, wp, unit, r);
                if (cdist > 0) {
                    const PairConst pc = load_pair_const(cps + (size_t)w * cp_stride);
                    const d3 dv = P.rolling ? -(ivel + cross(iomega, r * unit)) : -ivel;
                    const Fc c = get_constant(pc, r, 0.0, m, 0.0);
                    dhs(c, 0, 0, 0, 0, 0, 0, pc.coh, cdist, dv, unit, P.dt, Ft, Fn, M);
                }
                f += Fn + Ft;
                mo += M;
            }
            st3(force, id, f);
            st3(moment, id, mo);
        }
        __syncthreads();
    }
}

// The same with tangential history, a thread per particle.
__global__ void __launch_bounds__(128) k_planes_hist(Params P, const xd_plane_info* __restrict__ planes,
                                                const xd_contact_property* __restrict__ cps,
                                                unsigned cp_stride, unsigned nplanes,
                                                const double* __restrict__ pos,
                                                const double* __restrict__ vel,
                                                const double* __restrict__ omega,
                                                double* __restrict__ force,
                                                double* __restrict__ moment,
                                                const double* __restrict__ mass, unsigned np,
                                                HistTable ht)
{
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= np) return;
    HistState hs;
    hist_begin(ht, id, hs);
    double m = __ldg(mass + id);
    d4 ip = ld4(pos, id);
    d3 ipos3 = xyz(ip);
    double r = ip.w;
    d3 ivel = ld3(vel, id);
    d3 iomega = ld3(omega, id);
    d3 f = ld3rw(force, id);
    d3 mo = ld3rw(moment, id);
    for (unsigned w = 0; w < nplanes; ++w) {
        PlaneD pe = load_plane(planes + w);
        d3 Fn = mk(0, 0, 0), Ft = mk(0, 0, 0), M = mk(0, 0, 0);
        d3 dp = ipos3 - pe.xw;
        d3 unit = mk(0, 0, 0);
        d3 wp = mk(dot(dp, pe.u1), dot(dp, pe.u2), dot(dp, pe.uw));
        double cdist = plane_detection(pe, ipos3, wp, unit, r);
        if (cdist > 0) {
            const xd_contact_property* cp = cps + (size_t)w * cp_stride;
            PairConst pc = load_pair_const(cp);
            d3 dv = P.rolling ? -(ivel + cross(iomega, r * unit)) : -ivel;
            Fc c = get_constant(pc, r, 0.0, m, 0.0);
            Fn = normal_force(c, 0, 0, 0, 0, 0, 0, pc.coh, cdist, dv, unit);
            d3 d;
            int sl = hist_slot(ht, hs, id, kHistPlane | w, d);
            hist_tangential(c, 0.0, dv, unit, P.dt, Fn, d, Ft, M);
            hist_store(ht, sl, id, d);
        }
        f += Fn + Ft;
        mo += M;
    }
    hist_end(ht, hs, id, 1u);
    st3(force, id, f);
    st3(moment, id, mo);
}

// ---------------------------------------------------------------- cylinder

// particle_cylinder_contact_detection (impl:652-719): the contact depth (the
// reference returns it as float), the unit normal u towards the cylinder and
// the contact point cp.  Rows A1..A3 of the Euler-parameter matrix
// (makeTFM_1..3, impl:624-637); toLocal multiplies by the transpose.
__device__ __forceinline__ double cylinder_detection(const xd_cylinder_info& cy, d3 p, double r, d3& u, d3& cp)
{
    const d3 pbase = mk(cy.pbase[0], cy.pbase[1], cy.pbase[2]);
    const d3 ptop = mk(cy.ptop[0], cy.ptop[1], cy.ptop[2]);
    const d3 ab = ptop - pbase;
    const double t = dot(p - pbase, ab) / dot(ab, ab);
    d3 c = pbase + t * ab;
    double dist = length(p - c);
    if (t >= 0 && t <= 1) {
        u = (c - p) / dist;
        cp = c - cy.rbase * u;
        return (double)(float)(cy.rtop + r - dist);
    }
    if (dist < cy.rbase) {
        const d3 o2c = mk(cy.origin[0], cy.origin[1], cy.origin[2]) - c;
        const double lo = length(o2c);
        u = o2c / lo;
        cp = c - cy.rbase * u;
        return (double)(float)(cy.len * 0.5 + r - lo);
    }
    const double ex = cy.ep[0], ey = cy.ep[1], ez = cy.ep[2], ew = cy.ep[3];
    const d3 A1 = mk(2.0 * (ex * ex + ey * ey - 0.5), 2.0 * (ey * ez - ex * ew), 2.0 * (ey * ew + ex * ez));
    const d3 A2 = mk(2.0 * (ey * ez + ex * ew), 2.0 * (ex * ex + ez * ez - 0.5), 2.0 * (ez * ew - ex * ey));
    const d3 A3 = mk(2.0 * (ey * ew - ex * ez), 2.0 * (ez * ew + ex * ey), 2.0 * (ex * ex + ew * ew - 0.5));
    d3 v = p - ptop;
    d3 at = mk(A1.x * v.x + A2.x * v.y + A3.x * v.z, A1.y * v.x + A2.y * v.y + A3.y * v.z,
               A1.z * v.x + A2.z * v.y + A3.z * v.z);
    cp = ptop;
    if (fabs(at.y) > cy.len) {
        v = p - pbase;
        at = mk(A1.x * v.x + A2.x * v.y + A3.x * v.z, A1.y * v.x + A2.y * v.y + A3.y * v.z,
                A1.z * v.x + A2.z * v.y + A3.z * v.z);
        cp = pbase;
    }
    const double ang = atan(at.x / at.z);
    if ((ang < 0 && at.z < 0) || (ang > 0 && at.x < 0 && at.z < 0)) c.x = cy.rbase * sin(-ang);
    else c.x = cy.rbase * sin(ang);
    c.z = cy.rbase * cos(ang);
    if ((at.z < 0 && c.z > 0) || (at.z > 0 && c.z < 0)) c.z = -c.z;
    c.y = 0.;
    cp = cp + mk(dot(A1, c), dot(A2, c), dot(A3, c));
    const d3 dis = cp - p;
    dist = length(dis);
    u = dis / dist;
    if (dist < r) return (double)(float)(r - dist);
    return -1.0;
}

// cylinder_hertzian_contact_force_kernel<1> (impl:721-760), one thread per
// particle.
__global__ void __launch_bounds__(256) k_cylinder(Params P, const xd_cylinder_info* __restrict__ cyl,
                                                  const xd_contact_property* __restrict__ cps,
                                                  const double* __restrict__ pos, const double* __restrict__ vel,
                                                  const double* __restrict__ omega, double* __restrict__ force,
                                                  double* __restrict__ moment, const double* __restrict__ mass,
                                                  unsigned np, const double* __restrict__ mpos,
                                                  double* __restrict__ mf, double* __restrict__ mm)
{
    const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= np) return;
    const xd_cylinder_info cy = *cyl;
    const double m = __ldg(mass + id);
    const d4 ip = ld4(pos, id);
    const d3 ivel = ld3(vel, id), iomega = ld3(omega, id);
    d3 unit = mk(0, 0, 0), cpt = mk(0, 0, 0);
    const double cdist = cylinder_detection(cy, xyz(ip), ip.w, unit, cpt);
    const d3 si = cpt - mk(__ldg(mpos), __ldg(mpos + 1), __ldg(mpos + 2));
    const d3 cy2cp = cpt - mk(cy.origin[0], cy.origin[1], cy.origin[2]);
    d3 Ft = mk(0, 0, 0), Fn = mk(0, 0, 0), M = mk(0, 0, 0);
    if (cdist > 0) {
        const d3 dv = mk(cy.vel[0], cy.vel[1], cy.vel[2]) + cross(mk(cy.omega[0], cy.omega[1], cy.omega[2]), cy2cp) -
                      (ivel + cross(iomega, ip.w * unit));
        const PairConst pc = load_pair_const(cps);
        const Fc c = get_constant(pc, ip.w, 0.0, m, 0.0);
        dhs(c, 0, 0, 0, 0, 0, 0, 0.0, cdist, dv, unit, P.dt, Ft, Fn, M);
    }
    st3(force, id, ld3rw(force, id) + (Fn + Ft));
    st3(moment, id, ld3rw(moment, id) + M);
    st3(mf, id, -Fn);
    st3(mm, id, cross(si, -Fn));
}

int launch_cylinder(const Params& P, const xd_cylinder_info* cyl, const xd_contact_property* cp,
                    const double* pos, const double* vel, const double* omega, double* force,
                    double* moment, const double* mass, unsigned np, const double* mpos, double* mf,
                    double* mm, cudaStream_t s)
{
    if (np == 0) return XD_OK;
    k_cylinder<<<div_up(np, 256), 256, 0, s>>>(P, cyl, cp, pos, vel, omega, force, moment, mass, np, mpos, mf, mm);
    return launch_status("cylinder contact");
}

// ---------------------------------------------------------------- polygons

__device__ __forceinline__ d3 ldp(const double* a) { return mk(__ldg(a), __ldg(a + 1), __ldg(a + 2)); }

__device__ __forceinline__ bool triangle_near(const Near4& p, const xd_polygon_info* __restrict__ t)
{
    return tri_near(p.x, p.y, p.z, p.r, p.size, f32_of(__ldg(t->P)), f32_of(__ldg(t->P + 1)), f32_of(__ldg(t->P + 2)),
                    f32_of(__ldg(t->Q)), f32_of(__ldg(t->Q + 1)), f32_of(__ldg(t->Q + 2)), f32_of(__ldg(t->R)),
                    f32_of(__ldg(t->R + 1)), f32_of(__ldg(t->R + 2)));
}

// particle_polygonObject_collision_kernel<1> (impl:923-1021), a warp for
// 32 / LP particles.
//
// A mesh's cells are as large as its triangles: here a particle's 27 cells
// hold a thousand particles and a hundred triangles or none, and few
// triangles touch it.  Entries are tested in FP32 (tri_near) and the
// FP64 closest point and law run on those that pass, one per lane, each
// particle adding its own in search order (xd_scan.cuh).  A bed of 17,159
// spheres on a cone of 4,096 triangles: 130 us, 3,512 with the closest point
// of every triangle in the cells formed in FP64 by a thread per particle.
//
// Reaction on the polygon bodies: NB > 0 keeps sums for NB bodies, summed per
// warp over all its particles by a fixed shuffle tree and over the warps by
// k_polygon_reaction_final; NB == 0 adds with atomics (used when the caller
// does not say how many bodies there are).
enum { kMoment = 4u, kBodyShift = 3u };

template <int NB, int LP, int NW>
__global__ void __launch_bounds__(32 * NW) k_polygon(Params P, const xd_polygon_info* __restrict__ dpi,
                                                xd_polygon_mass_info* __restrict__ dpmi,
                                                const double* __restrict__ pos, const double* __restrict__ vel,
                                                const double* __restrict__ omega, double* __restrict__ force,
                                                double* __restrict__ moment, const double* __restrict__ mass,
                                                const unsigned* __restrict__ sorted,
                                                const unsigned* __restrict__ cstart,
                                                const unsigned* __restrict__ cend,
                                                const xd_contact_property* __restrict__ cp,
                                                double* __restrict__ partials, unsigned each)
{
    using Buf = ScanBuf<LP, NW, double, 12>;
    __shared__ Buf B;
    constexpr int NBR = NB > 0 ? NB : 1;
    constexpr unsigned NP = 32 / LP;
    double react[NBR][6];
#pragma unroll
    for (int b = 0; b < NBR; ++b)
#pragma unroll
        for (int q = 0; q < 6; ++q) react[b][q] = 0.0;
    bool reacted = false;
    const unsigned cnp = P.np, lane = threadIdx.x & 31u;
    const unsigned warp = blockIdx.x * NW + threadIdx.x / 32u;
    for (unsigned b0 = blockIdx.x * each; b0 < cnp; b0 += gridDim.x * each) {
        const unsigned id0 = b0 + threadIdx.x / 32u * NP, id = id0 + lane / LP, end = min(cnp, b0 + each);
        const bool valid = id < end;
        d4 ip = d4{ 0, 0, 0, 0 };
        int3 gp = make_int3(0, 0, 0);
        if (valid) {
            ip = ld4(pos, id);
            gp = grid_pos_fast(P, ip.x, ip.y, ip.z);
        }
        const Near4 mine = near_of(ip);
        const unsigned runs = stage_runs<LP>(B, valid, gp, cstart, cend,
                                             [&](int x, int y, int z) { return grid_hash(P, x, y, z); });
        d3 Ft = mk(0, 0, 0), sumF = mk(0, 0, 0), sumM = mk(0, 0, 0);
        bool touched = false;
        scan_contacts<LP>(
            B, runs, sorted,
            [&](unsigned k, unsigned) { return k >= cnp && triangle_near(mine, dpi + (k - cnp)); },
            // values: Fn + Ft, Ft and the reaction's moment, or without slip Fn, -- and the contact point
            // from the body's origin; then M, where it is not zero (a normal that is not a number)
            [&](unsigned o, unsigned k, unsigned l) {
                const unsigned i = b0 + o;
                const xd_polygon_info* tri = dpi + (k - cnp);
                const d4 a = ld4(pos, i);
                const d3 ipos = xyz(a);
                const d3 Pv = ldp(tri->P), Qv = ldp(tri->Q), Rv = ldp(tri->R);
                const d3 cpt = closest_pt_triangle(Pv, Qv, Rv, ipos);
                const double dist = length(ipos - cpt);
                const double cdist = a.w - dist;
                if (!(cdist > 0)) return 0u;
                const unsigned pidx = (unsigned)__ldg(&tri->id);
                const xd_polygon_mass_info* pmi = dpmi + pidx;
                const d3 po2cp = cpt - ldv(pmi->origin);
                const d3 ivel = ld3(vel, i), iomega = ld3(omega, i);
                d3 unit = -cross(Qv - Pv, Rv - Pv);
                unit = unit / length(unit);
                const d3 pvel = ldv(pmi->vel), pom = ldv(pmi->omega);
                const d3 dv = P.rolling ? (pvel + cross(pom, po2cp)) - (ivel + cross(iomega, a.w * unit))
                                        : (pvel - ivel);
                const PairConst pc = load_pair_const(cp + pidx);
                const Fc c = get_constant(pc, a.w, 0, __ldg(mass + i), 0);
                d3 Fn, t = mk(0, 0, 0), m = mk(0, 0, 0);
                const bool slip = dhs(c, 0, 0, 0, 0, 0, 0, 0, cdist, dv, unit, P.dt, t, Fn, m);
                unsigned code = kContact | (pidx << kBodyShift);
                if (slip) {
                    code |= kSlip;
                    put3(B.res, 0, l, Fn + t);
                    put3(B.res, 3, l, t);
                    put3(B.res, 6, l, -cross(po2cp, Fn + t));
                    if (m.x != 0.0 || m.y != 0.0 || m.z != 0.0) {
                        code |= kMoment;
                        put3(B.res, 9, l, m);
                    }
                } else {
                    put3(B.res, 0, l, Fn);
                    put3(B.res, 6, l, po2cp);
                }
                return code;
            },
            [&](unsigned code, unsigned l) {
                d3 t = get3(B.res, 0, l), rm = get3(B.res, 6, l);
                if (code & kSlip) {
                    Ft = get3(B.res, 3, l);
                } else {
                    t = t + Ft;
                    rm = -cross(rm, t);
                }
                sumF += t;
                if (code & kMoment) sumM += get3(B.res, 9, l);
                touched = true;
                const unsigned pidx = code >> kBodyShift;
                if (NB == 0 || pidx >= (unsigned)NBR) {
                    // body count not declared, or an id beyond it: no slot, add directly
                    atomicAdd(dpmi[pidx].force + 0, -t.x);
                    atomicAdd(dpmi[pidx].force + 1, -t.y);
                    atomicAdd(dpmi[pidx].force + 2, -t.z);
                    atomicAdd(dpmi[pidx].moment + 0, rm.x);
                    atomicAdd(dpmi[pidx].moment + 1, rm.y);
                    atomicAdd(dpmi[pidx].moment + 2, rm.z);
                    return;
                }
#pragma unroll
                for (int b = 0; b < NBR; ++b)
                    if ((unsigned)b == pidx) {
                        react[b][0] -= t.x; react[b][1] -= t.y; react[b][2] -= t.z;
                        react[b][3] += rm.x; react[b][4] += rm.y; react[b][5] += rm.z;
                    }
            });
        const unsigned me = id0 + lane;
        if (touched) {   // lanes that own a particle; the others add zero
            st3(force, me, ld3rw(force, me) + sumF);
            st3(moment, me, ld3rw(moment, me) + sumM);
            reacted = true;
        }
    }
    if (NB > 0) {
        const bool any = __any_sync(kFullWarp, reacted);
#pragma unroll
        for (int b = 0; b < NBR; ++b)
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double v = react[b][q];
                if (any)
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFullWarp, v, o);
                if (lane == 0) partials[((size_t)warp * NBR + b) * 6 + q] = v;
            }
    }
}

// The same with tangential history, a thread per particle; the reactions
// summed by block (the tables are read and written contact by contact).
template <int NB>
__global__ void __launch_bounds__(128) k_polygon_hist(Params P, const xd_polygon_info* __restrict__ dpi,
                                                 xd_polygon_mass_info* __restrict__ dpmi,
                                                 const double* __restrict__ pos,
                                                 const double* __restrict__ vel,
                                                 const double* __restrict__ omega,
                                                 double* __restrict__ force,
                                                 double* __restrict__ moment,
                                                 const double* __restrict__ mass,
                                                 const unsigned* __restrict__ sorted,
                                                 const unsigned* __restrict__ cstart,
                                                 const unsigned* __restrict__ cend,
                                                 const xd_contact_property* __restrict__ cp,
                                                 double* __restrict__ partials, HistTable ht)
{
    constexpr int NBR = NB > 0 ? NB : 1;
    double react[NBR][6];
#pragma unroll
    for (int b = 0; b < NBR; ++b)
#pragma unroll
        for (int q = 0; q < 6; ++q) react[b][q] = 0.0;

    const unsigned cnp = P.np;
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id < cnp) {
        double im = __ldg(mass + id);
        d4 ip = ld4(pos, id);
        d3 ipos = xyz(ip);
        d3 ivel = ld3(vel, id);
        d3 iomega = ld3(omega, id);
        int3 gp = grid_pos(P, ip.x, ip.y, ip.z);
        double ir = ip.w;
        d3 M = mk(0, 0, 0), Fn = mk(0, 0, 0), Ft = mk(0, 0, 0);
        d3 sum_force = mk(0, 0, 0), sum_moment = mk(0, 0, 0);
        HistState hs;
        hist_begin(ht, id, hs);
        for (int z = -1; z <= 1; z++)
            for (int y = -1; y <= 1; y++)
                for (int x = -1; x <= 1; x++) {
                    unsigned h = grid_hash(P, gp.x + x, gp.y + y, gp.z + z);
                    unsigned st = __ldg(cstart + h);
                    if (st == 0xffffffffu) continue;
                    unsigned en = __ldg(cend + h);
                    for (unsigned j = st; j < en; j++) {
                        unsigned k = __ldg(sorted + j);
                        if (k < cnp) continue;
                        k -= cnp;
                        const xd_polygon_info* tri = dpi + k;
                        unsigned pidx = (unsigned)__ldg(&tri->id);
                        const xd_polygon_mass_info* pmi = dpmi + pidx;
                        d3 Pv = ldp(tri->P), Qv = ldp(tri->Q), Rv = ldp(tri->R);
                        d3 cpt = closest_pt_triangle(Pv, Qv, Rv, ipos);
                        d3 po2cp = cpt - ldv(pmi->origin);
                        d3 distVec = ipos - cpt;
                        double dist = length(distVec);
                        double cdist = ir - dist;
                        Fn = mk(0, 0, 0);
                        if (cdist > 0) {
                            d3 qp = Qv - Pv, rp = Rv - Pv;
                            d3 unit = -cross(qp, rp);
                            unit = unit / length(unit);
                            d3 pvel = ldv(pmi->vel), pom = ldv(pmi->omega);
                            d3 dv = P.rolling ? (pvel + cross(pom, po2cp)) - (ivel + cross(iomega, ir * unit))
                                              : (pvel - ivel);
                            PairConst pc = load_pair_const(cp + pidx);
                            Fc c = get_constant(pc, ir, 0, im, 0);
                            Fn = normal_force(c, 0, 0, 0, 0, 0, 0, 0, cdist, dv, unit);
                            d3 d;
                            int sl = hist_slot(ht, hs, id, kHistTri | k, d);
                            hist_tangential(c, 0.0, dv, unit, P.dt, Fn, d, Ft, M);
                            hist_store(ht, sl, id, d);
                            sum_force += Fn + Ft;
                            sum_moment += M;
                            d3 rf = -(Fn + Ft);
                            d3 rm = -cross(po2cp, Fn + Ft);
                            if (NB == 0) {
                                atomicAdd(dpmi[pidx].force + 0, rf.x);
                                atomicAdd(dpmi[pidx].force + 1, rf.y);
                                atomicAdd(dpmi[pidx].force + 2, rf.z);
                                atomicAdd(dpmi[pidx].moment + 0, rm.x);
                                atomicAdd(dpmi[pidx].moment + 1, rm.y);
                                atomicAdd(dpmi[pidx].moment + 2, rm.z);
                            } else if (pidx >= (unsigned)NBR) {
                                // body id beyond the declared count: no slot, add directly
                                atomicAdd(dpmi[pidx].force + 0, rf.x);
                                atomicAdd(dpmi[pidx].force + 1, rf.y);
                                atomicAdd(dpmi[pidx].force + 2, rf.z);
                                atomicAdd(dpmi[pidx].moment + 0, rm.x);
                                atomicAdd(dpmi[pidx].moment + 1, rm.y);
                                atomicAdd(dpmi[pidx].moment + 2, rm.z);
                            } else {
#pragma unroll
                                for (int b = 0; b < NBR; ++b)
                                    if ((unsigned)b == pidx) {
                                        react[b][0] += rf.x; react[b][1] += rf.y; react[b][2] += rf.z;
                                        react[b][3] += rm.x; react[b][4] += rm.y; react[b][5] += rm.z;
                                    }
                            }
                        }
                    }
                }
        hist_end(ht, hs, id, 2u);
        double* f = force + 3 * (size_t)id;
        double* m = moment + 3 * (size_t)id;
        f[0] += sum_force.x; f[1] += sum_force.y; f[2] += sum_force.z;
        m[0] += sum_moment.x; m[1] += sum_moment.y; m[2] += sum_moment.z;
    }
    if (NB > 0) {
        // fixed-order block tree reduction of the per-thread reactions
        __shared__ double red[128];
        for (int b = 0; b < NBR; ++b)
            for (int q = 0; q < 6; ++q) {
                red[threadIdx.x] = react[b][q];
                __syncthreads();
                for (int o = 64; o > 0; o >>= 1) {
                    if (threadIdx.x < (unsigned)o) red[threadIdx.x] += red[threadIdx.x + o];
                    __syncthreads();
                }
                if (threadIdx.x == 0) partials[((size_t)blockIdx.x * NBR + b) * 6 + q] = red[0];
                __syncthreads();
            }
    }
}

// Sums the partials of each body (of a warp, or of a block with history) in a
// fixed order and adds the total to dpmi[b].force / .moment: a block per
// component, so that its FP64 additions run on an SM of their own; thread t
// takes partials t, t + 128, ..., then a shuffle tree and the warps in order.
__global__ void __launch_bounds__(128) k_polygon_reaction_final(const double* __restrict__ partials, unsigned count,
                                                                unsigned nbr,
                                                                xd_polygon_mass_info* __restrict__ dpmi)
{
    __shared__ double part[4];
    const unsigned b = blockIdx.x / 6u, q = blockIdx.x % 6u;
    double s = 0.0;
#pragma unroll 4
    for (unsigned k = threadIdx.x; k < count; k += 128u) s += partials[((size_t)k * nbr + b) * 6 + q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(kFullWarp, s, o);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x / 32u] = s;
    __syncthreads();
    if (threadIdx.x) return;
    s = (part[0] + part[1]) + (part[2] + part[3]);
    if (q < 3u) dpmi[b].force[q] += s;
    else dpmi[b].moment[q - 3u] += s;
}

// ----------------------------------------------------------- mesh update

// toGlobal(double3&, double4&) (impl:1898-1909)

// updatePolygonObjectData_kernel (impl:1911-1956); t = 0 where the
// reference leaves it uninitialised (all three determinants <= 1e-13).
__global__ void __launch_bounds__(256) k_update_polygon(const xd_polygon_mass_info* __restrict__ dpmi,
                                                        const double* __restrict__ vlist,
                                                        double* __restrict__ sphere,
                                                        xd_polygon_info* __restrict__ dpi,
                                                        unsigned ntri)
{
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= ntri) return;
    d3 Pv, Qv, Rv;
    update_polygon_one(dpmi, nullptr, vlist, sphere, dpi, id, Pv, Qv, Rv);
}

// ----------------------------------------------------------- reductionD3

constexpr int kRedThreads = 256;
constexpr int kRedBlocksMax = 1024;

__global__ void __launch_bounds__(kRedThreads) k_reduce_d3_partial(const double* __restrict__ in,
                                                                   unsigned n,
                                                                   double* __restrict__ partial)
{
    __shared__ double red[3][kRedThreads];
    double s[3] = { 0.0, 0.0, 0.0 };
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        s[0] += in[3 * i];
        s[1] += in[3 * i + 1];
        s[2] += in[3 * i + 2];
    }
    for (int q = 0; q < 3; ++q) red[q][threadIdx.x] = s[q];
    __syncthreads();
    for (int o = kRedThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < (unsigned)o)
            for (int q = 0; q < 3; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; ++q) partial[3 * blockIdx.x + q] = red[q][0];
}

__global__ void k_reduce_d3_final(const double* __restrict__ partial, unsigned nb, double* __restrict__ out)
{
    if (threadIdx.x >= 3) return;
    double s = 0.0;
    for (unsigned b = 0; b < nb; ++b) s += partial[3 * b + threadIdx.x];
    out[threadIdx.x] = s;
}

// ------------------------------------------------------------- pair list

__device__ __forceinline__ unsigned pair_scan(const Params& P, const double* pos,
                                              const unsigned* sorted, const unsigned* cstart,
                                              const unsigned* cend, unsigned np, unsigned id,
                                              unsigned* out, unsigned cap_left)
{
    d4 ip = ld4(pos, id);
    int3 gp = grid_pos(P, ip.x, ip.y, ip.z);
    unsigned cnt = 0;
    for (int z = -1; z <= 1; z++)
        for (int y = -1; y <= 1; y++)
            for (int x = -1; x <= 1; x++) {
                unsigned h = grid_hash(P, gp.x + x, gp.y + y, gp.z + z);
                unsigned st = __ldg(cstart + h);
                if (st == 0xffffffffu) continue;
                unsigned en = __ldg(cend + h);
                for (unsigned j = st; j < en; j++) {
                    unsigned k = __ldg(sorted + j);
                    if (id == k || k >= np) continue;
                    d4 jp = ld4(pos, k);
                    d3 rp = mk(jp.x - ip.x, jp.y - ip.y, jp.z - ip.z);
                    double cdist = (ip.w + jp.w) - length(rp);
                    if (cdist > 0) {
                        if (out && cnt < cap_left) {
                            out[2 * cnt] = id;
                            out[2 * cnt + 1] = k;
                        }
                        cnt++;
                    }
                }
            }
    return cnt;
}

__global__ void k_pair_count(Params P, const double* __restrict__ pos, const unsigned* __restrict__ sorted,
                             const unsigned* __restrict__ cstart, const unsigned* __restrict__ cend,
                             unsigned np, unsigned* __restrict__ counts)
{
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= np) return;
    counts[id] = pair_scan(P, pos, sorted, cstart, cend, np, id, nullptr, 0);
}

__global__ void k_pair_fill(Params P, const double* __restrict__ pos, const unsigned* __restrict__ sorted,
                            const unsigned* __restrict__ cstart, const unsigned* __restrict__ cend,
                            unsigned np, const unsigned long long* __restrict__ offsets,
                            unsigned* __restrict__ pairs, unsigned long long cap)
{
    unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= np) return;
    unsigned long long o = offsets[id];
    if (o >= cap) return;
    unsigned long long left = cap - o;
    pair_scan(P, pos, sorted, cstart, cend, np, id, pairs + 2 * o,
              left > 0xffffffffull ? 0xffffffffu : (unsigned)left);
}

__global__ void k_pair_offsets(const unsigned* __restrict__ counts, unsigned np,
                               unsigned long long* __restrict__ offsets)
{
    // single thread: exclusive prefix in 64-bit (diagnostic path)
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    unsigned long long run = 0;
    for (unsigned i = 0; i < np; ++i) {
        offsets[i] = run;
        run += counts[i];
    }
    offsets[np] = run;
}

// ------------------------------------------------------------- launchers

int launch_p2p(const Params& P, const double* pos, const double* vel, const double* omega,
               double* force, double* moment, const double* mass, const unsigned* sorted,
               const unsigned* cstart, const unsigned* cend, const xd_contact_property* cp,
               unsigned np, cudaStream_t s, const HistTable* ht)
{
    if (np == 0) return XD_OK;
    if (ht) {
        k_p2p_hist<<<div_up(np, 128), 128, 0, s>>>(P, pos, vel, omega, force, moment, mass, sorted, cstart, cend,
                                                   cp, np, *ht);
        return launch_status("calculate_p2p");
    }
    scan_shape(np, [&](auto lp, auto nw) {
        constexpr int LP = decltype(lp)::value, NW = decltype(nw)::value;
        const ScanGrid g = scan_grid(np, LP, NW);
        k_p2p<LP, NW><<<g.blocks, 32 * NW, 0, s>>>(P, pos, vel, omega, force, moment, mass, sorted, cstart, cend, cp, np,
                                                   g.each);
    });
    return launch_status("calculate_p2p");
}

int launch_planes(const Params& P, const xd_plane_info* planes, const xd_contact_property* cps,
                  unsigned cp_stride, unsigned nplanes, const double* pos, const double* vel,
                  const double* omega, double* force, double* moment, const double* mass,
                  unsigned np, cudaStream_t s, const HistTable* ht)
{
    if (np == 0 || nplanes == 0) return XD_OK;
    if (ht)
        k_planes_hist<<<div_up(np, 128), 128, 0, s>>>(P, planes, cps, cp_stride, nplanes, pos, vel, omega, force,
                                                      moment, mass, np, *ht);
    else
        k_planes<<<div_up(np, 256), 256, 0, s>>>(P, planes, cps, cp_stride, nplanes, pos, vel, omega, force, moment,
                                                 mass, np);
    return launch_status("plane_contact_force");
}

static unsigned nbr_for(unsigned nbodies)
{
    if (nbodies == 0 || nbodies > 8) return 0;
    if (nbodies == 1) return 1;
    if (nbodies == 2) return 2;
    if (nbodies <= 4) return 4;
    return 8;
}

// Partials of the reaction: one per warp of the scan, or per block with history.
size_t polygon_scratch_bytes(unsigned np, unsigned nbodies)
{
    const unsigned nbr = nbr_for(nbodies);
    if (nbr == 0) return 0;
    const unsigned parts = div_up(np ? np : 1u, 128);
    return sizeof(double) * 6 * (size_t)nbr * (parts > kScanWarps ? parts : kScanWarps);
}

int launch_polygon(const Params& P, const xd_polygon_info* dpi, xd_polygon_mass_info* dpmi,
                   const double* pos, const double* vel, const double* omega, double* force,
                   double* moment, const double* mass, const unsigned* sidx,
                   const unsigned* cstart, const unsigned* cend, const xd_contact_property* cp,
                   unsigned nbodies, void* scratch, cudaStream_t s, const HistTable* ht)
{
    unsigned np = P.np;
    if (np == 0) return XD_OK;
    const unsigned nbr = nbr_for(nbodies);
    const unsigned nb = div_up(np, 128);
    unsigned parts = nb;   // of the reaction
    double* part = static_cast<double*>(scratch);
#define XD_POLY(NBV)                                                                                              \
    do {                                                                                                          \
        if (ht) {                                                                                                 \
            k_polygon_hist<NBV><<<nb, 128, 0, s>>>(P, dpi, dpmi, pos, vel, omega, force, moment, mass, sidx,      \
                                                   cstart, cend, cp, part, *ht);                                  \
        } else {                                                                                                  \
            scan_shape(np, [&](auto lp, auto nw) {                                                                \
                constexpr int LP = decltype(lp)::value, NW = decltype(nw)::value;                                 \
                const ScanGrid g = scan_grid(np, LP, NW);                                                         \
                parts = g.blocks * NW;                                                                            \
                k_polygon<NBV, LP, NW><<<g.blocks, 32 * NW, 0, s>>>(P, dpi, dpmi, pos, vel, omega, force, moment, \
                                                                    mass, sidx, cstart, cend, cp, part, g.each);  \
            });                                                                                                   \
        }                                                                                                         \
    } while (0)
    switch (nbr) {
    case 0: XD_POLY(0); break;
    case 1: XD_POLY(1); break;
    case 2: XD_POLY(2); break;
    case 4: XD_POLY(4); break;
    default: XD_POLY(8); break;
    }
#undef XD_POLY
    int st = launch_status("particle_polygon_collision");
    if (st != XD_OK || nbr == 0) return st;
    k_polygon_reaction_final<<<6 * nbodies, 128, 0, s>>>(part, parts, nbr, dpmi);
    return launch_status("particle_polygon_collision (reaction)");
}

// One step of prescribed body motion (an extension; the reference moves its
// bodies through the multibody solver on the host): origin += dt vel, the
// Euler parameters p <- q (x) p with q the rotation of angle |omega| dt about
// omega, normalised.  One thread per body.  The pose reached goes to pose (the
// mixed form's, which the mesh update then takes and gives to the body: the
// pose is computed while a contact pass still reads the body's), or in place.
__global__ void k_body_advance(xd_polygon_mass_info* __restrict__ pmi, unsigned nbodies, double dt,
                               double* __restrict__ pose, StepGate g)
{
    const unsigned b = threadIdx.x;
    if (b >= nbodies || (g.words && !step_moves(g, step_todo(g.words)))) return;
    xd_polygon_mass_info* m = pmi + b;
    double* o = pose ? pose + kPose * b : m->origin;
    double* ep = pose ? pose + kPose * b + 3 : m->ep;
    for (int a = 0; a < 3; ++a) o[a] = m->origin[a] + dt * m->vel[a];
    const double p0 = m->ep[0], p1 = m->ep[1], p2 = m->ep[2], p3 = m->ep[3];
    const double wx = m->omega[0], wy = m->omega[1], wz = m->omega[2];
    const double w = sqrt(wx * wx + wy * wy + wz * wz);
    if (w > 0.0) {
        const double h = 0.5 * w * dt;
        const double c = cos(h), sn = sin(h) / w;
        const double a0 = c, a1 = sn * wx, a2 = sn * wy, a3 = sn * wz;
        const double r0 = a0 * p0 - (a1 * p1 + a2 * p2 + a3 * p3);
        const double r1 = a0 * p1 + p0 * a1 + (a2 * p3 - a3 * p2);
        const double r2 = a0 * p2 + p0 * a2 + (a3 * p1 - a1 * p3);
        const double r3 = a0 * p3 + p0 * a3 + (a1 * p2 - a2 * p1);
        const double nr = sqrt(r0 * r0 + r1 * r1 + r2 * r2 + r3 * r3);
        ep[0] = r0 / nr;
        ep[1] = r1 / nr;
        ep[2] = r2 / nr;
        ep[3] = r3 / nr;
    } else if (pose) {
        ep[0] = p0;
        ep[1] = p1;
        ep[2] = p2;
        ep[3] = p3;
    }
}

int launch_body_advance(xd_polygon_mass_info* pmi, unsigned nbodies, double dt, cudaStream_t s, double* pose,
                        const StepGate& g)
{
    if (nbodies == 0) return XD_OK;
    k_body_advance<<<1, 32, 0, s>>>(pmi, nbodies, dt, pose, g);
    return launch_status("kinematic bodies");
}

// The mesh update and, for the mixed form, whether a vertex has moved from
// its position at the last list build (ref: FP32, relative to the grid origin
// wo) by disp2 or more: *flag is raised then.  rec (the mixed form's
// triangle records) is rewritten from the new vertices.  pose (nullable): the
// poses to place it at, which the bodies take over.  In a graph (g) it is
// part of a step: it runs beside the advance, and its blocks count with the
// advance's.
constexpr unsigned kMeshThreads = 64;

__global__ void __launch_bounds__(kMeshThreads) k_mesh_move(xd_polygon_mass_info* __restrict__ dpmi,
                                                            const double* __restrict__ pose, unsigned nbodies,
                                                            const double* __restrict__ vlist,
                                                            double* __restrict__ sphere,
                                                            xd_polygon_info* __restrict__ dpi, unsigned ntri,
                                                            const float* __restrict__ ref, double wo0, double wo1,
                                                            double wo2, float disp2, unsigned* __restrict__ flag,
                                                            TriRec* __restrict__ rec, StepGate g)
{
    const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned todo = g.words ? step_todo(g.words) : 0u;
    if (g.words && todo == 0) return;
    bool out = false;
    const bool moves = !g.words || step_moves(g, todo);
    if (moves && pose && id < nbodies) {   // (nobody else reads the bodies' poses here)
        for (int a = 0; a < 3; ++a) dpmi[id].origin[a] = pose[kPose * id + a];
        for (int a = 0; a < 4; ++a) dpmi[id].ep[a] = pose[kPose * id + 3 + a];
    }
    if (id < ntri && moves) {
        d3 V[3];
        update_polygon_one(dpmi, pose, vlist, sphere, dpi, id, V[0], V[1], V[2]);
        if (rec) write_tri_rec(rec + id, V[0], V[1], V[2], (unsigned)dpi[id].id);
        const double wo[3] = { wo0, wo1, wo2 };
        for (int k = 0; k < 3; ++k) {
            const double c[3] = { V[k].x, V[k].y, V[k].z };
            float d2 = 0.f;
            for (int a = 0; a < 3; ++a) {
                const float d = (float)(c[a] - wo[a]) - ref[9 * (size_t)id + 3 * k + a];
                d2 += d * d;
            }
            out |= !(d2 < disp2);
        }
    }
    if (!g.words) {
        if (__any_sync(0xffffffffu, out) && (threadIdx.x & 31u) == 0) atomicOr(flag, 1u);
        return;
    }
    const int raised = __syncthreads_or(out);
    if (threadIdx.x == 0) step_end(g, todo, raised != 0);
}

unsigned mesh_move_blocks(unsigned ntri) { return div_up(ntri, kMeshThreads); }

int launch_mesh_move(xd_polygon_mass_info* dpmi, const double* pose, unsigned nbodies, const double* vlist,
                     double* sphere, xd_polygon_info* dpi,
                     unsigned ntri, const float* ref, const double wo[3], float disp2, unsigned* flag,
                     TriRec* rec, cudaStream_t s, const StepGate& g)
{
    if (ntri == 0) return XD_OK;
    k_mesh_move<<<mesh_move_blocks(ntri), kMeshThreads, 0, s>>>(dpmi, pose, nbodies, vlist, sphere, dpi, ntri, ref,
                                                                wo[0], wo[1], wo[2], disp2, flag, rec, g);
    return launch_status("mesh move");
}

// The mixed form's triangle records of the mesh as it stands.
__global__ void __launch_bounds__(64) k_tri_records(const xd_polygon_info* __restrict__ dpi, unsigned ntri,
                                                    TriRec* __restrict__ rec)
{
    const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= ntri) return;
    const xd_polygon_info* t = dpi + id;
    write_tri_rec(rec + id, ldp3(t->P), ldp3(t->Q), ldp3(t->R), (unsigned)__ldg(&t->id));
}

int launch_tri_records(const xd_polygon_info* dpi, unsigned ntri, TriRec* rec, cudaStream_t s)
{
    if (ntri == 0) return XD_OK;
    k_tri_records<<<div_up(ntri, 64), 64, 0, s>>>(dpi, ntri, rec);
    return launch_status("triangle records");
}

int launch_update_polygon(const xd_polygon_mass_info* dpmi, const double* vlist, double* sphere,
                          xd_polygon_info* dpi, unsigned ntri, cudaStream_t s)
{
    if (ntri == 0) return XD_OK;
    // FP64-heavy and short: small blocks spread the triangles over every SM
    k_update_polygon<<<div_up(ntri, 64), 64, 0, s>>>(dpmi, vlist, sphere, dpi, ntri);
    return launch_status("update_polygon_object_data");
}

size_t reduction_scratch_bytes(unsigned n)
{
    (void)n;
    return sizeof(double) * 3 * (kRedBlocksMax + 1);
}

int reduction_d3(const double* in, unsigned n, double out[3], void* scratch, cudaStream_t s)
{
    double* part = static_cast<double*>(scratch);
    unsigned nb = div_up(n ? n : 1u, kRedThreads);
    if (nb > (unsigned)kRedBlocksMax) nb = kRedBlocksMax;
    k_reduce_d3_partial<<<nb, kRedThreads, 0, s>>>(in, n, part);
    k_reduce_d3_final<<<1, 32, 0, s>>>(part, nb, part + 3 * kRedBlocksMax);
    int st = launch_status("reductionD3");
    if (st != XD_OK) return st;
    cudaError_t e = cudaMemcpyAsync(out, part + 3 * kRedBlocksMax, 3 * sizeof(double),
                                    cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return cuda_status(e, "reductionD3 read-back");
}

size_t pair_list_scratch_bytes(unsigned np) { return sizeof(unsigned long long) * ((size_t)np + 1); }

int pair_list(const Params& P, const double* pos, const unsigned* sorted, const unsigned* cstart,
              const unsigned* cend, unsigned np, unsigned* counts, unsigned* pairs,
              unsigned long long cap, unsigned long long* total, void* scratch, cudaStream_t s)
{
    *total = 0;
    if (np == 0) return XD_OK;
    unsigned long long* off = static_cast<unsigned long long*>(scratch);
    k_pair_count<<<div_up(np, 128), 128, 0, s>>>(P, pos, sorted, cstart, cend, np, counts);
    k_pair_offsets<<<1, 1, 0, s>>>(counts, np, off);
    k_pair_fill<<<div_up(np, 128), 128, 0, s>>>(P, pos, sorted, cstart, cend, np, off, pairs, cap);
    int st = launch_status("pair_list");
    if (st != XD_OK) return st;
    cudaError_t e = cudaMemcpyAsync(total, off + np, sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    st = cuda_status(e, "pair_list read-back");
    if (st != XD_OK) return st;
    if (*total > cap) return set_error(XD_ERR_CAPACITY, "pair_list: %llu pairs > cap %llu", *total, cap);
    return XD_OK;
}

}  // namespace xd
