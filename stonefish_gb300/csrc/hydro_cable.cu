// hydro_cable.cu -- CableEntity::ComputeHydrodynamicForces
// (Library/src/entities/CableEntity.cpp:240-376) for many cables at once.
//
// A cable is a chain of nodes; each segment between consecutive nodes is a
// cylinder of the cable's radius.  Per segment: the submerged volume from the
// depths of its end points (eight cases of partial submersion), buoyancy
// (-V rho g), form drag and skin friction from the mean node velocity
// relative to the current at the segment's midpoint; each segment gives half
// of each force to both of its nodes, and the end nodes' forces are doubled.
// A CTA takes 127 consecutive nodes of a cable: its 128 threads compute the
// segments around them into shared memory, then the nodes gather their two
// segments in the reference's order (the segment before, then the segment
// after).  All arithmetic is FP64 as in the reference; depths go through the
// FP32 Ocean::GetDepth as there.
//
// Bound: GB300 retires about two FP64 lanes per clock per SM, so the time is
// the number of FP64 operations.  A segment wholly on one side of the surface
// by more than the radius, which is most of them, needs neither its angle nor
// a share of its volume.  What is left runs the reference's operations one by
// one: the angle's cosine and sine as quotients of the sides are no faster
// (51.5 and 53.7 us) and a tenth less accurate where a segment crosses the
// surface; fused and regrouped drag products save 2 us.  300 cables of 100 to
// 400 nodes: 147 us with one warp per cable going through its segments 32 at
// a time, all with the angle, 54 us now.
#include <cstdint>
#include <cuda_runtime.h>

#include "hydro_internal.h"

namespace sfh {

namespace cable {

constexpr double kPi = 3.14159265358979323846;
constexpr double kEps = 2.220446049250313080847e-16;   // SIMD_EPSILON (double)

__device__ __forceinline__ bool fuzzy_zero(double x) { return fabs(x) < kEps; }

__device__ __forceinline__ double bt_acos(double x)
{
    if (x < -1.0) x = -1.0;
    if (x > 1.0) x = 1.0;
    return acos(x);
}

// CableEntity::circularSegmentArea (CableEntity.cpp:218-238)
__device__ double circular_segment_area(double h, double r)
{
    if (h <= 0.0) return 0.0;
    if (h >= 2.0 * r) return kPi * r * r;
    if (h > r) {
        h = 2.0 * r - h;
        const double theta = 2.0 * bt_acos((r - h) / r);
        return r * r * (kPi - (theta - sin(theta)) / 2.0);
    }
    const double theta = 2.0 * bt_acos((r - h) / r);
    return (r * r / 2.0) * (theta - sin(theta));
}

// Ocean::GetFluidVelocity(const Vector3&) (Ocean.cpp:183-196): FP64 sum of
// the enabled currents.
__device__ void fluid_velocity64(const OceanDev& o, const double* p, double* fv)
{
    fv[0] = fv[1] = fv[2] = 0.0;
    for (int i = 0; i < o.n_currents; ++i) {
        const hydro_current& c = o.currents[i];
        if (!c.enabled) continue;
        if (c.type == HYDRO_CURRENT_UNIFORM) {
            for (int k = 0; k < 3; ++k) fv[k] += c.vel[k];
        } else if (c.type == HYDRO_CURRENT_JET) {
            add_jet_velocity(c, p, fv);
        } else if (c.type == HYDRO_CURRENT_PIPE) {
            add_pipe_velocity<true>(c, p, fv);
        }
    }
}

// Ocean::GetDepth(const Vector3&) (Ocean.cpp:170-173): through FP32
__device__ __forceinline__ float depth32(const OceanDev& o, const double* p)
{
    return depth_at(o, (float)p[0], (float)p[1], (float)p[2]);
}

// One segment's contribution (Fb, Fdq, Fdf), to be halved onto its nodes.
__device__ void segment(const OceanDev& o, SettingsDev st, const hydro_cable& cb, const double* xa,
                        const double* xb, const double* va, const double* vb, double* out9)
{
    for (int k = 0; k < 9; ++k) out9[k] = 0.0;
    const double r = cb.radius;
    // the shallower point's depth first; the order of the points themselves
    // reaches the result only through squares and magnitudes
    const float da = depth32(o, xa), db = depth32(o, xb);
    const float f1 = da > db ? db : da, f2 = da > db ? da : db;
    // margin = r cos(alpha) is at most r, so beyond r on either side the
    // case is known without the angle
    const float rf = __double2float_ru(r);
    if (f2 < -rf && rf > 0.f) return;                         // out of the water
    const double d1 = (double)f1, d2 = (double)f2;
    const double sv[3] = {xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]};
    const double h2 = sv[0] * sv[0] + sv[1] * sv[1];
    const double L = sqrt(h2 + sv[2] * sv[2]);
    double V = 0.0;
    bool full = f1 > rf && rf > 0.f;
    if (full) {
        V = kPi * r * r * L;
    } else {
        const double dz = d2 - d1;
        const double dxy = h2 > kEps ? sqrt(h2) : 0.0;        // btVector3::safeNorm
        const double alpha = atan(dz / dxy), ca = cos(alpha), sa = sin(alpha);
        const double margin = fuzzy_zero(dxy) ? 0.0 : r * ca;
        if (d2 < -margin) {
            return;                                           // out of the water
        } else if (d1 > margin) {
            V = kPi * r * r * L;                              // fully submerged
            full = true;
        } else if (fuzzy_zero(dxy)) {                         // vertical
            const double l = d2 < dz ? d2 : dz;               // btMin
            V = kPi * r * r * l;
        } else if (fuzzy_zero(dz)) {                          // horizontal
            V = circular_segment_area(d1 + r, r) * L;
        } else if (fabs(d1) <= margin && fabs(d2) <= margin) {   // both caps partly submerged
            const double A1 = circular_segment_area(d1 / ca + r, r);
            const double A2 = circular_segment_area(d2 / ca + r, r);
            V = (A1 + A2) / 2.0 * L;
        } else if (d1 < -margin && d2 > margin) {             // first cap out, second submerged
            const double l1 = (d2 - r * ca) / sa;
            const double l2 = 2.0 * r * ca;
            V = kPi * r * r * (l1 + l2 / 2.0);
        } else if (d2 <= margin) {                            // first cap out, second partly
            const double a = r + d2 / ca;
            const double l = a / sa;
            V = circular_segment_area(a, r) * l / 2.0;
        } else if (d1 >= -margin) {                           // first cap partly, second submerged
            const double a = r - d1 / ca;
            const double l = a / sa;
            V = kPi * r * r * L - circular_segment_area(a, r) * l / 2.0;
        }
    }
    if (cb.buoyancy && st.buoyancy) {                         // :325-333
        const double k = -V * o.density;
        out9[0] = out9[1] = k * 0.0;
        out9[2] = k * o.gravity;
    }
    if (st.damping && V > 0.0) {                              // :335-364
        double rv[3];
        if (o.field_currents) {
            const double p[3] = {(xa[0] + xb[0]) * 0.5, (xa[1] + xb[1]) * 0.5, (xa[2] + xb[2]) * 0.5};
            fluid_velocity64(o, p, rv);
        } else {                                              // the same at every point
            fluid_velocity64(o, xa, rv);
        }
        for (int k = 0; k < 3; ++k) rv[k] = fma(va[k] + vb[k], 0.5, -rv[k]);
        const double Cd = 0.5;
        const double f1v = fabs(sv[0] * rv[0] + sv[1] * rv[1] + sv[2] * rv[2]);
        // a full segment's share is its volume over itself, one (not so for an infinite volume)
        const double share = full && V < 1e300 ? 1.0 : V / (kPi * r * r * L);
        const double rl = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
        const double S = 2.0 * r * L;
        const double q = -(1.0 - f1v) * share * 0.5 * o.density * Cd * S * rl;
        const double Sf = -(share * ((2.0 * kPi) * r * L));
        for (int k = 0; k < 3; ++k) {
            out9[3 + k] = q * rv[k];
            out9[6 + k] = Sf * rv[k];
        }
    }
}

}  // namespace cable

// Work item w = cable * per_cable + y takes the cable's chunks of 127 nodes
// y, y + per_cable, ...  A scene's cables of one kind tend to stand at a
// regular distance in the list and a grid that is resident all at once goes
// to the SMs in order, so consecutive items would load some SMs with wet
// chunks and others with dry or empty ones (the SMs were active 43% of the
// time); CTAs therefore take the items `stride` apart.
constexpr int kCableThreads = 128;
constexpr int kCableNodes = kCableThreads - 1;

__global__ void __launch_bounds__(kCableThreads) cable_kernel(const hydro_cable* __restrict__ cables,
                                                              uint32_t n_nodes_total, uint32_t per_cable,
                                                              uint64_t stride, const double* __restrict__ x,
                                                              const double* __restrict__ v, OceanDev o, SettingsDev st,
                                                              hydro_cable_node_forces* __restrict__ out)
{
    __shared__ double seg[kCableThreads][9];   // segment before the chunk's first node, ...
    static_assert(sizeof(hydro_cable_node_forces) == 9 * sizeof(double), "nodal forces are written as nine doubles");
    const uint64_t w = blockIdx.x * stride % gridDim.x;
    const hydro_cable cb = cables[w / per_cable];
    if (cb.mode != HYDRO_MODE_FLOATING && cb.mode != HYDRO_MODE_SUBMERGED) return;   // :242
    const uint32_t n = cb.n_nodes, f = cb.first_node;
    if ((uint64_t)f + n > n_nodes_total) return;              // node range outside the arrays
    for (uint64_t base = w % per_cable * kCableNodes; base < n; base += (uint64_t)per_cable * kCableNodes) {
        const uint64_t i = base + threadIdx.x;               // this thread's segment joins nodes i - 1 and i
        if (i > 0 && i < n) {
            const size_t a = 3 * (size_t)(f + i - 1);
            cable::segment(o, st, cb, x + a, x + a + 3, v + a, v + a + 3, seg[threadIdx.x]);
        }
        __syncthreads();
        const uint32_t count = (uint32_t)min((uint64_t)kCableNodes, n - base);
        double* dst = reinterpret_cast<double*>(out + f + base);
        for (uint32_t e = threadIdx.x; e < 9u * count; e += kCableThreads) {
            const uint32_t j = e / 9u, k = e - 9u * j;
            const uint64_t node = base + j;
            // from zero (:245-246): half of each of the node's segments; at an end node doubled (:367-373)
            double acc = 0.0;
            if (node > 0) acc += seg[j][k];
            if (node + 1 < n) acc += seg[j + 1][k];
            if (node > 0 && node + 1 < n) acc *= 0.5;
            dst[e] = acc;
        }
        __syncthreads();
    }
}

cudaError_t launch_cable(const hydro_cable* cables, uint32_t n_cables, uint32_t n_nodes_total, const double* x,
                         const double* v, OceanDev o, SettingsDev st, hydro_cable_node_forces* out, cudaStream_t s)
{
    if (n_cables == 0) return cudaSuccess;
    // four CTAs per cable take chunks in turn (one where that would exceed
    // the grid): a cable of up to 508 nodes is one chunk per CTA, and idle
    // CTAs return at once
    const uint32_t per_cable = n_nodes_total <= (uint32_t)kCableNodes || n_cables > (1u << 28) ? 1u : 4u;
    const uint32_t grid = n_cables * per_cable;
    uint64_t stride = 1;   // a prime that does not divide the grid, so that every item is taken once
    for (uint64_t p : {613u, 617u, 619u, 631u, 641u, 643u})
        if (grid % p != 0) {
            stride = p;
            break;
        }
    cable_kernel<<<grid, kCableThreads, 0, s>>>(cables, n_nodes_total, per_cable, stride, x, v, o, st, out);
    return cudaGetLastError();
}

}  // namespace sfh
