// hydro_rollout.cu -- device-resident rigid-body integration for rollouts of
// many independent hulls, without contacts, with the hydrodynamic wrench from
// either the exact step or the learned surrogate.  The reference steps its
// bodies with Bullet on the CPU; this restates, for free bodies only, how
// Bullet integrates a Stonefish rigid body (btRigidBody with
// BT_ENABLE_GYROSCOPIC_FORCE_IMPLICIT_BODY, set in SolidEntity.cpp:1086),
// so that thousands of environments can be rolled out without leaving the
// GPU.  Per step and hull, with R the body-to-world rotation of q:
//   F     = F_hydro + R f_thrust + (0, 0, mass g)           (NED: +z down)
//   tau_b = R^T T_hydro + t_thrust                           (body frame)
//   v'    = v + dt F / inertial_mass
//   w_b'  = w_b + dt I^-1 tau_b + dW_gyro(w_b)
//   p'    = p + dt v',   q' = exp(dt w') q   (exponential map, normalised)
// where dW_gyro is one Newton step of implicit Euler on I dw/dt = -w x I w
// (Catto, "Numerical Methods", GDC 2015; the method Bullet uses):
//   J = I + dt (skew(w) I - skew(I w)),  dW_gyro = -J^-1 (dt w x I w).
// The body record the hydrodynamics step reads is rewritten from the new
// state (T_CG = T_C = (R(q'), p'), R_O = R(q'), v', w', the rotated AABB).
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/stonefish_hydro.h"
#include "hydro_internal.h"

namespace sfh {

// GB300 retires about two FP64 lanes per clock per SM, so the step's time is
// its FP64 operation count: products are fused, divisions by the same number
// share a reciprocal, the Newton system is written in the differences of the
// inertias, and the exponential map of a small rotation is its Taylor series
// (no square root, division, sine or cosine).  16,384 hulls: 28 us with
// 463 FP64 instructions per hull and the records written field by field,
// 15.6 us now (246).
constexpr int kRigidBlock = 128;
// The two runs of words of hydro_body that a pose rewrites (8-byte words):
// T_CG, T_C, R_O, v, omega and the AABB.
constexpr uint32_t kBodyWords = sizeof(hydro_body) / 8;
constexpr uint32_t kPoseWords = 39, kBoxWord = 50, kBoxWords = 6;
constexpr uint32_t kOutWords = kPoseWords + kBoxWords;   // 45: odd, so a lane's rows are free of bank conflicts
static_assert(offsetof(hydro_body, T_CG) == 0 && offsetof(hydro_body, T_C) == 12 * 8 &&
                  offsetof(hydro_body, R_O) == 24 * 8 && offsetof(hydro_body, v) == 33 * 8 &&
                  offsetof(hydro_body, omega) == 36 * 8 && offsetof(hydro_body, aabb_min) == kBoxWord * 8 &&
                  offsetof(hydro_body, aabb_max) == (kBoxWord + 3) * 8,
              "pose words of hydro_body");

// row . u and column . u of a row-major 3 x 3 matrix
__device__ __forceinline__ double row_dot(const double* r, const double* u) { return fma(r[2], u[2], fma(r[1], u[1], r[0] * u[0])); }
__device__ __forceinline__ double col_dot(const double* r, const double* u) { return fma(r[6], u[2], fma(r[3], u[1], r[0] * u[0])); }

__device__ __forceinline__ void quat_to_rot(const double* q, double* R)
{
    const double w = q[0], x = q[1], y = q[2], z = q[3];
    const double x2 = x + x, y2 = y + y, z2 = z + z;
    R[0] = fma(-z, z2, fma(-y, y2, 1.0));
    R[1] = fma(x, y2, -(w * z2));
    R[2] = fma(x, z2, w * y2);
    R[3] = fma(x, y2, w * z2);
    R[4] = fma(-z, z2, fma(-x, x2, 1.0));
    R[5] = fma(y, z2, -(w * x2));
    R[6] = fma(x, z2, -(w * y2));
    R[7] = fma(y, z2, w * x2);
    R[8] = fma(-y, y2, fma(-x, x2, 1.0));
}

// The words of a body record that follow from a state, to `out` (45 words).
__device__ __forceinline__ void pose_words(const hydro_rigid_state& s, double* out)
{
    double R[9];
    quat_to_rot(s.q, R);
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k] = out[12 + k] = out[24 + k] = R[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        out[9 + k] = out[21 + k] = s.p[k];
        out[33 + k] = s.v[k];
        out[36 + k] = s.w[k];
        const double e = fma(fabs(R[3 * k + 2]), s.half_extents[2],
                             fma(fabs(R[3 * k + 1]), s.half_extents[1], fabs(R[3 * k]) * s.half_extents[0]));
        out[39 + k] = s.p[k] - e;
        out[42 + k] = s.p[k] + e;
    }
}

// A warp writes its lanes' pose words from shared memory, consecutive lanes
// consecutive words (bodies first ..., `count` of them).
__device__ __forceinline__ void store_poses(const double* rows, hydro_body* bodies, uint32_t first, uint32_t count)
{
    double* dst = reinterpret_cast<double*>(bodies + first);
    for (uint32_t e = threadIdx.x & 31u; e < count * kOutWords; e += 32u) {
        const uint32_t b = e / kOutWords, k = e - b * kOutWords;
        dst[(size_t)b * kBodyWords + (k < kPoseWords ? k : k - kPoseWords + kBoxWord)] = rows[e];
    }
}

// x = A^-1 b for a 3x3 row-major matrix (Cramer's rule; A is the Newton
// Jacobian I + O(dt), far from singular).
__device__ __forceinline__ void solve3(const double* A, const double* b, double* x)
{
    const double c0 = fma(A[4], A[8], -(A[5] * A[7]));
    const double c1 = fma(A[5], A[6], -(A[3] * A[8]));
    const double c2 = fma(A[3], A[7], -(A[4] * A[6]));
    const double inv = 1.0 / fma(A[2], c2, fma(A[1], c1, A[0] * c0));
    const double p = fma(b[2], A[5], -(b[1] * A[8])), q = fma(b[1], A[7], -(b[2] * A[4]));
    const double r = fma(b[2], A[3], -(b[1] * A[6]));
    x[0] = fma(A[2], q, fma(A[1], p, b[0] * c0)) * inv;
    x[1] = fma(A[2], r, fma(-A[0], p, b[0] * c1)) * inv;
    x[2] = fma(b[0], c2, fma(-A[0], q, -(A[1] * r))) * inv;
}

__global__ void __launch_bounds__(kRigidBlock) rigid_step_kernel(hydro_rigid_state* __restrict__ states,
                                                                 hydro_body* __restrict__ bodies,
                                                                 const hydro_wrench* __restrict__ exact,
                                                                 const float* __restrict__ body_wrench, uint32_t n,
                                                                 double dt, double gravity)
{
    __shared__ double rows[kRigidBlock / 32][32 * kOutWords];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    if (i < n) {
        hydro_rigid_state s = states[i];
        double R[9];
        quat_to_rot(s.q, R);
        // world force and body torque: the wrench, the thrusters, gravity
        double F[3] = {0, 0, 0}, Tb[3], fb[3];
        for (int k = 0; k < 3; ++k) {
            fb[k] = s.thrust_force[k];
            Tb[k] = s.thrust_torque[k];
        }
        if (exact) {
            const hydro_wrench& x = exact[i];
            double T[3];
            for (int k = 0; k < 3; ++k) {
                F[k] = x.Fb[k] + x.Fdq[k] + x.Fdf[k];
                T[k] = x.Tb[k] + x.Tdq[k] + x.Tdf[k];
            }
            for (int k = 0; k < 3; ++k) Tb[k] += col_dot(R + k, T);
        } else if (body_wrench) {
            const float* w = body_wrench + (size_t)i * 6;
            for (int k = 0; k < 3; ++k) {
                fb[k] += (double)w[k];
                Tb[k] += (double)w[3 + k];
            }
        }
        for (int k = 0; k < 3; ++k) F[k] += row_dot(R + 3 * k, fb);
        F[2] = fma(s.mass, gravity, F[2]);
        // angular velocity, body frame: external torque impulse plus the
        // implicit gyroscopic step, both from the current angular velocity.
        // With J = I + dt (skew(w) diag(I) - skew(I w)) and f = dt w x I w,
        // every off-diagonal entry is dt times a difference of inertias times
        // a component of w, and f's components are its entries times another.
        const double* I = s.inertia;
        double wb[3];
        for (int k = 0; k < 3; ++k) wb[k] = col_dot(R + k, s.w);
        const double a = dt * (I[2] - I[1]), b = dt * (I[0] - I[2]), c = dt * (I[1] - I[0]);
        const double J[9] = {I[0], a * wb[2], a * wb[1], b * wb[2], I[1], b * wb[0], c * wb[1], c * wb[0], I[2]};
        const double f[3] = {J[1] * wb[1], J[3] * wb[0], J[6] * wb[0]};
        double dg[3];
        solve3(J, f, dg);
        for (int k = 0; k < 3; ++k) wb[k] += dt * Tb[k] / I[k] - dg[k];
        for (int k = 0; k < 3; ++k) s.w[k] = row_dot(R + 3 * k, wb);
        // linear velocity and position
        const double dm = dt / s.inertial_mass;
        for (int k = 0; k < 3; ++k) {
            s.v[k] = fma(F[k], dm, s.v[k]);
            s.p[k] = fma(dt, s.v[k], s.p[k]);
        }
        // orientation: rotation by |w| dt about w, applied in the world
        // frame: (cos h, sin h w / |w|), h = |w| dt / 2.  Below h = 1/4 by
        // the series of cos h and of sin h / h, whose first term left out is
        // below 2^-64 of the sum.
        const double w2 = row_dot(s.w, s.w);
        const double h2 = 0.25 * dt * dt * w2;
        double co, sc;
        if (h2 < 0.0625) {
            co = fma(h2, -1.0 / 87178291200.0, 1.0 / 479001600.0);
            co = fma(h2, co, -1.0 / 3628800.0);
            co = fma(h2, co, 1.0 / 40320.0);
            co = fma(h2, co, -1.0 / 720.0);
            co = fma(h2, co, 1.0 / 24.0);
            co = fma(h2, co, -0.5);
            co = fma(h2, co, 1.0);
            sc = fma(h2, 1.0 / 6227020800.0, -1.0 / 39916800.0);
            sc = fma(h2, sc, 1.0 / 362880.0);
            sc = fma(h2, sc, -1.0 / 5040.0);
            sc = fma(h2, sc, 1.0 / 120.0);
            sc = fma(h2, sc, -1.0 / 6.0);
            sc = fma(h2, sc, 1.0) * (0.5 * dt);
        } else {
            const double wn = sqrt(w2);
            const double half = 0.5 * wn * dt;
            co = cos(half);
            sc = sin(half) / wn;
        }
        const double dq[4] = {co, sc * s.w[0], sc * s.w[1], sc * s.w[2]};
        const double qw = s.q[0], qx = s.q[1], qy = s.q[2], qz = s.q[3];
        const double nq[4] = {fma(-dq[3], qz, fma(-dq[2], qy, fma(-dq[1], qx, dq[0] * qw))),
                              fma(-dq[3], qy, fma(dq[2], qz, fma(dq[1], qw, dq[0] * qx))),
                              fma(dq[3], qx, fma(dq[2], qw, fma(-dq[1], qz, dq[0] * qy))),
                              fma(dq[3], qw, fma(-dq[2], qx, fma(dq[1], qy, dq[0] * qz)))};
        const double inv = rsqrt(fma(nq[3], nq[3], fma(nq[2], nq[2], fma(nq[1], nq[1], nq[0] * nq[0]))));
        for (int k = 0; k < 4; ++k) s.q[k] = nq[k] * inv;
        hydro_rigid_state& out = states[i];   // p, q, v and w; the rest stays
        for (int k = 0; k < 3; ++k) {
            out.p[k] = s.p[k];
            out.v[k] = s.v[k];
            out.w[k] = s.w[k];
        }
        for (int k = 0; k < 4; ++k) out.q[k] = s.q[k];
        pose_words(s, rows[wib] + lane * kOutWords);
    }
    __syncwarp();
    const uint32_t first = i - lane;
    if (first < n) store_poses(rows[wib], bodies, first, min(32u, n - first));
}

__global__ void __launch_bounds__(kRigidBlock) rigid_write_bodies_kernel(const hydro_rigid_state* __restrict__ states,
                                                                         hydro_body* __restrict__ bodies, uint32_t n)
{
    __shared__ double rows[kRigidBlock / 32][32 * kOutWords];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    if (i < n) pose_words(states[i], rows[wib] + lane * kOutWords);
    __syncwarp();
    const uint32_t first = i - lane;
    if (first < n) store_poses(rows[wib], bodies, first, min(32u, n - first));
}

cudaError_t launch_rigid_step(hydro_rigid_state* states, hydro_body* bodies, const hydro_wrench* exact,
                              const float* body_wrench, uint32_t n, double dt, double gravity, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    rigid_step_kernel<<<(n + kRigidBlock - 1) / kRigidBlock, kRigidBlock, 0, s>>>(states, bodies, exact, body_wrench, n, dt, gravity);
    return cudaGetLastError();
}

cudaError_t launch_rigid_write_bodies(const hydro_rigid_state* states, hydro_body* bodies, uint32_t n,
                                      cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    rigid_write_bodies_kernel<<<(n + kRigidBlock - 1) / kRigidBlock, kRigidBlock, 0, s>>>(states, bodies, n);
    return cudaGetLastError();
}

}  // namespace sfh
