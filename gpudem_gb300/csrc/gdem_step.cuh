// What the step kernels of both precisions share: the tangential spring law
// and the history search.  The kernels themselves are in gdem_step_fp64.cu and
// gdem_step_mixed.cu.
#pragma once

#include "gdem_internal.cuh"

namespace gdem {

// SMs of the current device (asked every time: an engine of another device of the
// process has its own).
inline int sm_count() {
    int dev = 0, cnt = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cnt, cudaDevAttrMultiProcessorCount, dev);
    return cnt > 0 ? cnt : 1;
}

// A chained step kernel's first question: does it pass?  Several steps run one
// after another in a graph without asking the rebuild conditions in between
// (10 us a step); when a step asks for new rows, those behind it in the chain
// pass, the rows are rebuilt, and the loop around the chain goes on with the
// steps that remain.  `hold` is written by the last CTA of an earlier kernel
// only, so every CTA of a kernel sees the same answer.
__device__ __forceinline__ bool chain_passes(Ctl* ctl, int use_cond, cudaGraphConditionalHandle half) {
    if (!(use_cond & kChained) || ctl->hold == 0u) return false;
    if ((use_cond & kChainMid) && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(half, 0u);
    return true;
}

// End of a step, by one thread of its last CTA: the bank flip, the step count,
// and the graph's conditions.
__device__ __forceinline__ void step_close(Ctl* ctl, int s, int use_cond, int inner, cudaGraphConditionalHandle cond,
                                           cudaGraphConditionalHandle cond2) {
    const unsigned long long steps = ctl->steps + 1ull;
    ctl->s = s ^ 1;
    ctl->steps = steps;
    if (!use_cond) return;
    const unsigned r = atomicAdd(&ctl->refresh, 0u), ri = inner ? atomicAdd(&ctl->irefresh, 0u) : 0u;
    if (use_cond & kCondLists) cudaGraphSetConditional(cond, r ? 1u : 0u);
    if (use_cond & kCondInner) cudaGraphSetConditional(cond2, ri ? 1u : 0u);
    if (use_cond & (kChained | kOften)) {
        const bool asked = (r | ri) != 0u;
        const int left = ctl->remaining - 1;
        ctl->remaining = left;
        if (use_cond & kChained) ctl->hold = asked || left <= 0 ? 1u : 0u;
        if (use_cond & kChainMid) cudaGraphSetConditional(cond2, asked || left <= 0 ? 0u : 1u);
        if (use_cond & kOften) {
            if (asked) ctl->asked_at = steps;
            const bool often = asked || steps - ctl->asked_at < (unsigned long long)ctl->span;
            cudaGraphSetConditional(cond2, often && left > 0 ? 1u : 0u);
        }
    }
}

template <typename R>
struct Vec3 {
    R x, y, z;
};

template <typename R>
__device__ __forceinline__ R sqrt_(R a);
template <>
__device__ __forceinline__ double sqrt_<double>(double a) { return sqrt(a); }
template <>
__device__ __forceinline__ float sqrt_<float>(float a) { return sqrtf(a); }

// Tangential spring update + Coulomb cap (calc_tangential_force,
// cpu_dem.cu:824-891; the wall twin :677-772).  s holds the previous spring on
// entry, the new one on exit; c is its compensation term (mixed mode); ft is
// the force to add.  kt and gt are the tangential stiffness and damping (the
// linear law uses k_i and the normal damping for both).
template <class T>
__device__ __forceinline__ void tangential(typename T::real nx, typename T::real ny, typename T::real nz,
                                           typename T::real fnsq, typename T::real vtx,
                                           typename T::real vty, typename T::real vtz,
                                           typename T::real gt, typename T::real kt,
                                           typename T::real mu, typename T::real dt,
                                           Vec3<typename T::real>& s, Vec3<typename T::real>& c,
                                           Vec3<typename T::real>& ft) {
    using R = typename T::real;
    R dx, dy, dz;
    if (T::mixed) {
        // compensated accumulation of vt*dt
        const R yx = vtx * dt - c.x, yy = vty * dt - c.y, yz = vtz * dt - c.z;
        const R tx = s.x + yx, ty = s.y + yy, tz = s.z + yz;
        c.x = (tx - s.x) - yx;
        c.y = (ty - s.y) - yy;
        c.z = (tz - s.z) - yz;
        dx = tx;
        dy = ty;
        dz = tz;
        const R cdn = c.x * nx + c.y * ny + c.z * nz;
        c.x = c.x - cdn * nx;
        c.y = c.y - cdn * ny;
        c.z = c.z - cdn * nz;
    } else {
        dx = s.x + vtx * dt;
        dy = s.y + vty * dt;
        dz = s.z + vtz * dt;
    }
    const R ddn = dx * nx + dy * ny + dz * nz;
    dx = dx - ddn * nx;
    dy = dy - ddn * ny;
    dz = dz - ddn * nz;
    R tx = -kt * dx, ty = -kt * dy, tz = -kt * dz;
    const R ftsq = tx * tx + ty * ty + tz * tz;
    if (ftsq > (mu * mu) * fnsq) {
        if (ftsq != R(0.)) {
            const R inv = R(1.) / (sqrt_<R>(ftsq) + R(1e-15));
            const R ux = inv * tx, uy = inv * ty, uz = inv * tz;
            const R fnn = sqrt_<R>(fnsq);
            const R sc = mu * fnn;
            tx = sc * ux;
            ty = sc * uy;
            tz = sc * uz;
            const R ik = R(-1.) / kt;
            dx = ik * tx;
            dy = ik * ty;
            dz = ik * tz;
            c.x = R(0.);
            c.y = R(0.);
            c.z = R(0.);
        } else {
            tx = R(0.);
            ty = R(0.);
            tz = R(0.);
        }
    } else {
        tx -= gt * vtx;
        ty -= gt * vty;
        tz -= gt * vtz;
    }
    s.x = dx;
    s.y = dy;
    s.z = dz;
    ft.x = tx;
    ft.y = ty;
    ft.z = tz;
}

// History slot of `key` in row i (linear search, calc_tangential_force
// cpu_dem.cu:795-813), appended when absent; -1 when the row is full.
template <class T>
__device__ __forceinline__ int find_slot(const int* hid, int n, int i, int& nc, int key, int cap,
                                         bool& fresh) {
    for (int q = 0; q < nc; q++)
        if (hid[(size_t)q * n + i] == key) {
            fresh = false;
            return q;
        }
    fresh = true;
    if (nc >= cap) return -1;
    return nc++;
}

}  // namespace gdem
