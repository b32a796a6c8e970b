// FP64 step kernel of the GB300 DEM engine: particle-particle contacts from
// the Verlet list, particle-wall contacts from the wall list,
// tangential-history bookkeeping, symplectic Euler, the list-refresh test and
// out-of-bounds marking, in one pass.
//
// It computes one call of device_dem_verlet_verlet (device_dem.cu:1195-1236)
// with the arithmetic of the reference CPU path (cpu_dem.cu):
// particle_collision_verlet :1084, calc_normal_force :953,
// calc_tangential_force :783, update_history :587, wall_collision_verlet :238,
// calc_normal_force_wall :536, calc_tangential_force_wall :636,
// update_history_wall :611, the update loop :1622-1652,
// shouldRefreshNeighborList :1529 and checkOoB :1575.  Compiled with
// -fmad=false: no multiply-add is contracted, so the linear law reproduces the
// reference CPU build (-ffp-contract=off) bit for bit.  A particle's force and
// torque are sums in list order, without atomics, whatever lane computed each
// term, so they do not depend on how the work is spread.
//
// What bounds it is the FP64 pipe: an SM of this chip retires two FP64
// operations per cycle, so a warp instruction holds the pipe for 16 cycles
// however few of its lanes are active.  With one thread per particle (the
// form before) 4.8 of 32 lanes were active per FP64 instruction, since a
// warp's particles reach their contacts at different entries of their rows.
// Here a warp takes a tile of 8, 16 or 32 particles:
//  * the rows are tested in FP32 (coordinates truncated from the FP64 ones by
//    integer operations, so the test costs the FP64 pipe nothing), four lanes
//    to a particle; entries that touch or may touch go, compacted, into a ring;
//  * 32 of the ring at a time, one per lane, take the exact FP64 test and the
//    contact law; each particle's lane then adds its own results in row order;
//  * wall candidates likewise, 32 at a time over the tile's rows.
// One step kernel on dense beds (3 to 5 contacts a sphere), one thread per
// particle and now: 100 spheres (linear law) 100 and 27 us, 3,000
// (Hertz-Mindlin) 686 and 41 us, 40,000 (linear) 1164 and 141 us, 300,000
// (Hertz-Mindlin) 5444 and 813 us with the pipe 83 % busy at 22 active lanes.
#include "gdem_step.cuh"

namespace gdem {

namespace {

// x truncated to FP32 by integer operations (a conversion would go through
// the FP64 pipe): the sign, the exponent rebased and the 23 leading fraction
// bits; magnitudes below FP32's normal range give 0.  Within one FP32 ulp of x.
__device__ __forceinline__ float truncf64(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned m = (__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu;
    return (hi & 0x7ff00000u) < (897u << 20) ? 0.f : __uint_as_float(m | (hi & 0x80000000u));
}

// May particles at a and b (FP32 within an ulp) touch?  `delta` bounds what the
// rounding of the coordinates can move the distance; the factor covers the
// test's own rounding.
__device__ __forceinline__ bool may_touch(const View<FP64>& v, float4 a, float4 b) {
    const float dx = image_dxf(v, a.x - b.x), dy = a.y - b.y, dz = a.z - b.z;
    const float R = a.w + b.w + v.nb_delta;
    return !(dx * dx + dy * dy + dz * dz > R * R * 1.0000019f);
}

// A warp's shared memory: the ring of candidates that may touch (a batch of 32
// is drained whenever 32 are there, and one pass over the rows adds 4 x 32 at
// most), and the results of the batch being drained.
constexpr int kRing64 = 192;
struct Warp64 {
    double r[12][32];     // normal force, tangential force, torque, rolling torque
    int j[kRing64];       // partner's storage index
    int ow[kRing64];      // owning particle within the tile
    int fl[32];           // what the batch position holds (kNone...), slot above
    unsigned owned[32];   // batch positions of each particle
    int nc0[32], nc[32];  // history length at the start of the step, now
};
enum { kNone = 0, kNormalOnly = 1, kFull = 2, kRolling = 3 };

// Everything of one contact's law after its geometry: n the unit normal, lap
// the overlap, vr the relative velocity, a the surface-velocity lever
// (r_i w_i [+ r_j w_j]), Rs the effective radius, ms the effective mass.
// Normal force into fn; the tangential part follows once the history slot is
// known.
struct Law64 {
    double nx, ny, nz, vtx, vty, vtz, fnx, fny, fnz, kt, gt;
};

// tangential spring, its torque and rolling resistance into the results
template <int MODEL>
__device__ __forceinline__ int finish64(const View<FP64>& v, const Law64& c, double mu, double ri, double Rroll,
                                        double rx, double ry, double rz, double* hx, double* hy, double* hz, size_t h,
                                        bool fresh, Warp64& S, int lane) {
    Vec3<double> sp, cp, ft;
    cp.x = cp.y = cp.z = 0.;
    if (fresh) {
        sp.x = sp.y = sp.z = 0.;
    } else {
        sp.x = hx[h];
        sp.y = hy[h];
        sp.z = hz[h];
    }
    const double fnsq = c.fnx * c.fnx + c.fny * c.fny + c.fnz * c.fnz;
    tangential<FP64>(c.nx, c.ny, c.nz, fnsq, c.vtx, c.vty, c.vtz, c.gt, c.kt, mu, v.dt, sp, cp, ft);
    hx[h] = sp.x;
    hy[h] = sp.y;
    hz[h] = sp.z;
    const double cx = c.ny * ft.z - c.nz * ft.y;
    const double cy = c.nz * ft.x - c.nx * ft.z;
    const double cz = c.nx * ft.y - c.ny * ft.x;
    S.r[3][lane] = ft.x;
    S.r[4][lane] = ft.y;
    S.r[5][lane] = ft.z;
    S.r[6][lane] = ri * cx;
    S.r[7][lane] = ri * cy;
    S.r[8][lane] = ri * cz;
    if (MODEL == 1 && v.mat.mu_roll > 0.) {
        // rolling resistance, constant torque opposing the relative spin
        const double wn = sqrt(rx * rx + ry * ry + rz * rz);
        if (wn > 0.) {
            const double tr = -v.mat.mu_roll * Rroll * sqrt(fnsq) / wn;
            S.r[9][lane] = tr * rx;
            S.r[10][lane] = tr * ry;
            S.r[11][lane] = tr * rz;
            return kRolling;
        }
    }
    return kFull;
}

struct Sum64 {
    double fx, fy, fz, mx, my, mz;
};
// one batch result added as the reference adds it: the normal force, the
// tangential force, the torque, the rolling torque
__device__ __forceinline__ void add64(Sum64& F, const Warp64& S, int y, int kind) {
    F.fx += S.r[0][y];
    F.fy += S.r[1][y];
    F.fz += S.r[2][y];
    if (kind == kNormalOnly) return;
    F.fx += S.r[3][y];
    F.fy += S.r[4][y];
    F.fz += S.r[5][y];
    F.mx += S.r[6][y];
    F.my += S.r[7][y];
    F.mz += S.r[8][y];
    if (kind == kRolling) {
        F.mx += S.r[9][y];
        F.my += S.r[10][y];
        F.mz += S.r[11][y];
    }
}

// History slot of `key` in the row of particle i (calc_tangential_force,
// cpu_dem.cu:795-813), or -1 when it has none: four keys at a time, their
// loads in flight together.
__device__ __forceinline__ int search64(const int* hid, int n, int i, int nc, int key) {
    for (int q0 = 0; q0 < nc; q0 += 4) {
        int k[4];
#pragma unroll
        for (int q = 0; q < 4; q++) k[q] = q0 + q < nc ? hid[(size_t)(q0 + q) * n + i] : -1;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (k[q] == key) return q0 + q;
    }
    return -1;
}

// Slots of a batch's contacts: those without one (`found` < 0 on a lane that is
// `hit`) are appended to their particle's row in batch order, which is row
// order; -1 when the row is full.  `grp`: the lanes of the same particle.
__device__ __forceinline__ int slot64(Warp64& S, int lane, int ow, bool hit, int found, unsigned grp, int cap,
                                      bool& fresh) {
    fresh = hit && found < 0;
    const unsigned fm = __ballot_sync(0xffffffffu, fresh) & grp;
    int slot = found;
    if (fresh) {
        slot = S.nc[ow] + __popc(fm & ((1u << lane) - 1u));
        if (slot >= cap) slot = -1;
    }
    __syncwarp();
    if (hit && fm != 0u && lane == __ffs((int)fm) - 1) S.nc[ow] = min(S.nc[ow] + __popc(fm), cap);
    return slot;
}

// The oldest B (<= 32) candidates of the ring: exact test, contact law,
// history; results added to their particles' sums.
template <int MODEL>
__device__ __forceinline__ void drain64(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Warp64& S,
                                        int base, int head, int B, int lane, Sum64& F, unsigned long long& touched,
                                        unsigned& err) {
    const int n = v.n;
    const int x = (head + lane) % kRing64;
    const bool in = lane < B;
    const int ow = in ? S.ow[x] : 0;
    const int i = base + ow;
    int kind = kNone, found = -1, key = 0;
    bool hit = false;
    Law64 c = {};
    double ri = 0., Rstar = 0., mu = 0., rx = 0., ry = 0., rz = 0.;
    S.owned[lane] = 0u;
    if (in) {
        const int j = S.j[x];
        const double4_32a pi = A.pos[i], pj = A.pos[j];
        const double4_32a vi = A.vel[i], vj = A.vel[j];
        const double4_32a wi = A.rot[i], wj = A.rot[j];
        const double4_32a mi = P.mat[i];
        key = P.pid[j];
        const double dx = image_dx(v, pi.x - pj.x), dy = pi.y - pj.y, dz = pi.z - pj.z;
        const double distsq = dx * dx + dy * dy + dz * dz;
        ri = pi.w;
        const double rj = pj.w;
        const double Rs = ri + rj;
        hit = wj.w == 1. && distsq < Rs * Rs;
        if (hit) {
            found = search64(P.hid, n, i, S.nc0[ow], key);
            const double dist = sqrt(distsq);
            const double delMag = Rs - dist;
            c.nx = dx / dist;
            c.ny = dy / dist;
            c.nz = dz / dist;
            const double vrx = vi.x - vj.x, vry = vi.y - vj.y, vrz = vi.z - vj.z;
            const double vdn = vrx * c.nx + vry * c.ny + vrz * c.nz;
            const double vnx = vdn * c.nx, vny = vdn * c.ny, vnz = vdn * c.nz;
            // Hertz-Mindlin per-particle materials: both particles of a contact
            // belong to the same scene, so the particle's own values serve
            const bool pm = MODEL == 1 && v.per_particle_mat;
            mu = pm ? mi.x : v.mat.mu;
            const double invm = vi.w + vj.w;
            if (MODEL == 0) {
                // calc_normal_force (cpu_dem.cu:953-1011)
                const double ki = mi.x, etai = mi.y;
                const double delx = -delMag * c.nx, dely = -delMag * c.ny, delz = -delMag * c.nz;
                const double meff = 1. / invm;
                const double eta = etai * sqrt(meff);
                c.fnx = -ki * delx - eta * vnx;
                c.fny = -ki * dely - eta * vny;
                c.fnz = -ki * delz - eta * vnz;
                c.kt = ki;
                c.gt = eta;
            } else {
                // Hertz normal, Mindlin tangential stiffness
                const double damp_c = pm ? mi.y : v.mat.damp_c;
                Rstar = ri * rj / (ri + rj);
                const double mstar = 1. / invm;
                const double sqrtRd = sqrt(Rstar * delMag);
                const double fel = v.mat.kn_c * sqrtRd * delMag;
                const double gn = damp_c * sqrt(v.mat.sn_c * sqrtRd * mstar);
                const double fnm = fel - gn * vdn;
                c.fnx = fnm * c.nx;
                c.fny = fnm * c.ny;
                c.fnz = fnm * c.nz;
                c.kt = v.mat.kt_c * sqrtRd;
                c.gt = damp_c * sqrt(c.kt * mstar);
            }
            const double ax_ = ri * wi.x + rj * wj.x;
            const double ay_ = ri * wi.y + rj * wj.y;
            const double az_ = ri * wi.z + rj * wj.z;
            const double crx = ay_ * c.nz - az_ * c.ny;
            const double cry = az_ * c.nx - ax_ * c.nz;
            const double crz = ax_ * c.ny - ay_ * c.nx;
            c.vtx = (vrx - vnx) + crx;
            c.vty = (vry - vny) + cry;
            c.vtz = (vrz - vnz) + crz;
            rx = wi.x - wj.x;
            ry = wi.y - wj.y;
            rz = wi.z - wj.z;
            S.r[0][lane] = c.fnx;
            S.r[1][lane] = c.fny;
            S.r[2][lane] = c.fnz;
        }
    }
    const unsigned grp = __match_any_sync(0xffffffffu, hit ? ow : 32 + lane);
    bool fresh;
    const int slot = slot64(S, lane, ow, hit, found, grp, v.hist_cap, fresh);
    if (hit) {
        if (slot < 0) {
            err |= 0x4u;
            kind = kNormalOnly;
        } else {
            const size_t h = (size_t)slot * n + i;
            if (fresh) P.hid[h] = key;
            kind = finish64<MODEL>(v, c, mu, ri, Rstar, rx, ry, rz, P.hx, P.hy, P.hz, h, fresh, S, lane);
        }
        if ((grp & ((1u << lane) - 1u)) == 0u) S.owned[ow] = grp;
    }
    S.fl[lane] = kind | (slot << 2);
    __syncwarp();
    for (unsigned m = S.owned[lane]; m != 0u; m &= m - 1u) {
        const int y = __ffs((int)m) - 1;
        const int fl = S.fl[y];
        add64(F, S, y, fl & 3);
        if ((fl & 3) != kNormalOnly) touched |= 1ull << (fl >> 2);
    }
    __syncwarp();
}

// The tile's wall contacts (wall_collision_verlet, cpu_dem.cu:238): its wall
// rows, one after another, 32 candidates at a time through the closest
// feature, one per lane; each particle's lane drops features it met before in
// its row; the candidates that remain take the force where they are, and each
// particle's lane adds its own in row order.
template <int MODEL>
__device__ __forceinline__ void walls64(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Warp64& S,
                                        int base, int lane, int nw, Sum64& F, unsigned long long& touched,
                                        unsigned& err) {
    const int n = v.n;
    int incl = nw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const int excl = incl - nw;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int vore[64];  // features met (wall rows hold at most 64)
    int nvore = 0;
    for (int c0 = 0; c0 < total; c0 += 32) {
        const int cand = c0 + lane;
        // the candidate's particle: the first lane whose running count passes it
        int ow = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1)
            if (__shfl_sync(0xffffffffu, incl, ow + step - 1) <= cand) ow += step;
        const int k = cand - __shfl_sync(0xffffffffu, excl, ow);
        const int i = base + ow;
        int t = 0, hitf = -3;
        Feature f;
        double rid = 0.;
        if (cand < total) {
            t = v.neiw[(size_t)k * n + i];
            const double4_32a pi = A.pos[i];
            rid = pi.w;
            f = closest_feature(image_x_near(v, pi.x, v.tri[t].v0[0]), pi.y, pi.z, rid * rid, v.tri[t]);
            if (f.dist < rid) hitf = f.hit;
        }
        S.fl[lane] = hitf;
        if (!__any_sync(0xffffffffu, hitf != -3)) continue;
        __syncwarp();
        // a vertex or edge shared by triangles acts once per step
        const int y0 = max(excl, c0) - c0, y1 = min(incl, c0 + 32) - c0;
        for (int y = y0; y < y1; y++) {
            const int fh = S.fl[y];
            if (fh == -3 || fh == -1) continue;
            bool dup = false;
            for (int q = 0; q < nvore; q++)
                if (vore[q] == fh) {
                    dup = true;
                    break;
                }
            if (dup) S.fl[y] = -3;
            else if (nvore < 64) vore[nvore++] = fh;
        }
        __syncwarp();
        const bool hit = S.fl[lane] != -3;
        int kind = kNone, found = -1;
        Law64 c = {};
        double mu = 0.;
        double4_32a wi = make_double4_32a(0., 0., 0., 0.);
        if (hit) {
            found = search64(P.hwid, n, i, S.nc0[ow], t);
            const double4_32a vi = A.vel[i], mi = P.mat[i];
            wi = A.rot[i];
            const double invmi = vi.w;
            const bool pm = MODEL == 1 && v.per_particle_mat;
            mu = pm ? mi.x : v.mat.mu;
            const double delmag = rid - f.dist;
            c.nx = f.nx;
            c.ny = f.ny;
            c.nz = f.nz;
            const double vdn = vi.x * c.nx + vi.y * c.ny + vi.z * c.nz;
            const double vnx = vdn * c.nx, vny = vdn * c.ny, vnz = vdn * c.nz;
            if (MODEL == 0) {
                // calc_normal_force_wall (cpu_dem.cu:536-585): static wall
                const double ki = mi.x, etai = mi.y, sqrtmi = mi.z;
                const double delx = -delmag * c.nx, dely = -delmag * c.ny, delz = -delmag * c.nz;
                const double eta = etai * sqrtmi;
                c.fnx = -ki * delx - eta * vnx;
                c.fny = -ki * dely - eta * vny;
                c.fnz = -ki * delz - eta * vnz;
                c.kt = ki;
                c.gt = eta;
            } else {
                const double damp_c = pm ? mi.y : v.mat.damp_c;
                const double mstar = 1. / invmi;
                const double sqrtRd = sqrt(rid * delmag);
                const double fel = v.mat.kn_c * sqrtRd * delmag;
                const double gn = damp_c * sqrt(v.mat.sn_c * sqrtRd * mstar);
                const double fnm = fel - gn * vdn;
                c.fnx = fnm * c.nx;
                c.fny = fnm * c.ny;
                c.fnz = fnm * c.nz;
                c.kt = v.mat.kt_c * sqrtRd;
                c.gt = damp_c * sqrt(c.kt * mstar);
            }
            const double ax_ = rid * wi.x, ay_ = rid * wi.y, az_ = rid * wi.z;
            const double crx = ay_ * c.nz - az_ * c.ny;
            const double cry = az_ * c.nx - ax_ * c.nz;
            const double crz = ax_ * c.ny - ay_ * c.nx;
            c.vtx = (vi.x - vnx) + crx;
            c.vty = (vi.y - vny) + cry;
            c.vtz = (vi.z - vnz) + crz;
            S.r[0][lane] = c.fnx;
            S.r[1][lane] = c.fny;
            S.r[2][lane] = c.fnz;
        }
        const unsigned grp = __match_any_sync(0xffffffffu, hit ? ow : 32 + lane);
        bool fresh;
        const int slot = slot64(S, lane, ow, hit, found, grp, v.histw_cap, fresh);
        if (hit) {
            if (slot < 0) {
                err |= 0x8u;
                kind = kNormalOnly;
            } else {
                const size_t h = (size_t)slot * n + i;
                if (fresh) P.hwid[h] = t;
                kind = finish64<MODEL>(v, c, mu, rid, rid, wi.x, wi.y, wi.z, P.hwx, P.hwy, P.hwz, h, fresh, S, lane);
            }
        }
        S.fl[lane] = kind | (slot << 2);
        __syncwarp();
        for (int y = y0; y < y1; y++) {
            const int fl = S.fl[y];
            if ((fl & 3) == kNone) continue;
            add64(F, S, y, fl & 3);
            if ((fl & 3) != kNormalOnly) touched |= 1ull << (fl >> 2);
        }
        __syncwarp();
    }
}

// One step of the 8 G particles from `base` on, by one warp.
template <int MODEL, int G>
__device__ __forceinline__ void tile64(const View<FP64>& v, const SBank<FP64>& A, const SBank<FP64>& B,
                                       const PBank<FP64>& P, int base, Warp64& S, int lane, bool& refresh,
                                       unsigned& err) {
    const int n = v.n;
    const int i = base + lane;  // the particle this lane sums and integrates
    const bool mine = lane < 8 * G && i < n;
    bool active = false;
    int nw = 0;
    if (mine) {
        active = A.rot[i].w == 1.;
        S.nc0[lane] = S.nc[lane] = P.nc[i];
        nw = active ? v.nneiw[i] : 0;
    }
    __syncwarp();
    // ---- rows: four lanes to a particle, 8 particles to a group
    float4 own[G];
    int nn[G], most = 0;
#pragma unroll
    for (int g = 0; g < G; g++) {
        const int ig = base + 8 * g + (lane >> 2);
        nn[g] = 0;
        if (ig < n) {
            const double4_32a p = A.pos[ig];
            own[g] = make_float4(truncf64(p.x), truncf64(p.y), truncf64(p.z), truncf64(p.w));
            if (A.rot[ig].w == 1.) nn[g] = v.nnei[ig];
        }
        most = max(most, nn[g]);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    Sum64 F = {0., 0., 0., 0., 0., 0.};
    unsigned long long touched = 0ull;
    int head = 0, tail = 0;
    for (int k0 = 0; k0 < most; k0 += 4) {
        const int k = k0 + (lane & 3);
        int jj[G];
#pragma unroll
        for (int g = 0; g < G; g++)
            jj[g] = k < nn[g] ? v.nei[(size_t)k * n + base + 8 * g + (lane >> 2)] : -1;
        double4_32a pj[G];
#pragma unroll
        for (int g = 0; g < G; g++)
            if (jj[g] >= 0) pj[g] = A.pos[jj[g]];
#pragma unroll
        for (int g = 0; g < G; g++) {
            const bool near = jj[g] >= 0 && may_touch(v, own[g],
                                                      make_float4(truncf64(pj[g].x), truncf64(pj[g].y),
                                                                  truncf64(pj[g].z), truncf64(pj[g].w)));
            const unsigned m = __ballot_sync(0xffffffffu, near);
            if (near) {
                const int x = (tail + __popc(m & ((1u << lane) - 1u))) % kRing64;
                S.j[x] = jj[g];
                S.ow[x] = 8 * g + (lane >> 2);
            }
            tail += __popc(m);
        }
        __syncwarp();
        const bool last = k0 + 4 >= most;
        while (tail - head >= 32 || (last && tail > head)) {
            const int cnt = min(32, tail - head);
            drain64<MODEL>(v, A, P, S, base, head, cnt, lane, F, touched, err);
            head += cnt;
        }
    }
    int ncw = 0;
    if (mine) {
        if (active) P.nc[i] = surviving(touched, S.nc[lane]);
        ncw = P.ncw[i];
    }
    // ---- walls
    if (__any_sync(0xffffffffu, nw > 0)) {
        S.nc0[lane] = S.nc[lane] = ncw;
        __syncwarp();
        touched = 0ull;
        walls64<MODEL>(v, A, P, S, base, lane, nw, F, touched, err);
        if (active) P.ncw[i] = surviving(touched, S.nc[lane]);
    } else if (active && ncw > 0) {
        P.ncw[i] = 0;
    }
    __syncwarp();
    if (!mine) return;
    const double4_32a pi = A.pos[i], vi = A.vel[i];
    double4_32a wi = A.rot[i];
    if (!active) {
        // inactive, or left the box last step (status 2): frozen from now on
        B.pos[i] = pi;
        B.vel[i] = vi;
        wi.w = 0.;
        B.rot[i] = wi;
        if (v.store_forces) {
            v.fx[i] = 0.; v.fy[i] = 0.; v.fz[i] = 0.;
            v.tx[i] = 0.; v.ty[i] = 0.; v.tz[i] = 0.;
        }
        return;
    }
    // ---------------- symplectic Euler (cpu_dem.cu:1622-1652)
    const double invmi = vi.w, invmoi = P.mat[i].w, dt = v.dt;
    const double ax = F.fx * invmi + v.gx;
    const double ay = F.fy * invmi + v.gy;
    const double az = F.fz * invmi + v.gz;
    const double nvx = vi.x + ax * dt, nvy = vi.y + ay * dt, nvz = vi.z + az * dt;
    double nxp = pi.x + nvx * dt;
    const double nyp = pi.y + nvy * dt;
    const double nzp = pi.z + nvz * dt;
    // periodic x: back into the period (a step moves far less than one)
    if (v.per_x) {
        if (nxp >= v.maxx) nxp -= v.Lx;
        else if (nxp < v.minx) nxp += v.Lx;
    }
    const double aax = F.mx * invmoi, aay = F.my * invmoi, aaz = F.mz * invmoi;
    const double nwx = wi.x + aax * dt, nwy = wi.y + aay * dt, nwz = wi.z + aaz * dt;
    // ---------------- refresh test (shouldRefreshNeighborList, cpu_dem.cu:1529):
    // every particle active at the start of the step takes part
    {
        const double4_32a rf = v.ref[i];
        const double ex = image_dx(v, nxp - rf.x), ey = nyp - rf.y, ez = nzp - rf.z;
        const double d2 = ex * ex + ey * ey + ez * ez;
        if (d2 > v.thresh_sq) refresh = true;
    }
    // ---------------- out of bounds (checkOoB, cpu_dem.cu:1575).  The
    // reference CPU loop deactivates after the list rebuild of this
    // step (main.cu:312-316), so a particle leaving the box is marked 2:
    // still in this step's rebuild, inactive from the next step on.
    double status = 1.;
    if ((!v.per_x && (nxp < v.minx || nxp > v.maxx)) || nyp < v.miny || nyp > v.maxy || nzp < v.minz || nzp > v.maxz)
        status = 2.;
    if (!(nxp == nxp && nyp == nyp && nzp == nzp)) {
        err |= 0x20u;
        status = 2.;
    }
    B.pos[i] = make_double4_32a(nxp, nyp, nzp, pi.w);
    B.vel[i] = make_double4_32a(nvx, nvy, nvz, invmi);
    B.rot[i] = make_double4_32a(nwx, nwy, nwz, status);
    if (v.store_forces) {
        v.fx[i] = F.fx; v.fy[i] = F.fy; v.fz[i] = F.fz;
        v.tx[i] = F.mx; v.ty[i] = F.my; v.tz[i] = F.mz;
    }
}

// One warp per CTA: the hardware hands tiles to SMs as they come free, and few
// tiles spread over as many SMs (FP64 pipes) as there are.
template <int MODEL, int G>
__global__ void __launch_bounds__(32) k_step64(View<FP64> v, cudaGraphConditionalHandle cond,
                                               cudaGraphConditionalHandle /*inner rows: mixed mode only*/,
                                               int use_cond) {
    __shared__ Warp64 S;
    Ctl* ctl = v.ctl;
    if (chain_passes(ctl, use_cond, 0, cond)) return;
    const int s = ctl->s, p = ctl->p;
    bool refresh = false;
    unsigned err = 0u;
    tile64<MODEL, G>(v, v.S[s], v.S[s ^ 1], v.P[p], (int)blockIdx.x * 8 * G, S, threadIdx.x, refresh, err);
    if (__any_sync(0xffffffffu, refresh) && threadIdx.x == 0) atomicOr(&ctl->refresh, 1u);
    if (err) atomicOr(&ctl->error, err);
    if (last_block(&ctl->done[0])) {
        if (threadIdx.x == 0) {
            ctl->done[0] = 0;
            step_close(ctl, s, use_cond, 0, cond, cond);
        }
    }
}

}  // namespace

StepLaunch step_launch(const View<FP64>& v, int) {
    const bool hm = v.mat.model == 1;
    // Tile width: a tile's batches of 32 run one after another, so few
    // particles take narrow tiles (more warps, on more SMs), many take wide
    // ones (fuller batches: 51 % of the lanes at 8 particles, 81 % at 32).
    // Step of a Hertz-Mindlin bed at 8 / 16 / 32 to a tile: 3,000 spheres
    // 49 / 61 / 92 us, 10,000 65 / 64 / 84, 20,000 120 / 90 / 94, 30,000
    // 140 / 127 / 110.
    const int tiles8 = (v.n + 7) / 8;
    const int g = tiles8 <= 8 * sm_count() ? 1 : (tiles8 <= 18 * sm_count() ? 2 : 4);
    void* fn = g == 1   ? (hm ? (void*)k_step64<1, 1> : (void*)k_step64<0, 1>)
               : g == 2 ? (hm ? (void*)k_step64<1, 2> : (void*)k_step64<0, 2>)
                        : (hm ? (void*)k_step64<1, 4> : (void*)k_step64<0, 4>);
    return StepLaunch{fn, dim3((v.n + 8 * g - 1) / (8 * g)), dim3(32), 0};
}

void launch_step(const View<FP64>& v, cudaStream_t st, cudaGraphConditionalHandle cond, int use_cond) {
    const StepLaunch L = step_launch(v);
    View<FP64> vv = v;
    cudaGraphConditionalHandle ci = cond;
    void* args[4] = {(void*)&vv, (void*)&cond, (void*)&ci, (void*)&use_cond};
    cudaLaunchKernel(L.fn, L.grid, L.block, args, L.smem, st);
}

}  // namespace gdem
