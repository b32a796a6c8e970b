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
// operations per cycle, half a one in each of its four partitions, so a warp
// instruction holds its partition's pipe for 64 cycles however few of its lanes
// are active.  With one thread per particle (the first form) 4.8 of 32 lanes
// were active, since a warp's particles reach their contacts at different
// entries of their rows.  Here a CTA of four warps, one to a partition, takes a
// tile of up to 64 particles:
//  * the rows are tested in FP32 (coordinates truncated from the FP64 ones by
//    integer operations, so the test costs the FP64 pipe nothing), four to 32
//    lanes to a particle; what touches or may touch goes into a list, particle
//    by particle in row order;
//  * the list takes the exact FP64 test and the search for the history slots,
//    an entry per thread, and the wall rows their closest features;
//  * the contact laws run 32 entries at a time, handed to whichever warp is
//    free; then a thread to every component of a particle's force and torque
//    adds its results in row order and integrates it.
// Large scenes take a warp to a tile instead (below).  A step of a dense bed (3
// to 5 contacts a sphere), one thread per particle and now: 100 spheres (linear
// law) 84 and 18 us, 3,000 (Hertz-Mindlin) 668 and 30, 40,000 (linear) 1171 and
// 140, 300,000 (Hertz-Mindlin) 5511 and 830.
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
__device__ __forceinline__ float4 truncf64(double4_32a p) {
    return make_float4(truncf64(p.x), truncf64(p.y), truncf64(p.z), truncf64(p.w));
}

// ---------------------------------------------------------------- one CTA to a tile
constexpr int kTile64 = 64;    // particles of a tile at most
constexpr int kPairs64 = 448;  // entries of a tile's pair list: 7 a particle
constexpr int kWalls64 = 160;  // wall candidates of a tile
constexpr int kThreads64 = 128;
constexpr int kRes64 = kPairs64 + kWalls64;
// A tile with more of either is taken in halves, and so on.
static_assert(kPairs64 >= 128 && kWalls64 >= 64, "one particle must fit");

// what an entry turned out to be
enum { kNone = 0, kNormalOnly = 1, kFull = 2, kRolling = 3 };
// slot of an entry after the search: its slot, or
constexpr int kFresh = -1, kNoHit = -2;

struct __align__(16) Cta64 {
    double out[9][kTile64];             // new position, velocity, spin
    int ej[kPairs64];                   // partner's storage index
    short es[kPairs64];                 // slot, kFresh or kNoHit
    unsigned char eo[kPairs64];         // particle within the tile
    int wt[kWalls64], whit[kWalls64];  // triangle; feature touched, -3: none
    short ws[kWalls64];
    unsigned char wo[kWalls64];
    short fl[kRes64];                   // kind | slot << 2
    int cnt[kTile64], start[kTile64 + 1];  // list entries of each particle
    int nw[kTile64], wstart[kTile64 + 1];  // wall candidates
    int nc0[kTile64], ncw0[kTile64];       // history lengths at the start of the step
    int on[kTile64];                        // active
    int item;                            // next batch to be computed
};
// results: normal force, tangential force, torque (and rolling torque) of every
// entry, after the Cta64; a wall candidate's normal and distance until then
template <int MODEL>
constexpr size_t smem64(bool rolling) {
    return sizeof(double) * (MODEL == 1 && rolling ? 12 : 9) * kRes64 + sizeof(Cta64);
}

// One contact's law after its geometry.
struct Law64 {
    double nx, ny, nz, vtx, vty, vtz, fnx, fny, fnz, kt, gt;
    double mu, Rstar;  // friction; effective radius of the rolling resistance
};

// Particles at pi and pj in contact (dx, dy, dz: their separation).
template <int MODEL>
__device__ __forceinline__ Law64 pair_law64(const View<FP64>& v, double dx, double dy, double dz, double distsq,
                                            double4_32a pi, double4_32a pj, double4_32a vi, double4_32a vj,
                                            double4_32a wi, double4_32a wj, double4_32a mi) {
    Law64 c;
    c.Rstar = 0.;
    const double ri = pi.w, rj = pj.w;
    const double Rs = ri + rj;
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
    c.mu = pm ? mi.x : v.mat.mu;
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
        c.Rstar = ri * rj / (ri + rj);
        const double mstar = 1. / invm;
        const double sqrtRd = sqrt(c.Rstar * delMag);
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
    return c;
}

// A particle (mass 1 / invmi, radius rid) in contact with a wall whose feature
// lies at distance dist along the normal n.
template <int MODEL>
__device__ __forceinline__ Law64 wall_law64(const View<FP64>& v, double nx, double ny, double nz, double dist,
                                            double rid, double4_32a vi, double4_32a wi, double4_32a mi) {
    Law64 c;
    c.Rstar = rid;
    c.nx = nx;
    c.ny = ny;
    c.nz = nz;
    const double delmag = rid - dist;
    const bool pm = MODEL == 1 && v.per_particle_mat;
    c.mu = pm ? mi.x : v.mat.mu;
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
        const double mstar = 1. / vi.w;
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
    return c;
}

// Results are kept component by component, RES entries to each.  The normal
// force of entry e, and the rest once its history slot is known: the tangential
// spring, its torque and the rolling resistance (rx, ry, rz: relative spin).
template <int RES>
__device__ __forceinline__ void normal64(const Law64& c, double* r, int e) {
    r[e] = c.fnx;
    r[RES + e] = c.fny;
    r[2 * RES + e] = c.fnz;
}
template <int RES, int MODEL>
__device__ __forceinline__ int finish64(const View<FP64>& v, const Law64& c, double ri, double rx, double ry,
                                        double rz, double* hx, double* hy, double* hz, size_t h, bool fresh, double* r,
                                        int e) {
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
    tangential<FP64>(c.nx, c.ny, c.nz, fnsq, c.vtx, c.vty, c.vtz, c.gt, c.kt, c.mu, v.dt, sp, cp, ft);
    hx[h] = sp.x;
    hy[h] = sp.y;
    hz[h] = sp.z;
    const double cx = c.ny * ft.z - c.nz * ft.y;
    const double cy = c.nz * ft.x - c.nx * ft.z;
    const double cz = c.nx * ft.y - c.ny * ft.x;
    r[3 * RES + e] = ft.x;
    r[4 * RES + e] = ft.y;
    r[5 * RES + e] = ft.z;
    r[6 * RES + e] = ri * cx;
    r[7 * RES + e] = ri * cy;
    r[8 * RES + e] = ri * cz;
    if (MODEL == 1 && v.mat.mu_roll > 0.) {
        // rolling resistance, constant torque opposing the relative spin
        const double wn = sqrt(rx * rx + ry * ry + rz * rz);
        if (wn > 0.) {
            const double tr = -v.mat.mu_roll * c.Rstar * sqrt(fnsq) / wn;
            r[9 * RES + e] = tr * rx;
            r[10 * RES + e] = tr * ry;
            r[11 * RES + e] = tr * rz;
            return kRolling;
        }
    }
    return kFull;
}

// Sum over a particle's entries [e0, e1) of one component, c = 0..2 of the
// force, 3..5 of the torque, added as the reference adds it: a contact's normal
// force, then its tangential force; its torque, then its rolling torque.  The
// contact's slot joins `touched`, `fresh` counts the new ones.
__device__ __forceinline__ void sum64(double& sum, const double* r, const short* fl, const short* es, int off, int e0,
                                      int e1, int c, unsigned long long& touched, int& fresh) {
    const int first = c < 3 ? kNormalOnly : kFull;
    const double* x = r + (size_t)(c < 3 ? c : c + 3) * kRes64 + off;
    for (int e = e0; e < e1; e++) {
        const int f = fl[off + e], kind = f & 3;
        if (kind >= first) sum += x[e];
        if (kind > first) sum += x[3 * kRes64 + e];
        if (kind >= kFull) touched |= 1ull << (f >> 2);
        fresh += es[e] == kFresh ? 1 : 0;
    }
}

// History slot of `key` in the row of particle i (calc_tangential_force,
// cpu_dem.cu:795-813), kFresh when it has none: four keys at a time, their
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
    return kFresh;
}

// Slot of an entry: as found, or the next of its particle's row after the
// entries before it that are fresh too; -1 when the row is full.
__device__ __forceinline__ int slot64(const short* es, int first, int e, int nc0, int cap, bool& fresh) {
    int slot = es[e];
    fresh = slot == kFresh;
    if (fresh) {
        slot = nc0;
        for (int q = first; q < e; q++) slot += es[q] == kFresh ? 1 : 0;
        if (slot >= cap) slot = -1;
    }
    return slot;
}

// Contact law of the pair list's entry e.
template <int MODEL>
__device__ __forceinline__ void pair64(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Cta64& S,
                                       double* r, int base, int e, unsigned& err) {
    const int n = v.n;
    const int a = S.eo[e], i = base + a, j = S.ej[e];
    bool fresh;
    const int slot = slot64(S.es, S.start[a], e, S.nc0[a], v.hist_cap, fresh);
    const double4_32a pi = A.pos[i], pj = A.pos[j];
    const double4_32a vi = A.vel[i], vj = A.vel[j];
    const double4_32a wi = A.rot[i], wj = A.rot[j];
    const double4_32a mi = P.mat[i];
    const double dx = image_dx(v, pi.x - pj.x), dy = pi.y - pj.y, dz = pi.z - pj.z;
    const double distsq = dx * dx + dy * dy + dz * dz;
    const Law64 c = pair_law64<MODEL>(v, dx, dy, dz, distsq, pi, pj, vi, vj, wi, wj, mi);
    normal64<kRes64>(c, r, e);
    int kind = kNormalOnly;
    if (slot < 0) {
        err |= 0x4u;
    } else {
        const size_t h = (size_t)slot * n + i;
        if (fresh) P.hid[h] = P.pid[j];
        kind = finish64<kRes64, MODEL>(v, c, pi.w, wi.x - wj.x, wi.y - wj.y, wi.z - wj.z, P.hx, P.hy, P.hz, h,
                                        fresh, r, e);
    }
    S.fl[e] = (short)(kind | (slot << 2));
}

// Contact law of wall candidate w (its feature is in contact and new).
template <int MODEL>
__device__ __forceinline__ void wall64(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Cta64& S,
                                       double* r, int base, int w, unsigned& err) {
    const int n = v.n;
    const int a = S.wo[w], i = base + a, e = kPairs64 + w;
    bool fresh;
    const int slot = slot64(S.ws, S.wstart[a], w, S.ncw0[a], v.histw_cap, fresh);
    const double4_32a vi = A.vel[i], wi = A.rot[i], mi = P.mat[i];
    const double rid = A.pos[i].w;
    const Law64 c = wall_law64<MODEL>(v, r[e], r[kRes64 + e], r[2 * kRes64 + e], r[3 * kRes64 + e], rid, vi, wi, mi);
    normal64<kRes64>(c, r, e);
    int kind = kNormalOnly;
    if (slot < 0) {
        err |= 0x8u;
    } else {
        const size_t h = (size_t)slot * n + i;
        if (fresh) P.hwid[h] = S.wt[w];
        kind = finish64<kRes64, MODEL>(v, c, rid, wi.x, wi.y, wi.z, P.hwx, P.hwy, P.hwz, h, fresh, r, e);
    }
    S.fl[e] = (short)(kind | (slot << 2));
}

// The law of one contact by four lanes, a component to each of the first three
// (the fourth repeats x and stores nothing): eight contacts a warp.  The vector
// work, two thirds of a contact's FP64 instructions, is then one instruction for
// three, and the scalars are computed by all; for tiles whose contacts would fill
// a fraction of a warp anyway.  Operation by operation the same as pair_law64,
// wall_law64 and finish64.
constexpr int kSplit = 8;  // contacts a batch

struct Quad {
    int c, first;  // this lane's component; the group's first lane
    __device__ __forceinline__ double at(double x, int k) const { return __shfl_sync(0xffffffffu, x, first + k); }
    __device__ __forceinline__ double dot(double a, double b) const {
        const double p = a * b, p0 = at(p, 0), p1 = at(p, 1), p2 = at(p, 2);
        return p0 + p1 + p2;
    }
    __device__ __forceinline__ double cross(double a, double b) const {
        const int u = c == 2 ? 0 : c + 1, w = c == 0 ? 2 : c - 1;
        const double au = at(a, u), aw = at(a, w), bu = at(b, u), bw = at(b, w);
        return au * bw - aw * bu;
    }
};
__device__ __forceinline__ double comp64(const double4_32a* p, int i, int c) {
    return reinterpret_cast<const double*>(p + i)[c];
}

// From the unit normal's component n on: overlap lap, relative velocity vr,
// surface lever lev and relative spin rel (components), effective radius and mass
// (Hertz-Mindlin), damping eta (linear).  `live`: the group holds a contact.
template <int MODEL>
__device__ __forceinline__ void law64_split(const View<FP64>& v, const Quad& G, bool live, double n, double lap, double vr,
                                            double lev, double rel, double ri, double Rstar, double mstar, double eta,
                                            double4_32a mi, int e, int slot, bool fresh, double* hx, double* hy,
                                            double* hz, size_t h, Cta64& S, double* r) {
    const int c = G.c;
    const bool store = live && (threadIdx.x & 3) != 3;
    const double vdn = G.dot(vr, n);
    const double vn = vdn * n;
    const bool pm = MODEL == 1 && v.per_particle_mat;
    const double mu = pm ? mi.x : v.mat.mu;
    double fn, kt, gt;
    if (MODEL == 0) {
        const double ki = mi.x;
        const double del = -lap * n;
        fn = -ki * del - eta * vn;
        kt = ki;
        gt = eta;
    } else {
        const double damp_c = pm ? mi.y : v.mat.damp_c;
        const double sqrtRd = sqrt(Rstar * lap);
        const double fel = v.mat.kn_c * sqrtRd * lap;
        const double gn = damp_c * sqrt(v.mat.sn_c * sqrtRd * mstar);
        const double fnm = fel - gn * vdn;
        fn = fnm * n;
        kt = v.mat.kt_c * sqrtRd;
        gt = damp_c * sqrt(kt * mstar);
    }
    const double vt = (vr - vn) + G.cross(lev, n);
    const double fnsq = G.dot(fn, fn);
    double* const hc = c == 0 ? hx : (c == 1 ? hy : hz);
    double d = live && slot >= 0 && !fresh ? hc[h] : 0.;
    d = d + vt * v.dt;
    const double ddn = G.dot(d, n);
    d = d - ddn * n;
    double t = -kt * d;
    const double ftsq = G.dot(t, t);
    if (ftsq > (mu * mu) * fnsq) {
        if (ftsq != 0.) {
            const double inv = 1. / (sqrt(ftsq) + 1e-15);
            const double u = inv * t;
            const double sc = mu * sqrt(fnsq);
            t = sc * u;
            const double ik = -1. / kt;
            d = ik * t;
        } else {
            t = 0.;
        }
    } else {
        t -= gt * vt;
    }
    const double tq = ri * G.cross(n, t);
    int kind = slot < 0 ? kNormalOnly : kFull;
    if (store) {
        r[c * kRes64 + e] = fn;
        if (slot >= 0) {
            hc[h] = d;
            r[(3 + c) * kRes64 + e] = t;
            r[(6 + c) * kRes64 + e] = tq;
        }
    }
    if (MODEL == 1 && v.mat.mu_roll > 0.) {
        // rolling resistance, constant torque opposing the relative spin
        const double wn = sqrt(G.dot(rel, rel));
        if (wn > 0. && slot >= 0) {
            const double tr = -v.mat.mu_roll * Rstar * sqrt(fnsq) / wn;
            if (store) r[(9 + c) * kRes64 + e] = tr * rel;
            kind = kRolling;
        }
    }
    if (store && c == 0) S.fl[e] = (short)(kind | (slot << 2));
}

// Entries [e0, e0 + kSplit) of the pair list by a warp.
template <int MODEL>
__device__ __forceinline__ void pairs64_split(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Cta64& S,
                                              double* r, int base, int e0, int pairs, int lane, unsigned& err) {
    const int n = v.n, c4 = lane & 3;
    const Quad G = {c4 == 3 ? 0 : c4, lane & ~3};
    const int e = min(e0 + (lane >> 2), pairs - 1);
    const bool live = e0 + (lane >> 2) < pairs && S.es[e] != kNoHit;
    const int a = S.eo[e], i = base + a, j = S.ej[e];
    bool fresh;
    const int slot = slot64(S.es, S.start[a], e, S.nc0[a], v.hist_cap, fresh);
    const double ri = A.pos[i].w, rj = A.pos[j].w, invm = A.vel[i].w + A.vel[j].w;
    const double wi = comp64(A.rot, i, G.c), wj = comp64(A.rot, j, G.c);
    const double4_32a mi = P.mat[i];
    double d = comp64(A.pos, i, G.c) - comp64(A.pos, j, G.c);
    if (G.c == 0) d = image_dx(v, d);
    const double dist = sqrt(G.dot(d, d));
    const double Rs = ri + rj;
    const double Rstar = MODEL == 1 ? ri * rj / (ri + rj) : 0., mstar = 1. / invm;
    const double eta = MODEL == 0 ? mi.y * sqrt(mstar) : 0.;
    const size_t h = (size_t)(slot < 0 ? 0 : slot) * n + i;
    if (live && (lane & 3) == 0) {
        if (slot < 0) err |= 0x4u;
        else if (fresh) P.hid[h] = P.pid[j];
    }
    law64_split<MODEL>(v, G, live, d / dist, Rs - dist, comp64(A.vel, i, G.c) - comp64(A.vel, j, G.c), ri * wi + rj * wj,
                       wi - wj, ri, Rstar, mstar, eta, mi, e, slot, fresh, P.hx, P.hy, P.hz, h, S, r);
    if (!live && (lane & 3) == 0 && e0 + (lane >> 2) < pairs) S.fl[e] = kNone;
}

// Wall candidates [w0, w0 + kSplit) by a warp.
template <int MODEL>
__device__ __forceinline__ void walls64_split(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, Cta64& S,
                                              double* r, int base, int w0, int walls, int lane, unsigned& err) {
    const int n = v.n, c4 = lane & 3;
    const Quad G = {c4 == 3 ? 0 : c4, lane & ~3};
    const int w = min(w0 + (lane >> 2), walls - 1), e = kPairs64 + w;
    const bool in = w0 + (lane >> 2) < walls, live = in && S.ws[w] != kNoHit;
    if (!__any_sync(0xffffffffu, live)) {
        if (in && (lane & 3) == 0) S.fl[e] = kNone;
        return;
    }
    const int a = S.wo[w], i = base + a;
    bool fresh;
    const int slot = slot64(S.ws, S.wstart[a], w, S.ncw0[a], v.histw_cap, fresh);
    const double rid = A.pos[i].w, invmi = A.vel[i].w, wi = comp64(A.rot, i, G.c);
    const double4_32a mi = P.mat[i];
    const double nrm = live ? r[G.c * kRes64 + e] : 1., lap = live ? rid - r[3 * kRes64 + e] : rid;
    __syncwarp();
    const double mstar = MODEL == 1 ? 1. / invmi : 0., eta = MODEL == 0 ? mi.y * mi.z : 0.;
    const size_t h = (size_t)(slot < 0 ? 0 : slot) * n + i;
    if (live && (lane & 3) == 0) {
        if (slot < 0) err |= 0x8u;
        else if (fresh) P.hwid[h] = S.wt[w];
    }
    law64_split<MODEL>(v, G, live, nrm, lap, comp64(A.vel, i, G.c), rid * wi, wi, rid, rid, mstar, eta, mi, e, slot, fresh,
                       P.hwx, P.hwy, P.hwz, h, S, r);
    if (!live && in && (lane & 3) == 0) S.fl[e] = kNone;
}

// Exclusive scan of x[0..m) into out[0..kTile] by one warp (m <= kTile <= 64).
__device__ __forceinline__ void scan64(const int* x, int* out, int m, int lane) {
    const int a = lane < m ? x[lane] : 0, b = lane + 32 < m ? x[lane + 32] : 0;
    int ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ya = __shfl_up_sync(0xffffffffu, ia, o), yb = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) {
            ia += ya;
            ib += yb;
        }
    }
    const int half = __shfl_sync(0xffffffffu, ia, 31);
    if (lane < kTile64) out[lane] = ia - a;
    if (lane + 32 < kTile64) out[lane + 32] = half + ib - b;
    if (lane == 31) out[kTile64] = half + ib;
}
// Particle whose run [start[a], start[a + 1]) holds position c.
__device__ __forceinline__ int owner64(const int* start, int c) {
    int a = 0;
#pragma unroll
    for (int step = 32; step >= 1; step >>= 1)
        if (a + step < kTile64 && start[a + step] <= c) a += step;
    return a;
}

// Symplectic Euler (cpu_dem.cu:1622-1652) of one component of particle i with
// its sum: the new velocity and position (c < 3) or spin into `out`.
__device__ __forceinline__ void advance64(const View<FP64>& v, const SBank<FP64>& A, const PBank<FP64>& P, int i, int c,
                                          double sum, Cta64& S, int a) {
    const double dt = v.dt;
    if (c < 3) {
        const double* p = reinterpret_cast<const double*>(A.pos + i);
        const double* u = reinterpret_cast<const double*>(A.vel + i);
        const double acc = sum * u[3] + (c == 0 ? v.gx : (c == 1 ? v.gy : v.gz));
        const double nv = u[c] + acc * dt;
        double np = p[c] + nv * dt;
        // periodic x: back into the period (a step moves far less than one)
        if (c == 0 && v.per_x) {
            if (np >= v.maxx) np -= v.Lx;
            else if (np < v.minx) np += v.Lx;
        }
        S.out[c][a] = np;
        S.out[3 + c][a] = nv;
        if (v.store_forces) (c == 0 ? v.fx : (c == 1 ? v.fy : v.fz))[i] = sum;
    } else {
        const double* w = reinterpret_cast<const double*>(A.rot + i);
        const double acc = sum * P.mat[i].w;
        S.out[3 + c][a] = w[c - 3] + acc * dt;
        if (v.store_forces) (c == 3 ? v.tx : (c == 4 ? v.ty : v.tz))[i] = sum;
    }
}

// The end of particle i's step: the refresh and out-of-box tests and the new
// state.
__device__ __forceinline__ void close64(const View<FP64>& v, const SBank<FP64>& A, const SBank<FP64>& B, int i,
                                        double nxp, double nyp, double nzp, double nvx, double nvy, double nvz,
                                        double nwx, double nwy, double nwz, bool& refresh, unsigned& err) {
    const double4_32a rf = v.ref[i];
    const double ri = A.pos[i].w, invmi = A.vel[i].w;
    // ---------------- refresh test (shouldRefreshNeighborList, cpu_dem.cu:1529):
    // every particle active at the start of the step takes part
    {
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
    B.pos[i] = make_double4_32a(nxp, nyp, nzp, ri);
    B.vel[i] = make_double4_32a(nvx, nvy, nvz, invmi);
    B.rot[i] = make_double4_32a(nwx, nwy, nwz, status);
}
// A particle that is inactive, or left the box last step (status 2): frozen from
// now on.
__device__ __forceinline__ void freeze64(const View<FP64>& v, const SBank<FP64>& A, const SBank<FP64>& B, int i) {
    B.pos[i] = A.pos[i];
    B.vel[i] = A.vel[i];
    double4_32a wi = A.rot[i];
    wi.w = 0.;
    B.rot[i] = wi;
    if (v.store_forces) {
        v.fx[i] = 0.; v.fy[i] = 0.; v.fz[i] = 0.;
        v.tx[i] = 0.; v.ty[i] = 0.; v.tz[i] = 0.;
    }
}

// One step of the m (<= kTile) particles from `base` on; false when the lists
// are too short for them (nothing has been written then).
template <int MODEL, bool SPLIT>
__device__ __forceinline__ bool tile64(const View<FP64>& v, const SBank<FP64>& A, const SBank<FP64>& B,
                                       const PBank<FP64>& P, int base, int m, Cta64& S, double* r, bool& refresh,
                                       unsigned& err) {
    const int n = v.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < m) {
        const int i = base + tid;
        const bool active = A.rot[i].w == 1.;
        S.on[tid] = active ? 1 : 0;
        S.nw[tid] = active ? v.nneiw[i] : 0;
        S.nc0[tid] = P.nc[i];
        S.ncw0[tid] = P.ncw[i];
    }
    // ---- rows: L lanes to a particle, as many passes of the CTA as the tile
    // takes with four, U entries of a lane in flight together.  Bit t of found[g]:
    // entry L t + q of the particle of pass g may touch.
    constexpr int U = 4, NP = 2;
    int L = 4;
    while (2 * L * m <= kThreads64 && L < 32) L *= 2;
    const int per = kThreads64 / L;
    const int passes = m <= per ? 1 : 2;
    const int q = lane & (L - 1), a0 = tid / L;
    unsigned found[NP];
    int nn[NP], most = 0;
    float4 own[NP];
#pragma unroll
    for (int g = 0; g < NP; g++) {
        const int a = a0 + g * per;
        found[g] = 0u;
        nn[g] = 0;
        if (a < m) {
            const int i = base + a;
            own[g] = truncf64(A.pos[i]);
            if (A.rot[i].w == 1.) nn[g] = v.nnei[i];
        }
        most = max(most, nn[g]);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    const int turns = (most + L - 1) / L, stride = U / passes;
    for (int t0 = 0; t0 < turns; t0 += stride) {
        int jj[U];
        double4_32a pj[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            // entry u of the round: pass u mod passes, turn u / passes
            const int g = u & (passes - 1), k = (t0 + (passes == 1 ? u : u >> 1)) * L + q;
            const int cnt = passes == 2 ? nn[u & 1] : nn[0];
            jj[u] = k < cnt ? v.nei[(size_t)k * n + base + a0 + g * per] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (jj[u] >= 0) pj[u] = A.pos[jj[u]];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (jj[u] < 0) continue;
            const float4 o = passes == 2 ? own[u & 1] : own[0];
            const unsigned bit = 1u << (t0 + (passes == 1 ? u : u >> 1));
            if (!may_touch(v, o, truncf64(pj[u]))) continue;
            if (passes == 2) found[u & 1] |= bit;
            else found[0] |= bit;
        }
    }
#pragma unroll
    for (int g = 0; g < NP; g++) {
        int c = __popc(found[g]);
        for (int o = L >> 1; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        const int a = a0 + g * per;
        if (q == 0 && a < m) S.cnt[a] = c;
    }
    __syncthreads();
    if (warp == 0) scan64(S.cnt, S.start, m, lane);
    if (warp == 3) scan64(S.nw, S.wstart, m, lane);
    if (tid == 1) S.item = 0;
    __syncthreads();
    const int pairs = S.start[kTile64], walls = S.wstart[kTile64];
    if (pairs > kPairs64 || walls > kWalls64) {
        __syncthreads();
        return false;
    }
    // ---- the list: every particle's entries in row order
#pragma unroll
    for (int g = 0; g < NP; g++) {
        const unsigned f = found[g];
        const int a = a0 + g * per;
        int at = a < m ? S.start[a] : 0;
        for (int t = 0; t < turns; t++) {
            const unsigned b = __ballot_sync(0xffffffffu, (f >> t) & 1u);
            const unsigned mine = L == 32 ? b : (b >> (lane & ~(L - 1))) & ((1u << L) - 1u);
            if ((f >> t) & 1u) {
                const int e = at + __popc(mine & ((1u << q) - 1u));
                S.ej[e] = v.nei[(size_t)(t * L + q) * n + base + a];
                S.eo[e] = (unsigned char)a;
            }
            at += __popc(mine);
        }
    }
    __syncthreads();
    // ---- exact test and history slot of every entry
    for (int e = tid; e < pairs; e += kThreads64) {
        const int a = S.eo[e], i = base + a, j = S.ej[e];
        const double4_32a pi = A.pos[i], pj = A.pos[j];
        const double stj = A.rot[j].w;
        const int slot = search64(P.hid, n, i, S.nc0[a], P.pid[j]);
        const double dx = image_dx(v, pi.x - pj.x), dy = pi.y - pj.y, dz = pi.z - pj.z;
        const double distsq = dx * dx + dy * dy + dz * dz;
        const double Rs = pi.w + pj.w;
        S.es[e] = (short)(stj == 1. && distsq < Rs * Rs ? slot : kNoHit);
    }
    // ---- closest feature (wall_collision_verlet, cpu_dem.cu:238) and history
    // slot of every wall candidate, the last warps first
    bool touch = false;
    for (int w = (3 - warp) * 32 + lane; w < walls; w += kThreads64) {
        const int a = owner64(S.wstart, w), i = base + a;
        const int t = v.neiw[(size_t)(w - S.wstart[a]) * n + i];
        const double4_32a pi = A.pos[i];
        const double rid = pi.w;
        const Feature f = closest_feature(image_x_near(v, pi.x, v.tri[t].v0[0]), pi.y, pi.z, rid * rid, v.tri[t]);
        S.wo[w] = (unsigned char)a;
        S.wt[w] = t;
        int hit = -3, slot = kNoHit;
        if (f.dist < rid) {
            hit = f.hit;
            touch = true;
            slot = search64(P.hwid, n, i, S.ncw0[a], t);
            r[kPairs64 + w] = f.nx;
            r[1 * kRes64 + kPairs64 + w] = f.ny;
            r[2 * kRes64 + kPairs64 + w] = f.nz;
            r[3 * kRes64 + kPairs64 + w] = f.dist;
        }
        S.whit[w] = hit;
        S.ws[w] = (short)slot;
    }
    const bool any_wall = __syncthreads_or(touch);
    if (any_wall) {
        // a vertex or edge shared by triangles acts once per step: of a
        // particle's candidates that touch the same one, the first
        if (tid < m) {
            const int w0 = S.wstart[tid], w1 = S.wstart[tid + 1];
            for (int w = w0; w < w1; w++) {
                const int h = S.whit[w];
                if (h == -3 || h == -1) continue;
                for (int u = w0; u < w; u++)
                    if (S.whit[u] == h && S.ws[u] != kNoHit) {
                        S.ws[w] = kNoHit;
                        break;
                    }
            }
        }
        __syncthreads();
    }
    // ---- contact laws, a batch at a time: the walls', then the pairs'
    constexpr int per_batch = SPLIT ? kSplit : 32;
    const int wb = any_wall ? (walls + per_batch - 1) / per_batch : 0, items = wb + (pairs + per_batch - 1) / per_batch;
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(&S.item, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= items) break;
        if constexpr (SPLIT) {
            if (it < wb) walls64_split<MODEL>(v, A, P, S, r, base, it * kSplit, walls, lane, err);
            else pairs64_split<MODEL>(v, A, P, S, r, base, (it - wb) * kSplit, pairs, lane, err);
        } else if (it < wb) {
            const int w = it * 32 + lane;
            if (w < walls) {
                if (S.ws[w] != kNoHit) wall64<MODEL>(v, A, P, S, r, base, w, err);
                else S.fl[kPairs64 + w] = kNone;
            }
        } else {
            const int e = (it - wb) * 32 + lane;
            if (e < pairs) {
                if (S.es[e] != kNoHit) pair64<MODEL>(v, A, P, S, r, base, e, err);
                else S.fl[e] = kNone;
            }
        }
    }
    __syncthreads();
    // ---- sums in row order and their integration, a component to a thread (a
    // particle's nine sums in one thread are a chain of nine pipe slots a contact)
    for (int k = tid; k < 6 * m; k += kThreads64) {
        const int c = k / m, a = k - c * m, i = base + a;
        if (!S.on[a]) continue;
        double sum = 0.;
        unsigned long long touched = 0ull;
        int fresh = 0;
        sum64(sum, r, S.fl, S.es, 0, S.start[a], S.start[a + 1], c, touched, fresh);
        if (c == 5) P.nc[i] = surviving(touched, min(S.nc0[a] + fresh, v.hist_cap));
        touched = 0ull;
        fresh = 0;
        if (any_wall) sum64(sum, r, S.fl, S.ws, kPairs64, S.wstart[a], S.wstart[a + 1], c, touched, fresh);
        if (c == 5 && S.ncw0[a] + fresh > 0) P.ncw[i] = surviving(touched, min(S.ncw0[a] + fresh, v.histw_cap));
        advance64(v, A, P, i, c, sum, S, a);
    }
    __syncthreads();
    if (tid < m) {
        if (S.on[tid])
            close64(v, A, B, base + tid, S.out[0][tid], S.out[1][tid], S.out[2][tid], S.out[3][tid], S.out[4][tid],
                    S.out[5][tid], S.out[6][tid], S.out[7][tid], S.out[8][tid], refresh, err);
        else freeze64(v, A, B, base + tid);
    }
    return true;
}

template <int MODEL, bool SPLIT>
__global__ void __launch_bounds__(kThreads64, 3) k_step64(View<FP64> v, cudaGraphConditionalHandle cond,
                                                              cudaGraphConditionalHandle cond2,
                                                              int use_cond) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cta64& S = *reinterpret_cast<Cta64*>(smem_raw);
    double* r = reinterpret_cast<double*>(smem_raw + sizeof(Cta64));
    Ctl* ctl = v.ctl;
    if (chain_passes(ctl, use_cond, cond2)) return;
    const int s = ctl->s, p = ctl->p;
    bool refresh = false;
    unsigned err = 0u;
    const int tile = (v.n + (int)gridDim.x - 1) / (int)gridDim.x;
    const int first = blockIdx.x * tile, end = min(v.n, first + tile);
    int part = end - first;
    for (int base = first; base < end;) {
        part = min(part, end - base);
        if (tile64<MODEL, SPLIT>(v, v.S[s], v.S[s ^ 1], v.P[p], base, part, S, r, refresh, err)) {
            base += part;
            __syncthreads();
        } else {
            part = (part + 1) / 2;
        }
    }
    if (__any_sync(0xffffffffu, refresh) && (threadIdx.x & 31) == 0) atomicOr(&ctl->refresh, 1u);
    if (err) atomicOr(&ctl->error, err);
    if (last_block(&ctl->done[0])) {
        if (threadIdx.x == 0) {
            ctl->done[0] = 0;
            step_close(ctl, s, use_cond, 0, cond, cond2);
        }
    }
}

// ---------------------------------------------------------------- one warp to a tile
// The form for many particles: 32 of them to a warp, which passes through the
// same phases by itself.  Its candidates go through a ring and are drained 32 at
// a time with their results, so its shared memory is small and 12 unrelated
// warps keep an SM's pipes busy where a CTA's warps would wait for one another
// (83 % against 71 % busy on the 300,000-sphere bed).

// A warp's shared memory: the ring of candidates that may touch (a batch of 32
// is drained whenever 32 are there, and one pass over the rows adds 4 x 32 at
// most), and the results of the batch being drained.
constexpr int kRing64 = 192;
struct Warp64 {
    double r[12 * 32];    // normal force, tangential force, torque, rolling torque
    int j[kRing64];       // partner's storage index
    int ow[kRing64];      // owning particle within the tile
    int fl[32];           // what the batch position holds (kNone...), slot above
    unsigned owned[32];   // batch positions of each particle
    int nc0[32], nc[32];  // history length at the start of the step, now
};

struct Sum64 {
    double fx, fy, fz, mx, my, mz;
};
// one batch result added as the reference adds it: the normal force, the
// tangential force, the torque, the rolling torque
__device__ __forceinline__ void add64(Sum64& F, const double* r, int y, int kind) {
    F.fx += r[y];
    F.fy += r[32 + y];
    F.fz += r[64 + y];
    if (kind == kNormalOnly) return;
    F.fx += r[96 + y];
    F.fy += r[128 + y];
    F.fz += r[160 + y];
    F.mx += r[192 + y];
    F.my += r[224 + y];
    F.mz += r[256 + y];
    if (kind == kRolling) {
        F.mx += r[288 + y];
        F.my += r[320 + y];
        F.mz += r[352 + y];
    }
}

// Slots of a batch's contacts: those without one (`found` < 0 on a lane that is
// `hit`) are appended to their particle's row in batch order, which is row
// order; -1 when the row is full.  `grp`: the lanes of the same particle.
__device__ __forceinline__ int ring_slot64(Warp64& S, int lane, int ow, bool hit, int found, unsigned grp, int cap,
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
    double ri = 0., rx = 0., ry = 0., rz = 0.;
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
            c = pair_law64<MODEL>(v, dx, dy, dz, distsq, pi, pj, vi, vj, wi, wj, mi);
            normal64<32>(c, S.r, lane);
            rx = wi.x - wj.x;
            ry = wi.y - wj.y;
            rz = wi.z - wj.z;
        }
    }
    const unsigned grp = __match_any_sync(0xffffffffu, hit ? ow : 32 + lane);
    bool fresh;
    const int slot = ring_slot64(S, lane, ow, hit, found, grp, v.hist_cap, fresh);
    if (hit) {
        if (slot < 0) {
            err |= 0x4u;
            kind = kNormalOnly;
        } else {
            const size_t h = (size_t)slot * n + i;
            if (fresh) P.hid[h] = key;
            kind = finish64<32, MODEL>(v, c, ri, rx, ry, rz, P.hx, P.hy, P.hz, h, fresh, S.r, lane);
        }
        if ((grp & ((1u << lane) - 1u)) == 0u) S.owned[ow] = grp;
    }
    S.fl[lane] = kind | (slot << 2);
    __syncwarp();
    for (unsigned m = S.owned[lane]; m != 0u; m &= m - 1u) {
        const int y = __ffs((int)m) - 1;
        const int fl = S.fl[y];
        add64(F, S.r, y, fl & 3);
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
        double4_32a wi = make_double4_32a(0., 0., 0., 0.);
        if (hit) {
            found = search64(P.hwid, n, i, S.nc0[ow], t);
            wi = A.rot[i];
            c = wall_law64<MODEL>(v, f.nx, f.ny, f.nz, f.dist, rid, A.vel[i], wi, P.mat[i]);
            normal64<32>(c, S.r, lane);
        }
        const unsigned grp = __match_any_sync(0xffffffffu, hit ? ow : 32 + lane);
        bool fresh;
        const int slot = ring_slot64(S, lane, ow, hit, found, grp, v.histw_cap, fresh);
        if (hit) {
            if (slot < 0) {
                err |= 0x8u;
                kind = kNormalOnly;
            } else {
                const size_t h = (size_t)slot * n + i;
                if (fresh) P.hwid[h] = t;
                kind = finish64<32, MODEL>(v, c, rid, wi.x, wi.y, wi.z, P.hwx, P.hwy, P.hwz, h, fresh, S.r, lane);
            }
        }
        S.fl[lane] = kind | (slot << 2);
        __syncwarp();
        for (int y = y0; y < y1; y++) {
            const int fl = S.fl[y];
            if ((fl & 3) == kNone) continue;
            add64(F, S.r, y, fl & 3);
            if ((fl & 3) != kNormalOnly) touched |= 1ull << (fl >> 2);
        }
        __syncwarp();
    }
}

// One step of the 32 particles from `base` on, by one warp.
template <int MODEL>
__device__ __forceinline__ void warp_tile64(const View<FP64>& v, const SBank<FP64>& A, const SBank<FP64>& B,
                                       const PBank<FP64>& P, int base, Warp64& S, int lane, bool& refresh,
                                       unsigned& err) {
    constexpr int G = 4;
    const int n = v.n;
    const int i = base + lane;  // the particle this lane sums and integrates
    const bool mine = i < n;
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
    if (!active) {
        freeze64(v, A, B, i);
        return;
    }
    // ---------------- symplectic Euler (cpu_dem.cu:1622-1652)
    const double4_32a pi = A.pos[i], vi = A.vel[i], wi = A.rot[i];
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
    close64(v, A, B, i, nxp, nyp, nzp, nvx, nvy, nvz, nwx, nwy, nwz, refresh, err);
    if (v.store_forces) {
        v.fx[i] = F.fx; v.fy[i] = F.fy; v.fz[i] = F.fz;
        v.tx[i] = F.mx; v.ty[i] = F.my; v.tz[i] = F.mz;
    }
}

// One warp per CTA: the hardware hands tiles to SMs as they come free.
template <int MODEL>
__global__ void __launch_bounds__(32) k_step64_warp(View<FP64> v, cudaGraphConditionalHandle cond,
                                                    cudaGraphConditionalHandle cond2,
                                                    int use_cond) {
    __shared__ Warp64 S;
    Ctl* ctl = v.ctl;
    if (chain_passes(ctl, use_cond, cond2)) return;
    const int s = ctl->s, p = ctl->p;
    bool refresh = false;
    unsigned err = 0u;
    warp_tile64<MODEL>(v, v.S[s], v.S[s ^ 1], v.P[p], (int)blockIdx.x * 32, S, threadIdx.x, refresh, err);
    if (__any_sync(0xffffffffu, refresh) && threadIdx.x == 0) atomicOr(&ctl->refresh, 1u);
    if (err) atomicOr(&ctl->error, err);
    if (last_block(&ctl->done[0])) {
        if (threadIdx.x == 0) {
            ctl->done[0] = 0;
            step_close(ctl, s, use_cond, 0, cond, cond2);
        }
    }
}

template <int MODEL, bool SPLIT>
StepLaunch launch64(const View<FP64>& v, int tile) {
    void* fn = (void*)k_step64<MODEL, SPLIT>;
    // per device, and cheap beside the graph it is built for
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem64<MODEL>(true));
    return StepLaunch{fn, dim3((v.n + tile - 1) / tile), dim3(kThreads64), smem64<MODEL>(v.mat.mu_roll > 0.)};
}

}  // namespace

StepLaunch step_launch(const View<FP64>& v, int) {
    const bool hm = v.mat.model == 1;
    const int sms = sm_count();
    // Three CTAs share an SM.  Up to three tiles to an SM, tiles of at most 32
    // particles; beyond, tiles of up to 64 in whole rounds of three.  Over 12
    // rounds (117,000 spheres) a warp to a tile is faster.  Step of a
    // Hertz-Mindlin bed, a CTA and a warp to a tile: 100 spheres 24 and 56 us,
    // 3,000 32 and 89, 10,000 50 and 87, 40,000 148 and 149, 100,000 322 and
    // 335, 300,000 945 and 855.
    int rounds = (v.n + 32 * sms - 1) / (32 * sms);
    if (rounds > 3) rounds = 3 * ((v.n + 3 * kTile64 * sms - 1) / (3 * kTile64 * sms));
    if (rounds > 12) {
        void* fn = hm ? (void*)k_step64_warp<1> : (void*)k_step64_warp<0>;
        return StepLaunch{fn, dim3((v.n + 31) / 32), dim3(32), 0};
    }
    int tile = (v.n + rounds * sms - 1) / (rounds * sms);
    if (tile < 4) tile = 4;
    // Four particles have 20 contacts at most on beds, a batch of whole contacts
    // for one warp and three of split ones for three.  Whole and split, a step: 100
    // spheres (linear law) 20.9 and 18.4 us, 600 (Hertz-Mindlin) 23.0 and 20.9; 900,
    // six to a tile, 24.4 and 24.1, and 2,000 25.0 and 31.8.
    if (tile <= 4) return hm ? launch64<1, true>(v, tile) : launch64<0, true>(v, tile);
    return hm ? launch64<1, false>(v, tile) : launch64<0, false>(v, tile);
}

void launch_step(const View<FP64>& v, cudaStream_t st, cudaGraphConditionalHandle cond, int use_cond) {
    const StepLaunch L = step_launch(v);
    View<FP64> vv = v;
    cudaGraphConditionalHandle ci = cond;
    void* args[4] = {(void*)&vv, (void*)&cond, (void*)&ci, (void*)&use_cond};
    cudaLaunchKernel(L.fn, L.grid, L.block, args, L.smem, st);
}

}  // namespace gdem
