// CUDA kernels of the TIS-RNA Langevin step for sm_103a.
//
// One step of every replica (E: = src/16SCD_Mg_Cl_K_COPY_fast.cpp):
//   k_forces      deterministic_forces_MPI   E:2524-2586   every force of a replica group:
//                 pair tasks (SR_interactions_lists E:1783-1847; LR_interactions_lists
//                 E:1851-1907 every lr_interval steps or after a rebuild), bonded terms
//                 (polymer_constraints E:2354-2520), stacks by term (E:1911-2141), H-bonds of
//                 a replica per block with the valence-limited Monte Carlo (E:2145-2350),
//                 full_forces' Gaussians (E:2590-2611)
//   k_integrate   full_forces (application) + move_rigid_units + leap_frog_move_atom + adjust_box
//                                             E:2612-2732, E:570-642
//   k_cells       check_shifts' skin check   E:1741-1766 (the drop-in move_rigid_units, after
//                 which a caller may look at anything, ends with it in k_integrate), the
//                 replica's frame, and of a rebuilding replica separate_in_cells E:1461-1542
//                 and the H-bond candidates' status E:1698-1736
//   rebuild       populate_lists + separate_in_cells E:1461-1737, gated per replica
#include <cstdio>

#include "tis_fixed.cuh"
#include "tis_kernels.cuh"
#include "tis_tasks.cuh"

namespace tis {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// Programmatic dependent launch: the kernels of a step's sequential chain are
// launched so that their blocks may be scheduled while the previous kernel on
// the stream drains; each waits here, before its first global access, until that
// kernel has finished and its writes are visible (a no-op for a normal launch).
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------
// position and force accessors
// ---------------------------------------------------------------------------
template <bool D>
struct Pos;

template <>
struct Pos<false> {  // exact int32 differences -> FP32
    const int4 *q;
    float sx, sy, sz;
    __device__ V3<float> vec(int a, int b) const  // position(b) - position(a)
    {
        int4 qa = q[a], qb = q[b];
        return {(float)(int)((unsigned)qb.x - (unsigned)qa.x) * sx, (float)(int)((unsigned)qb.y - (unsigned)qa.y) * sy,
                (float)(int)((unsigned)qb.z - (unsigned)qa.z) * sz};
    }
};

template <>
struct Pos<true> {  // FP64 raw differences, no image (as the reference's bonded terms)
    const double *x, *y, *z;
    __device__ V3<double> vec(int a, int b) const { return {x[b] - x[a], y[b] - y[a], z[b] - z[a]}; }
};

template <bool D>
struct Acc;

template <>
struct Acc<false> {
    unsigned long long *f;
    int P;
    int err;
    __device__ void add(int i, V3<float> v)
    {
        atomic_add_fix(f + i, to_fix(v.x, err));
        atomic_add_fix(f + P + i, to_fix(v.y, err));
        atomic_add_fix(f + 2 * P + i, to_fix(v.z, err));
    }
};

template <>
struct Acc<true> {
    double *f;
    int P;
    int err;
    __device__ void add(int i, V3<double> v)
    {
        atomicAdd(f + i, v.x);
        atomicAdd(f + P + i, v.y);
        atomicAdd(f + 2 * P + i, v.z);
    }
};

template <bool D>
using Real = typename std::conditional<D, double, float>::type;

template <bool D>
__device__ inline Pos<D> make_pos(const Dev &d, const RepParams *R);
template <>
__device__ inline Pos<false> make_pos<false>(const Dev &d, const RepParams *R)
{
    return Pos<false>{d.q, R->qstep[0], R->qstep[1], R->qstep[2]};
}
template <>
__device__ inline Pos<true> make_pos<true>(const Dev &d, const RepParams *)
{
    return Pos<true>{d.x, d.y, d.z};
}

__device__ inline float atan2_(float a, float b) { return atan2f(a, b); }
__device__ inline double atan2_(double a, double b) { return atan2(a, b); }
__device__ inline float exp_(float v) { return expf(v); }
__device__ inline double exp_(double v) { return exp(v); }
__device__ inline float sqrt_(float v) { return sqrtf(v); }
__device__ inline double sqrt_(double v) { return sqrt(v); }
__device__ inline float rsqrt_(float v) { return 1.0f / sqrtf(v); }
__device__ inline double rsqrt_(double v) { return 1.0 / sqrt(v); }

// ---------------------------------------------------------------------------
// geometry and restraint forces (E:924-1454)
// ---------------------------------------------------------------------------
// valence_angle (E:986-1027): the angle at i2, as atan2(|a x b|, a.b), which
// equals the reference's acos(a.b / |a||b|) and stays accurate near 0 and pi.
template <bool D>
__device__ Real<D> angle_of(const Pos<D> &P, int i1, int i2, int i3)
{
    using R = Real<D>;
    V3<R> a = P.vec(i2, i1), b = P.vec(i2, i3);
    V3<R> w = cross(a, b);
    return atan2_(sqrt_(dot(w, w)), dot(a, b));
}

// dihedral_angle (E:1255-1302)
template <bool D>
__device__ Real<D> dihedral_of(const Pos<D> &P, int i1, int i2, int i3, int i4)
{
    using R = Real<D>;
    V3<R> v1 = P.vec(i1, i2), v2 = P.vec(i2, i3), v3 = P.vec(i3, i4);
    V3<R> m = cross(v1, v2), n = cross(v2, v3);
    return atan2_(dot(v1, n) * sqrt_(dot(v2, v2)), dot(m, n));
}

// The geometry of a term, from which its value and its force follow; a term's thread
// keeps it in registers while the other terms of its restraint are summed.
template <bool D>
struct BondGeom {
    V3<Real<D>> v;
    Real<D> r;
};
template <bool D>
struct AngleGeom {
    V3<Real<D>> a, b, w;
    Real<D> aa, bb, ab, ww, th;
};
template <bool D>
struct DihedralGeom {
    V3<Real<D>> m, n;
    Real<D> mm, nn, l2, p, q, psi;
};

template <bool D>
__device__ __forceinline__ BondGeom<D> bond_geom(const Pos<D> &P, int i1, int i2)
{
    const V3<Real<D>> v = P.vec(i1, i2);
    return {v, sqrt_(dot(v, v))};
}

template <bool D>
__device__ __forceinline__ AngleGeom<D> angle_geom(const Pos<D> &P, int i1, int i2, int i3)
{
    AngleGeom<D> g;
    g.a = P.vec(i2, i1);
    g.b = P.vec(i2, i3);
    g.aa = dot(g.a, g.a);
    g.bb = dot(g.b, g.b);
    g.ab = dot(g.a, g.b);
    g.w = cross(g.a, g.b);
    g.ww = sqrt_(dot(g.w, g.w));
    g.th = atan2_(g.ww, g.ab);
    return g;
}

template <bool D>
__device__ __forceinline__ DihedralGeom<D> dihedral_geom(const Pos<D> &P, int i1, int i2, int i3, int i4)
{
    DihedralGeom<D> g;
    const V3<Real<D>> v1 = P.vec(i1, i2), v2 = P.vec(i2, i3), v3 = P.vec(i3, i4);
    g.m = cross(v1, v2);
    g.n = cross(v2, v3);
    g.mm = dot(g.m, g.m);
    g.nn = dot(g.n, g.n);
    const Real<D> v22 = dot(v2, v2);
    g.l2 = sqrt_(v22);
    g.psi = atan2_(dot(v1, g.n) * g.l2, dot(g.m, g.n));
    g.p = dot(v1, v2) / v22;
    g.q = dot(v3, v2) / v22;
    return g;
}

// harmonic bond k0 (r0 - r)^2 (bead_bond_force / stacking_bond_force, E:924-982)
template <bool D>
__device__ __forceinline__ void bond_apply(const BondGeom<D> &g, Acc<D> &A, int i1, int i2, Real<D> k0, Real<D> r0)
{
    using R = Real<D>;
    const R t = R(2) * k0 * (r0 - g.r) / g.r;
    const V3<R> f = t * g.v;
    A.add(i1, R(-1) * f);
    A.add(i2, f);
}

// harmonic angle k0 (theta0 - theta)^2 at i2 (bead_valence_force E:1031-1134;
// clamp = stacking_valence_force E:1138-1251, no force once cos theta < -0.99995).
// The reference writes the force as s d(cos theta)/dx with s = -2 k0 (theta0 -
// theta) / sin theta; this is the same vector, 2 k0 (theta0 - theta) d theta/dx,
// with d theta/dx1 = a x w / (|a|^2 |w|), d theta/dx3 = -b x w / (|b|^2 |w|),
// w = a x b, which keeps FP32 accurate where sin theta is small.
template <bool D, bool ROLL = true>
__device__ __forceinline__ void angle_apply(const AngleGeom<D> &g, Acc<D> &A, int i1, int i2, int i3, Real<D> k0,
                                            Real<D> th0, bool clamp)
{
    using R = Real<D>;
    if (clamp && g.ab * rsqrt_(g.aa * g.bb) < R(-0.99995)) return;  // theta = pi, no force
    if (g.ww == R(0)) return;
    const R s = R(2) * k0 * (th0 - g.th) / g.ww;
    const V3<R> g1 = (s / g.aa) * cross(g.a, g.w);
    const V3<R> g3 = (-s / g.bb) * cross(g.b, g.w);
    // a loop, so that the beads share one copy of the fixed-point sum's code (instruction cache:
    // step of one 346-nt replica 19.5 -> 19.2 us, drop-in 50.6 -> 48.9 us, with the dihedral's);
    // ROLL false, a copy each, in the persistent kernel's six-term restraints (six_force: one
    // 60-nt replica on one CTA 98.4 -> 93.1 us a step, 64 of 203 nt 301 -> 293 us)
    V3<R> f = g1, f2 = R(-1) * (g1 + g3), f3 = g3;
#pragma unroll (ROLL ? 1 : 3)
    for (int k = 0; k < 3; ++k) {
        A.add(i1, f);
        f = f2; f2 = f3;
        i1 = i2; i2 = i3;
    }
}

// harmonic dihedral k0 (psi0 - psi)^2 (stacking_dihedral_force, E:1306-1454).
// The reference's s d(cos psi)/dx with s = -2 k0 (psi0 - psi) / sin psi equals
// 2 k0 (psi0 - psi) d psi/dx; here d psi/dx uses the cross-product form
// d psi/dx1 = -|v2| m / |m|^2, d psi/dx4 = |v2| n / |n|^2,
// d psi/dx2 = -(1 + v1.v2/|v2|^2) d psi/dx1 + (v3.v2/|v2|^2) d psi/dx4,
// which has no 1/sin psi and so no FP32 cancellation at planar (psi ~ 0, pi) geometry.
template <bool D, bool ROLL = true>
__device__ __forceinline__ void dihedral_apply(const DihedralGeom<D> &g, Acc<D> &A, int i1, int i2, int i3, int i4,
                                               Real<D> k0, Real<D> psi0)
{
    using R = Real<D>;
    if (g.mm == R(0) || g.nn == R(0)) return;
    const R c = R(2) * k0 * (psi0 - g.psi);
    const V3<R> g1 = (-c * g.l2 / g.mm) * g.m;
    const V3<R> g4 = (c * g.l2 / g.nn) * g.n;
    const V3<R> g2 = (R(-1) - g.p) * g1 + g.q * g4;
    V3<R> f = g1, f2 = g2, f3 = R(-1) * (g1 + g2 + g4), f4 = g4;
#pragma unroll (ROLL ? 1 : 4)
    for (int k = 0; k < 4; ++k) {
        A.add(i1, f);
        f = f2; f2 = f3; f3 = f4;
        i1 = i2; i2 = i3; i3 = i4;
    }
}

template <bool D>
__device__ void bond_force(const Pos<D> &P, Acc<D> &A, int i1, int i2, Real<D> k0, Real<D> r0)
{
    bond_apply<D>(bond_geom<D>(P, i1, i2), A, i1, i2, k0, r0);
}

template <bool D, bool ROLL = true>
__device__ void angle_force(const Pos<D> &P, Acc<D> &A, int i1, int i2, int i3, Real<D> k0, Real<D> th0, bool clamp)
{
    angle_apply<D, ROLL>(angle_geom<D>(P, i1, i2, i3), A, i1, i2, i3, k0, th0, clamp);
}

template <bool D, bool ROLL = true>
__device__ void dihedral_force(const Pos<D> &P, Acc<D> &A, int i1, int i2, int i3, int i4, Real<D> k0, Real<D> psi0)
{
    dihedral_apply<D, ROLL>(dihedral_geom<D>(P, i1, i2, i3, i4), A, i1, i2, i3, i4, k0, psi0);
}

// native dihedral imaged to within pi of the current one (E:1999-2019): branch -1/0/+1
template <class R>
__device__ inline int psi_branch(R psi, R nat)
{
    const R pi = R(3.14159265358979323846);
    if (fabs(psi - nat) <= pi) return 0;
    return (psi - nat > pi) ? 1 : -1;
}

template <class R>
__device__ inline R psi_shift(R nat, int br)
{
    return nat + R(2.0 * 3.14159265358979323846) * R(br);
}

// six-term native-geometry restraint (E:1983-2056, E:2177-2231, E:2319-2349)
template <bool D>
__device__ Real<D> six_q(const Pos<D> &P, const int *k, const double *nat, Real<D> rdev, Real<D> init, int &code)
{
    using R = Real<D>;
    R t1 = angle_of<D>(P, k[0], k[1], k[4]);
    R t2 = angle_of<D>(P, k[3], k[4], k[1]);
    R p0 = dihedral_of<D>(P, k[0], k[1], k[4], k[3]);
    R p1 = dihedral_of<D>(P, k[4], k[1], k[0], k[2]);
    R p2 = dihedral_of<D>(P, k[1], k[4], k[3], k[5]);
    int b0 = psi_branch<R>(p0, (R)nat[3]), b1 = psi_branch<R>(p1, (R)nat[4]), b2 = psi_branch<R>(p2, (R)nat[5]);
    code = (b0 + 1) + 3 * (b1 + 1) + 9 * (b2 + 1);
    R d0 = p0 - psi_shift<R>((R)nat[3], b0), d1 = p1 - psi_shift<R>((R)nat[4], b1), d2 = p2 - psi_shift<R>((R)nat[5], b2);
    R q = init + R(5) * rdev * rdev;
    q += R(1.5) * (t1 - (R)nat[1]) * (t1 - (R)nat[1]);
    q += R(1.5) * (t2 - (R)nat[2]) * (t2 - (R)nat[2]);
    q += R(0.15) * d0 * d0;
    q += R(0.15) * d1 * d1;
    q += R(0.15) * d2 * d2;
    return q;
}

template <bool D>
__device__ void six_force(const Pos<D> &P, Acc<D> &A, const int *k, const double *nat, int code, Real<D> w)
{
    using R = Real<D>;
    int b0 = code % 3 - 1, b1 = (code / 3) % 3 - 1, b2 = code / 9 - 1;
    bond_force<D>(P, A, k[1], k[4], R(5) * w, (R)nat[0]);
    angle_force<D, false>(P, A, k[0], k[1], k[4], R(1.5) * w, (R)nat[1], true);
    angle_force<D, false>(P, A, k[3], k[4], k[1], R(1.5) * w, (R)nat[2], true);
    dihedral_force<D, false>(P, A, k[0], k[1], k[4], k[3], R(0.15) * w, psi_shift<R>((R)nat[3], b0));
    dihedral_force<D, false>(P, A, k[4], k[1], k[0], k[2], R(0.15) * w, psi_shift<R>((R)nat[4], b1));
    dihedral_force<D, false>(P, A, k[1], k[4], k[3], k[5], R(0.15) * w, psi_shift<R>((R)nat[5], b2));
}

// The beads of term s of the six-term restraint, as places in its six (1-2: an angle's
// three, 3-5: a dihedral's four): chosen by number, so that the kinds of term have one copy
// of their code each: the roles of k_forces share one instruction cache (step of one 346-nt
// replica 21.1 -> 20.0 us, of 64 replicas 87.8 -> 85.5 us; a call per kind, not inlined: 20.7, 85.6)
struct SixBeads {
    int a, b, c, d;
};
__device__ __forceinline__ SixBeads six_beads(int s)
{
    if (s <= 2) return {s == 1 ? 0 : 3, s == 1 ? 1 : 4, s == 1 ? 4 : 1, 0};
    return {s == 3 ? 0 : s == 4 ? 4 : 1, s == 5 ? 4 : 1, s == 3 ? 4 : s == 4 ? 0 : 3, s == 3 ? 3 : s == 4 ? 2 : 5};
}

// Term s of the six-term restraint (0: the central distance, from rdev; 1-2: the
// angles; 3-5: the dihedrals, with the imaging branch of each in br): its weighted
// squared deviation, as six_q adds it.
template <bool D>
__device__ inline Real<D> six_term(const Pos<D> &P, const int *k, const double *nat, int s, Real<D> rdev, int &br)
{
    using R = Real<D>;
    br = 0;
    if (s == 0) return R(5) * rdev * rdev;
    const SixBeads n6 = six_beads(s);
    if (s <= 2) {
        const R t = angle_of<D>(P, k[n6.a], k[n6.b], k[n6.c]);
        const R n = (R)nat[s];
        return R(1.5) * (t - n) * (t - n);
    }
    const R p = dihedral_of<D>(P, k[n6.a], k[n6.b], k[n6.c], k[n6.d]);
    br = psi_branch<R>(p, (R)nat[s]);
    const R dd = p - psi_shift<R>((R)nat[s], br);
    return R(0.15) * dd * dd;
}

// force of term s of the six-term restraint (six_force's six calls, one at a time); br:
// the imaging branch of a dihedral
template <bool D>
__device__ inline void six_force_term(const Pos<D> &P, Acc<D> &A, const int *k, const double *nat, int br, Real<D> w,
                                      int s)
{
    using R = Real<D>;
    const SixBeads n6 = six_beads(s);
    if (s == 0) bond_force<D>(P, A, k[1], k[4], R(5) * w, (R)nat[0]);
    else if (s <= 2) angle_force<D>(P, A, k[n6.a], k[n6.b], k[n6.c], R(1.5) * w, (R)nat[s], true);
    else dihedral_force<D>(P, A, k[n6.a], k[n6.b], k[n6.c], k[n6.d], R(0.15) * w, psi_shift<R>((R)nat[s], br));
}

template <bool D>
__device__ inline Real<D> distance(const Pos<D> &P, int a, int b)
{
    V3<Real<D>> v = P.vec(a, b);
    return sqrt_(dot(v, v));
}

// ---------------------------------------------------------------------------
// exact FP64 pair distance with the reference's image rule (CC_vector, E:674-683)
// ---------------------------------------------------------------------------
__device__ inline double exact_r2(const Dev &d, const RepParams *R, int i, int j)
{
    double a = __dsub_rn(d.x[i], d.x[j]);
    double b = __dsub_rn(d.y[i], d.y[j]);
    double c = __dsub_rn(d.z[i], d.z[j]);
    if (a > R->hbox[0]) a = __dsub_rn(a, R->box[0]);
    if (a < -R->hbox[0]) a = __dadd_rn(a, R->box[0]);
    if (b > R->hbox[1]) b = __dsub_rn(b, R->box[1]);
    if (b < -R->hbox[1]) b = __dadd_rn(b, R->box[1]);
    if (c > R->hbox[2]) c = __dsub_rn(c, R->box[2]);
    if (c < -R->hbox[2]) c = __dadd_rn(c, R->box[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
}

__device__ inline void exact_vec(const Dev &d, const RepParams *R, int i, int j, double v[3])
{
    v[0] = d.x[i] - d.x[j];
    v[1] = d.y[i] - d.y[j];
    v[2] = d.z[i] - d.z[j];
    for (int k = 0; k < 3; ++k) {
        if (v[k] > R->hbox[k]) v[k] = v[k] - R->box[k];
        if (v[k] < -R->hbox[k]) v[k] = v[k] + R->box[k];
    }
}

__device__ inline bool is_charged(int kind) { return kind != 1 && kind != 2; }

// Relative half-width of the band around a threshold inside which the FP32
// squared distance cannot decide a comparison and the exact FP64 one is used.
constexpr float kBand = 1.0e-5f;

// ---------------------------------------------------------------------------
// quantisation: fixed-point copy of the FP64 positions
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_quantize(Dev d)
{
    int p = blockIdx.x * kBlock + threadIdx.x;
    const RepParams *R = d.rp + d.blk_rep[blockIdx.x];
    int4 q = d.q[p];
    q.x = (int)(unsigned)(long long)floor(d.x[p] * R->qinv[0]);
    q.y = (int)(unsigned)(long long)floor(d.y[p] * R->qinv[1]);
    q.z = (int)(unsigned)(long long)floor(d.z[p] * R->qinv[2]);
    d.q[p] = q;
}

// packed (unpadded, replicas end to end) state <-> the padded device arrays; N is
// the group's particle count, stage holds the nine arrays of N values each
__global__ void __launch_bounds__(kBlock) k_put_state(Dev d, const double *stage, int N)
{
    const int p = blockIdx.x * kBlock + threadIdx.x;
    const RepParams *R = d.rp + d.blk_rep[blockIdx.x];
    const int i = p - R->p0;
    if (i >= R->n) return;
    double *dst[9] = {d.x, d.y, d.z, d.xo, d.yo, d.zo, d.vx, d.vy, d.vz};
    for (int c = 0; c < 9; ++c) dst[c][p] = stage[(size_t)c * N + R->pk0 + i];
    int4 q = d.q[p];
    q.x = (int)(unsigned)(long long)floor(d.x[p] * R->qinv[0]);
    q.y = (int)(unsigned)(long long)floor(d.y[p] * R->qinv[1]);
    q.z = (int)(unsigned)(long long)floor(d.z[p] * R->qinv[2]);
    d.q[p] = q;
}

__global__ void __launch_bounds__(kBlock) k_get_state(Dev d, double *stage, int N, unsigned mask)
{
    const int p = blockIdx.x * kBlock + threadIdx.x;
    const RepParams *R = d.rp + d.blk_rep[blockIdx.x];
    const int i = p - R->p0;
    if (i >= R->n) return;
    const double *src[9] = {d.x, d.y, d.z, d.xo, d.yo, d.zo, d.vx, d.vy, d.vz};
    for (int c = 0; c < 9; ++c)
        if ((mask >> c) & 1u) stage[(size_t)c * N + R->pk0 + i] = src[c][p];
}

// ---------------------------------------------------------------------------
// pair forces over the full (both-direction) neighbour lists
// ---------------------------------------------------------------------------
// Loads of data that the fused step kernel rewrites while it runs (positions, lists) go
// through L2 (__ldcg).  The step's separate kernels use plain loads: the read-only path
// (__ldg) is for data that nothing writes while the kernel exists, and theirs, launched
// while its predecessor drains, may exist before the last write has landed.  No
// difference in time: step of one 346-nt replica 17.60 and 17.61 us, of 64 replicas 79.33 and
// 79.37 us, of 16 large ones 186.0 and 185.8 us.

// the replica's FP32 pair tables as the pair code reads them (shared memory copies)
struct PairTables {
    const float *dlj2, *dm, *flj, *qclb;
};

// The force of one list entry (partner j, packed position qj, ljw: the weight of its LJ
// term) on the particle p of type tp: mixed precision, added to (ax, ay, az) in fixed
// point.  An LR entry has no LJ term (LR_interactions_lists, E:1851-1907), however far its
// pair is: LR known, or a weight of zero.  Each term takes its own root: leaving before a
// common one where neither applies cost the persistent kernel up to 8% (FP64, one 76-nt
// replica on one CTA: 399 -> 436 us a step) and gave the force launch nothing.
template <bool LR, bool EN>
__device__ __forceinline__ void pair_entry(const Dev &d, const RepParams *R, int p, const int4 &qp, int tp, bool chp,
                                           int j, const int4 &qj, float ljw, const PairTables &tb, float kap, float lo,
                                           float hi, long long &ax, long long &ay, long long &az, int &err,
                                           double &e_lj, double &e_c)
{
    const float dx = (float)(int)((unsigned)qp.x - (unsigned)qj.x) * R->qstep[0];
    const float dy = (float)(int)((unsigned)qp.y - (unsigned)qj.y) * R->qstep[1];
    const float dz = (float)(int)((unsigned)qp.z - (unsigned)qj.z) * R->qstep[2];
    const float r2 = dx * dx + dy * dy + dz * dz;
    const int tj = qj.w & 0xff, kj = (qj.w >> 8) & 0xff;
    const int J = jn12(tp, tj);
    const bool lj = !LR && ljw != 0.0f && r2 <= tb.dlj2[J];
    bool cou = (LR || (chp && is_charged(kj))) && r2 <= hi;
    if (cou && !(r2 <= lo)) cou = exact_r2(d, R, p, j) <= R->rc2;
    float F = 0.0f;
    if (lj) {  // LJ_FORCE (E:801-821)
        const float rr = sqrtf(r2);
        const float dr = rr - tb.dm[J];
        const float s = 1.5852f / dr;
        const float s2 = s * s, s4 = s2 * s2, s8 = s4 * s4, s14 = s8 * s4 * s2;
        F = ljw * (tb.flj[J] * (s14 - s8) * dr / rr);
        if (EN) {
            double e;
            if ((double)r2 < R->d2min_d[J]) e = R->elj_d[J] * 1001.0;
            else {
                const float s6 = s4 * s2, s12 = s6 * s6;
                e = (double)(R->elj[J] * (s12 - 2.0f * s6 + 1.0f));
            }
            e_lj += 0.5 * (double)ljw * e;
        }
    }
    if (cou) {  // COULOMB_TRUNCATED_FORCE (E:841-855)
        const float rr = sqrtf(r2);
        if (kap == 0.0f) {
            F += tb.qclb[J] / (r2 * rr);
            if (EN) e_c += 0.5 * (double)(tb.qclb[J] / rr);
        } else {  // screened: U = C exp(-kappa r) / r, F / r = U (1 + kappa r) / r^2
            const float kr = kap * rr, u = tb.qclb[J] * expf(-kr) / rr;
            F += u * (1.0f + kr) / r2;
            if (EN) e_c += 0.5 * (double)u;
        }
    }
    if (F != 0.0f) {
        ax += to_fix(F * dx, err);
        ay += to_fix(F * dy, err);
        az += to_fix(F * dz, err);
    }
}

// the same entry in FP64, from the FP64 positions with the reference's image rule
template <bool LR, bool EN>
__device__ __forceinline__ void pair_entry(const Dev &d, const RepParams *R, int p, int tp, bool chp, int j, int wj,
                                           double ljw, double &ax, double &ay, double &az, double &e_lj, double &e_c)
{
    const int tj = wj & 0xff, kj = (wj >> 8) & 0xff;
    const int J = jn12(tp, tj);
    double v[3];
    exact_vec(d, R, p, j, v);
    const double r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    const bool lj = !LR && ljw != 0.0 && r2 <= R->dlj2_d[J];
    const bool cou = (LR || (chp && is_charged(kj))) && r2 <= R->rc2;
    double F = 0.0;
    if (lj) {
        const double rr = sqrt(r2);
        const double dr = rr + kSig0 - R->dlj_d[J];
        const double s = kSig0 / dr;
        const double s2 = s * s, s4 = s2 * s2, s8 = s4 * s4, s14 = s8 * s4 * s2;
        F = ljw * (R->flj_d[J] * (s14 - s8) * dr / rr);
        if (EN) {
            double e;
            if (r2 < R->d2min_d[J]) e = R->elj_d[J] * 1001.0;
            else {
                const double s6 = s4 * s2, s12 = s6 * s6;
                e = R->elj_d[J] * (s12 - 2.0 * s6 + 1.0);
            }
            e_lj += 0.5 * ljw * e;
        }
    }
    if (cou) {
        const double rr = sqrt(r2);
        if (R->kappa == 0.0) {
            F += R->qclb_d[J] / (rr * r2);
            if (EN) e_c += 0.5 * R->qclb_d[J] / rr;
        } else {
            const double kr = R->kappa * rr, u = R->qclb_d[J] * exp(-kr) / rr;
            F += u * (1.0 + kr) / r2;
            if (EN) e_c += 0.5 * u;
        }
    }
    ax += v[0] * F;
    ay += v[1] * F;
    az += v[2] * F;
}

// The pair forces of particle p over its full list, by L threads (lane4 = its lane
// among them): slot k of the list goes to lane k % L; lane 0 adds the sum (LR: stores
// the held LR force).  The persistent fused step kernel's form; the separate kernel
// takes a block's list entries as tasks (k_pair).
template <bool D, bool LR, int L>
__device__ __forceinline__ void pair_particle(const Dev &d, const RepParams *R, int p, int lane4, const PairTables &tb,
                                              int &err)
{
    const int P = d.P;
    const int4 qp = d.q[p];
    const int tp = qp.w & 0xff, act = (qp.w >> 16) & 1;
    const bool chp = is_charged((qp.w >> 8) & 0xff);
    const int cnt = act ? (LR ? d.n_lr[p] : d.n_sr[p]) : 0;
    const int *nbr = LR ? d.nbr_lr : d.nbr_sr;
    double e0 = 0, e1 = 0;
    typename std::conditional<D, double, long long>::type ax = 0, ay = 0, az = 0;
    const float lo = R->rc2f * (1.0f - kBand), hi = R->rc2f * (1.0f + kBand);
    const float kap = R->kappaf;
    for (int k = lane4; k < cnt; k += L) {
        const int raw = __ldcg(nbr + nb_idx(k, p, P));
        const int j = raw & kIdxMask;
        if constexpr (!D) {
            const float ljw = LR ? 1.0f : (float)(1 - (raw >> kExclShift));
            pair_entry<LR, false>(d, R, p, qp, tp, chp, j, __ldcg(d.q + j), ljw, tb, kap, lo, hi, ax, ay, az, err,
                                  e0, e1);
        } else {
            const double ljw = LR ? 1.0 : (double)(1 - (raw >> kExclShift));
            pair_entry<LR, false>(d, R, p, tp, chp, j, d.q[j].w, ljw, ax, ay, az, e0, e1);
        }
    }
    for (int o = 1; o < L; o <<= 1) {
        ax += __shfl_xor_sync(kFull, ax, o);
        ay += __shfl_xor_sync(kFull, ay, o);
        az += __shfl_xor_sync(kFull, az, o);
    }
    if (lane4 != 0) return;
    if constexpr (!D) {
        if (LR) {  // the LR force is kept for the MTS interval: overwrite
            d.flr[p] = (unsigned long long)ax;
            d.flr[P + p] = (unsigned long long)ay;
            d.flr[2 * P + p] = (unsigned long long)az;
        } else if (act) {  // other force kernels run concurrently: accumulate
            atomic_add_fix(d.f + p, ax);
            atomic_add_fix(d.f + P + p, ay);
            atomic_add_fix(d.f + 2 * P + p, az);
        }
    } else {
        double *out = LR ? (double *)d.flr : (double *)d.f;
        if (LR) {
            out[p] = ax;
            out[P + p] = ay;
            out[2 * P + p] = az;
        } else if (act) {
            atomicAdd(out + p, ax);
            atomicAdd(out + P + p, ay);
            atomicAdd(out + 2 * P + p, az);
        }
    }
}

// barriers of the threads that run a block-level part: the whole CTA, or warps
// 0 .. n/32-1 of it on a named barrier (the fused step kernel's H-bond warps)
struct CtaBar {
    __device__ void operator()() const { __syncthreads(); }
};
struct NamedBar {
    int id, n;
    __device__ void operator()() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
};


template <bool D, int PB>
struct PairSmem {
    float dlj2[46], dm[46], flj[46], qclb[46];
    int4 q[PB];          // packed positions of the particles
    TaskSmem<PB> tasks;
};
template <int PB>
struct PairSmem<true, PB> : PairSmem<false, PB> {
    double f[3][kPairTasks];  // the forces of the window's tasks
};

// FP64 sums of the tasks' forces in an order that the lists alone set, so that the same state
// gives the same force, whatever the handle's other replicas and the launch's shape: one
// thread sums a particle's SR entries in list order, four its LR entries, entry k by
// thread k % 4.  One task is one entry here, and a particle's are numbered end to end, SR first.
template <int PB>
struct OrderedSums {
    double sr[3] = {0, 0, 0}, lr[3] = {0, 0, 0};
    // the tasks win .. win + nt - 1, between barriers
    __device__ __forceinline__ void window(const PairSmem<true, PB> &sm, int tid, int win, int nt)
    {
        if (tid < PB) {
            int lo, ns, nl;
            place(sm, tid, win, lo, ns, nl);
            for (int k = max(lo, 0), e = min(lo + ns, nt); k < e; ++k)
                for (int c = 0; c < 3; ++c) sr[c] += sm.f[c][k];
        }
        if (tid < 4 * PB) {
            int lo, ns, nl;
            place(sm, tid >> 2, win, lo, ns, nl);
            lo += ns;
            const int e = min(lo + nl, nt), j = tid & 3;
            for (int k = lo + (lo < 0 ? ((-lo - j + 3) & ~3) : 0) + j; k < e; k += 4)
                for (int c = 0; c < 3; ++c) lr[c] += sm.f[c][k];
        }
    }
    // a particle's first task, counted from the window's first, and its list lengths
    static __device__ __forceinline__ void place(const PairSmem<true, PB> &sm, int pl, int win, int &lo, int &ns, int &nl)
    {
        const int4 at = sm.tasks.at[pl];
        lo = at.x - win;
        for (int v = 0; v < (pl >> 5); ++v) lo += sm.tasks.cnt[v].x;
        ns = at.z;
        nl = at.w;
    }
    __device__ __forceinline__ void store(const Dev &d, int p0, int tid, bool do_lr) const
    {
        double *f = (double *)d.f, *flr = (double *)d.flr;
        const int P = d.P;
        if (tid < PB && (sr[0] != 0 || sr[1] != 0 || sr[2] != 0))  // beside the other terms' atomics
            for (int c = 0; c < 3; ++c) atomicAdd(f + c * P + p0 + tid, sr[c]);
        if (do_lr && tid < 4 * PB)
            for (int c = 0; c < 3; ++c) {
                double v = lr[c];
                v += __shfl_xor_sync(kFull, v, 1);
                v += __shfl_xor_sync(kFull, v, 2);
                if ((tid & 3) == 0) flr[c * P + p0 + (tid >> 2)] = v;
            }
    }
};

// Pair forces of PB particles (sub-block pb) by the TS threads of one sub-block, over
// their SR lists and, where the LR force is due (do_lr: 0 never, 1 when
// RepState::lr_now is set, 2 always), their LR lists.
//
// Their list entries are dealt out as tasks (tis_tasks.cuh): a thread per particle took one
// dependent load after another for as long as its warp's longest list.  FP64 tasks hold
// one entry: FP64 latency and the narrow FP64 pipe bound them; their sums keep an order (OrderedSums).
// Alone, SR lists of 5 replicas of a 346-nt chain: 22.3 -> 11.9 us; one 76-nt replica in
// FP64: 52 -> 15 us.
template <bool D, bool EN, bool EX, int PB, int TS, class Bar>
__device__ __forceinline__ void pair_tasks(const Dev &d, int pb, int do_sr, int do_lr, int tid, PairSmem<D, PB> &sm, Bar bar)
{
    constexpr int U = D ? 1 : 4;  // entries per task
    static_assert(TS >= (D ? 4 * PB : PB), "a thread per particle; for FP64 sums four");
    const int p0 = pb * PB, r = d.blk_rep[p0 / kBlock], P = d.P;
    const RepParams *R = d.rp + r;
    const bool lr = do_lr == 2 || (do_lr == 1 && d.rs[r].lr_now);
    if (!do_sr && !lr) return;
    if (!D)
        for (int t = tid; t < 46; t += TS) {
            sm.dlj2[t] = R->dlj2[t];
            sm.dm[t] = R->dm[t];
            sm.flj[t] = R->flj[t];
            sm.qclb[t] = R->qclb[t];
        }
    const PairTables tb{sm.dlj2, sm.dm, sm.flj, sm.qclb};
    const int lane = tid & 31;
    if (tid < PB) {
        const int p = p0 + tid;
        const int4 qp = d.q[p];
        sm.q[tid] = qp;
        const bool act = (qp.w >> 16) & 1;
        const int ns = act && do_sr ? d.n_sr[p] : 0, nl = act && lr ? d.n_lr[p] : 0;
        if (!D && lr)  // the LR force is kept for the MTS interval: started again here, its tasks add to it
            for (int c = 0; c < 3; ++c) d.flr[c * P + p] = 0ull;
        tasks_count<PB, U>(sm.tasks, tid, ns, nl);
    }
    bar();
    const int total = tasks_total(sm.tasks);
    int err = 0;
    double e_lj = 0, e_c = 0, e_cl = 0;
    typename std::conditional<D, OrderedSums<PB>, int>::type sums{};
    for (int win = 0; win < total; win += kPairTasks) {
        if (win) bar();  // the previous window's tasks are done
        if (tid < PB) tasks_window<PB, U>(sm.tasks, tid, win);
        bar();
        const int nt = min(total - win, kPairTasks);
        const float lo = R->rc2f * (1.0f - kBand), hi = R->rc2f * (1.0f + kBand);
        const float kap = R->kappaf;
        for (int t = tid; t < nt; t += TS) {
            const int task = sm.tasks.task[t];
            const int pl = task_particle(task), p = p0 + pl, cnt = task_entries(task);
            const bool tlr = task_lr(task);
            const int *nbr = tlr ? d.nbr_lr : d.nbr_sr;
            double ec = 0;
            if constexpr (!D) {
                const int4 e4 = ((const int4 *)nbr)[(size_t)task_chunk(task) * P + p];
                int raw[4] = {e4.x, e4.y, e4.z, e4.w};
                const int4 qp = sm.q[pl];
                const int tp = qp.w & 0xff;
                const bool chp = is_charged((qp.w >> 8) & 0xff);
                long long ax = 0, ay = 0, az = 0;
                int4 qj[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < cnt) qj[k] = d.q[raw[k] & kIdxMask];
                // one copy of the entry's code, the four taking turns in its registers: the roles of
                // this launch together overrun the instruction cache (64 replicas: 92.7 -> 87.7 us a step)
#pragma unroll 1
                for (int k = 0; k < cnt; ++k) {
                    const float ljw = tlr ? 0.0f : EX ? (float)(1 - (raw[0] >> kExclShift)) : 1.0f;
                    pair_entry<false, EN>(d, R, p, qp, tp, chp, raw[0] & kIdxMask, qj[0], ljw, tb, kap, lo, hi, ax, ay, az,
                                          err, e_lj, ec);
#pragma unroll
                    for (int u = 0; u < 3; ++u) {
                        raw[u] = raw[u + 1];
                        qj[u] = qj[u + 1];
                    }
                }
                if (ax | ay | az) {
                    unsigned long long *out = tlr ? d.flr : d.f;
                    atomic_add_fix(out + p, ax);
                    atomic_add_fix(out + P + p, ay);
                    atomic_add_fix(out + 2 * P + p, az);
                }
            } else {
                const int raw = nbr[nb_idx(task_chunk(task), p, P)];
                const int wp = sm.q[pl].w;
                const double ljw = tlr ? 0.0 : EX ? (double)(1 - (raw >> kExclShift)) : 1.0;
                double ax = 0, ay = 0, az = 0;
                pair_entry<false, EN>(d, R, p, wp & 0xff, is_charged((wp >> 8) & 0xff), raw & kIdxMask,
                                      d.q[raw & kIdxMask].w, ljw, ax, ay, az, e_lj, ec);
                sm.f[0][t] = ax;
                sm.f[1][t] = ay;
                sm.f[2][t] = az;
            }
            if (EN) {
                if (tlr) e_cl += ec;
                else e_c += ec;
            }
        }
        if constexpr (D) {
            bar();
            sums.window(sm, tid, win, nt);
        }
    }
    if constexpr (D) sums.store(d, p0, tid, lr);
    if (EN) {
        for (int o = 16; o > 0; o >>= 1) {
            e_lj += __shfl_down_sync(kFull, e_lj, o);
            e_c += __shfl_down_sync(kFull, e_c, o);
            e_cl += __shfl_down_sync(kFull, e_cl, o);
        }
        if (lane == 0) {
            if (do_sr) {
                atomicAdd(d.eterm + r * kNE + 0, e_lj);
                atomicAdd(d.eterm + r * kNE + 1, e_c);
            }
            if (lr) atomicAdd(d.eterm + r * kNE + 2, e_cl);
        }
    }
    if (err) atomicOr(&d.rs[r].err, err);
}

// the pair forces alone: with energies each bonded pair's LJ counts, as the reference's terms have
// it (tis_compute_forces); without, as the step leaves it out (stage timing)
constexpr int kPairAlone = 128;
template <bool D, bool EN>
__global__ void __launch_bounds__(kPairAlone) k_pair(Dev d, int do_sr, int do_lr)
{
    __shared__ PairSmem<D, 32> sm;
    pair_tasks<D, EN, !EN, 32, kPairAlone>(d, blockIdx.x, do_sr, do_lr, (int)threadIdx.x, sm, CtaBar{});
}

// ---------------------------------------------------------------------------
// block reductions
// ---------------------------------------------------------------------------
// sum of NV doubles over threads tid = 0 .. nthr-1 (a multiple of 32) into tid 0
template <int NV, class Bar>
__device__ void block_sum_t(double (&v)[NV], double *smem /* NV * 32 */, int tid, int nthr, Bar bar)
{
    const int lane = tid & 31, w = tid >> 5, nw = (nthr + 31) >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(kFull, v[i], o);
    bar();
    if (lane == 0)
        for (int i = 0; i < NV; ++i) smem[i * 32 + w] = v[i];
    bar();
    if (w == 0) {
        for (int i = 0; i < NV; ++i) {
            double t = lane < nw ? smem[i * 32 + lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(kFull, t, o);
            v[i] = t;
        }
    }
    bar();
}

template <int NV>
__device__ void block_sum(double (&v)[NV], double *smem /* NV * 32 */)
{
    block_sum_t<NV>(v, smem, (int)threadIdx.x, (int)blockDim.x, CtaBar{});
}

// ---------------------------------------------------------------------------
// integrator: noise application, leap-frog, recentring, ion wrap, skin check
// ---------------------------------------------------------------------------
template <bool D>
__device__ inline double total_force(const Dev &d, int p, int c)
{
    if (D) {
        const double *f = (const double *)d.f, *fl = (const double *)d.flr;
        return __ldcg(f + c * d.P + p) + __ldcg(fl + c * d.P + p);
    }
    const long long t = (long long)(__ldcg(d.f + c * d.P + p) + __ldcg(d.flr + c * d.P + p));
    return (double)t * (1.0 / kFixScale);
}

// the step's 3000 Gaussians of replica r (RepState::pending)
__device__ __forceinline__ const double *step_noise(const Dev &d, int r)
{
    const unsigned pending = __ldcg(&d.rs[r].pending), drawn = pending ? pending - 1u : 0u;  // written in this very kernel (k_forces)
    return d.gnoise + (size_t)r * kNoiseStride + (drawn <= kNoiseSpare ? drawn : kNoise + kNoiseSpare);
}

// leap_frog_move_atom (E:570-642) with the noise of full_forces (E:2612-2622).
// FP64 mode follows the reference's operation order.  Mixed mode evaluates the
// same update v' = K1 v + K2 (f + g sigma) as K1 v + (K2 2^-32) f_fix + (K2 sigma) g
// with fused multiply-adds, and x' = x + (x - x_old) + (v' - v) h; the velocity
// cap m v'^2 / (300 T) > 1 uses the precomputed m / (300 T) in both modes.
template <bool D, bool I>
__device__ inline void leap_frog(const Dev &d, const RepParams *R, int r, int p, double xn[3], double vn[3], float2 *e2 = nullptr)
{
    const int t = d.q[p].w & 0xff;
    const double v0[3] = {d.vx[p], d.vy[p], d.vz[p]};
    const double x0[3] = {d.x[p], d.y[p], d.z[p]};
    const double o0[3] = {d.xo[p], d.yo[p], d.zo[p]};
    const int k = (p - R->p0 + 1) % 1000;
    const double *g = step_noise(d, r);
    if (D) {
        double f[3] = {total_force<D>(d, p, 0), total_force<D>(d, p, 1), total_force<D>(d, p, 2)};
        if (d.noise == 0) {
            const double sg = R->sigma[t];
            for (int c = 0; c < 3; ++c) f[c] = __dadd_rn(f[c], __dmul_rn(g[k + 1000 * c], sg));
        }
        for (int c = 0; c < 3; ++c) vn[c] = __dadd_rn(__dmul_rn(R->k1[t], v0[c]), __dmul_rn(R->k2[t], f[c]));
    } else {
        const double k1 = R->k1[t], kf = R->k2fix[t], kg = d.noise == 0 ? R->k2sig[t] : 0.0;
        for (int c = 0; c < 3; ++c) {
            const long long fx = (long long)(__ldcg(d.f + c * d.P + p) + __ldcg(d.flr + c * d.P + p));
            vn[c] = fma(kg, g[k + 1000 * c], fma(kf, fix_to_double(fx), k1 * v0[c]));
        }
    }
    // a component below sqrt(0.33 / vcap) each (vcut: that value's high word) cannot reach
    // the cap; a runaway or NaN component has a larger high word and takes the FP64 test
    const int hv = max(max(__double2hiint(vn[0]) & 0x7fffffff, __double2hiint(vn[1]) & 0x7fffffff),
                       __double2hiint(vn[2]) & 0x7fffffff);
    if (hv >= R->vcut[t]) {
        double vsq = R->vcap[t] * (vn[0] * vn[0] + vn[1] * vn[1] + vn[2] * vn[2]);
        if (vsq > 1.0) {
            vsq = 1.0 / sqrt(vsq);
            for (int c = 0; c < 3; ++c) vn[c] *= vsq;
        }
    }
    // |x' - x|^2 in FP32, good to 1e-5 unless its two parts cancel (or it all but
    // vanishes): then nothing (x) and an upper bound (y)
    float s = 0.0f, parts = 0.0f;
    for (int c = 0; c < 3; ++c) {
        float a;
        const double t = axis_ahead<D, I>(R, c, x0[c], o0[c], a);
        const double dv = vn[c] - v0[c];
        xn[c] = D ? __dadd_rn(t, __dmul_rn(dv, R->h)) : fma(dv, R->h, t);
        const float b = cut_to_float(dv) * R->hf, e = a + b;
        s += e * e;
        parts += a * a + b * b;
    }
    if (e2) {
        const bool bad = s < R->e2min || parts > 64.0f * s;
        *e2 = make_float2(bad ? 0.0f : s, bad ? 2.1f * parts + R->e2pad : s);
    }
}

// two Gaussians of full_forces (E:2594-2606) from the draws v1 and v2
template <bool D>
__device__ __forceinline__ double2 gaussians(uint32_t v1, uint32_t v2)
{
    if (D) {  // Box-Muller as the reference forms it (E:2598-2606), in FP64
        const double a = sqrt(-2.0 * log(u31_ratio(v1)));
        const double b = 2.0 * 3.14159265358979323846 * u31_ratio(v2);
        double sn, cs;
        sincos(b, &sn, &cs);
        return make_double2(a * cs, a * sn);
    }
    // FP32 Box-Muller, radius accurate over the whole uniform range
    const float a = bm_radius(v1);
    float sn, cs;
    sincospif(2.0f * ((float)v2 * (1.0f / 2147483647.0f)), &sn, &cs);
    return make_double2((double)(a * cs), (double)(a * sn));
}

// Pairs of Gaussians from draw c0 on, pair k from draws c0 + 2 k and c0 + 2 k + 1: one Philox
// block holds four draws, so thread j forms the (up to two) pairs of [0, pairs) whose first
// draw lies in block c0 / 4 + j.  The Monte Carlo takes its draws in twos, so c0 is even and
// a block's draws suffice; after an odd count the last pair takes one of the next block.
// A quarter of the Philox blocks of a draw at a time: step of 64 replicas 85.6 -> 85.0 us,
// the drop-in step 50.8 -> 49.9 us.
__host__ __device__ constexpr int noise_blocks(int pairs) { return pairs / 2 + 1; }
template <bool D>
__device__ __forceinline__ void noise_block(unsigned long long seed, unsigned long long c0, int pairs, int j, double *out)
{
    const unsigned long long b = (c0 >> 2) + (unsigned long long)j;
    uint32_t c[4] = {(uint32_t)b, (uint32_t)(b >> 32), 0u, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    uint32_t v1 = rand_word(c[0]), v2 = rand_word(c[1]), v3 = rand_word(c[2]), v4 = rand_word(c[3]);
    if (c0 & 1u) {
        v1 = v2;
        v2 = v3;
        v3 = v4;
        v4 = rand_value(seed, 4 * b + 4);
    }
    int k = 2 * j - (int)((c0 >> 1) & 1u);
#pragma unroll 1
    for (int i = 0; i < 2; ++i, ++k) {
        if (k >= 0 && k < pairs) ((double2 *)out)[k] = gaussians<D>(v1, v2);
        v1 = v3;
        v2 = v4;
    }
}

// all Gaussians of one replica from draw c0 on, by the threads of one block
template <bool D>
__device__ void gen_noise(const Dev &d, int r, unsigned long long c0, double *out, int tid, int nthr)
{
    if (d.noise != 0) return;
    for (int j = tid; j < noise_blocks(kNoise / 2); j += nthr) noise_block<D>(d.rp[r].seed, c0, kNoise / 2, j, out);
}

// the step's Gaussians alone (the drop-in full_forces call), one block per replica;
// the reference draws them even when the noise amplitude is zero.  A thread per Philox
// block, launched while the forces drain (drop-in step of one 346-nt replica 46.1 -> 45.6 us)
constexpr int kNoiseThreads = (noise_blocks(kNoise / 2) + 31) / 32 * 32;
template <bool D>
__global__ void k_noise(Dev d)
{
    wait_prior_grid();
    const int r = blockIdx.x;
    const unsigned long long c0 = d.rs[r].ctr;
    gen_noise<D>(d, r, c0, d.gnoise + (size_t)r * kNoiseStride, (int)threadIdx.x, (int)blockDim.x);
    __syncthreads();
    if (threadIdx.x == 0) d.rs[r].ctr = c0 + kNoise;
}

// ---------------------------------------------------------------------------
// bonded terms and stacks of every replica, one thread per term
// ---------------------------------------------------------------------------

// LJ force of an excluded (bonded) pair, as reduce_forces subtracts it (E:880-897)
template <bool D, bool EN>
__device__ void exclusion_lj(const Dev &d, const RepParams *R, const Pos<D> &P, Acc<D> &A, int a, int ex,
                             double &e_excl)
{
    using Rl = Real<D>;
    const int ta = d.q[a].w & 0xff, tb = d.q[ex].w & 0xff;
    const int J = jn12(ta, tb);
    V3<Rl> v = P.vec(ex, a);  // x_a - x_ex, minimum image
    if (D) {
        double w[3];
        exact_vec(d, R, a, ex, w);
        v = V3<Rl>{(Rl)w[0], (Rl)w[1], (Rl)w[2]};
    }
    const Rl r2 = dot(v, v);
    if (!(r2 <= (Rl)(D ? R->dlj2_d[J] : R->dlj2[J]))) return;
    const Rl rr = sqrt_(r2);
    const Rl dr = D ? (Rl)(rr + kSig0 - R->dlj_d[J]) : (Rl)(rr - R->dm[J]);
    const Rl s = Rl(1.5852) / dr;
    const Rl s2 = s * s, s4 = s2 * s2, s8 = s4 * s4, s14 = s8 * s4 * s2;
    const Rl F = (Rl)(D ? R->flj_d[J] : R->flj[J]) * (s14 - s8) * dr / rr;
    if (EN) {
        double e;
        if ((double)r2 < R->d2min_d[J]) e = R->elj_d[J] * 1001.0;
        else {
            const Rl s6 = s4 * s2, s12 = s6 * s6;
            e = (double)((Rl)(D ? R->elj_d[J] : R->elj[J]) * (s12 - Rl(2) * s6 + Rl(1)));
        }
        e_excl -= e;
    }
    if (F != Rl(0)) {
        const V3<Rl> g = (Rl(-1) * F) * v;
        A.add(a, g);
        A.add(ex, Rl(-1) * g);
    }
}

template <bool D>
__device__ __forceinline__ Acc<D> force_acc(const Dev &d)
{
    Acc<D> A;
    A.f = (decltype(A.f))d.f;
    A.P = d.P;
    A.err = 0;
    return A;
}

// polymer_constraints (E:2354-2520): bonded term `item`, by one thread
template <bool D, bool EN>
__device__ __forceinline__ void bonded_item(const Dev &d, int item, int excl_in_list)
{
    using Rl = Real<D>;
    const int4 id = d.bt_idx[item];
    const double2 par = d.bt_par[item];
    const int r = d.rep_of[id.x];
    const RepParams *R = d.rp + r;
    const Pos<D> P = make_pos<D>(d, R);
    Acc<D> A = force_acc<D>(d);
    double e_excl = 0;
    const int ex = id.w == 0 ? id.y : id.z;  // excluded pair partner of id.x
    if (id.w == 0) bond_force<D>(P, A, id.x, id.y, (Rl)par.x, (Rl)par.y);
    else angle_force<D>(P, A, id.x, id.y, id.z, (Rl)par.x, (Rl)par.y, false);
    if (!excl_in_list || EN) exclusion_lj<D, EN>(d, R, P, A, id.x, ex, e_excl);
    if (EN) {
        double *e = d.eterm + r * kNE;
        if (id.w == 0) {
            const Rl rr = distance<D>(P, id.x, id.y);
            atomicAdd(e + 3, (double)((Rl)par.x * (rr - (Rl)par.y) * (rr - (Rl)par.y)));
        } else {
            const Rl th = angle_of<D>(P, id.x, id.y, id.z);
            atomicAdd(e + 4, (double)((Rl)par.x * (th - (Rl)par.y) * (th - (Rl)par.y)));
        }
        if (e_excl != 0) atomicAdd(e + 5, e_excl);
    }
    if (A.err) atomicOr(&d.rs[r].err, A.err);
}

// A secondary stack is off this step when a tertiary stack sharing one of its
// sites (ST_EXCESS == 1) is within 10 A of its native distance (E:1960-1981);
// each secondary stack checks the few tertiary stacks that can do that.
template <bool D>
__device__ __forceinline__ bool stack2_off(const Dev &d, const Pos<D> &P, int item)
{
    using Rl = Real<D>;
    for (int u = d.st2_offby_off[item]; u < d.st2_offby_off[item + 1]; ++u) {
        const int k = d.st2_offby_idx[u];
        const int *tid = d.st3_idx + 6 * k;
        if (distance<D>(P, tid[1], tid[4]) - (Rl)d.st3_nat[6 * k] < Rl(10)) return true;
    }
    return false;
}

// Stacks by term (stacking_interactions, E:1911-2141): a unit of 32 stacks is run by one
// warp per term, lane = stack, so that the lanes of a warp evaluate the same kind of term
// and the terms of a stack run side by side: value, exchange through q, force from the
// geometry still in registers.  Measured against one thread per stack, which ran the terms
// and then their forces one after another: 18.2 -> 9.8 us with the bonded terms (5 replicas
// of a 346-nt chain, alone), 80 -> 19 us in FP64 (one 76-nt replica).
// w: the warp's index in its unit (0 .. 7 tertiary: 0 distance, 1-2 angles, 3-5 dihedrals;
// 0 .. 3 secondary: 0 distance, 1-2 dihedrals, 3 the switch); q: 8 (4) x 32 values.
template <bool D, bool EN, class Bar>
__device__ __forceinline__ void stack3_unit(const Dev &d, int unit, int w, int lane, Real<D> *q, Bar bar)
{
    using Rl = Real<D>;
    const int item = unit * 32 + lane;
    const bool on = item < d.nst3 && w < 6;
    const int *id = d.st3_idx + 6 * item;
    const SixBeads n6 = six_beads(w);
    int r = 0;
    BondGeom<D> gb;
    AngleGeom<D> ga;
    DihedralGeom<D> gd;
    Rl nat = Rl(0), val = Rl(0);
    Pos<D> P;
    if (on) {
        r = d.rep_of[id[0]];
        P = make_pos<D>(d, d.rp + r);
        nat = (Rl)d.st3_nat[6 * item + w];
        if (w == 0) {
            gb = bond_geom<D>(P, id[1], id[4]);
            const Rl rdev = gb.r - nat;
            val = Rl(5) * rdev * rdev;
        } else if (w <= 2) {
            ga = angle_geom<D>(P, id[n6.a], id[n6.b], id[n6.c]);
            val = Rl(1.5) * (ga.th - nat) * (ga.th - nat);
        } else {
            gd = dihedral_geom<D>(P, id[n6.a], id[n6.b], id[n6.c], id[n6.d]);
            nat = psi_shift<Rl>(nat, psi_branch<Rl>(gd.psi, nat));
            val = Rl(0.15) * (gd.psi - nat) * (gd.psi - nat);
        }
        q[w * 32 + lane] = val;
    }
    bar();
    if (on) {
        Rl Dn = Rl(1);
        for (int s = 0; s < 6; ++s) Dn += q[s * 32 + lane];
        const Rl E = (Rl)d.st3_E[item] / Dn, wt = -E / Dn;
        Acc<D> A = force_acc<D>(d);
        if (w == 0) {
            bond_apply<D>(gb, A, id[1], id[4], Rl(5) * wt, nat);
            d.st_energy[item] = (double)E;
            atomicAdd(EN ? d.eterm + r * kNE + 7 : &d.rs[r].e3st_acc, (double)E);
        } else if (w <= 2) {
            angle_apply<D>(ga, A, id[n6.a], id[n6.b], id[n6.c], Rl(1.5) * wt, nat, true);
        } else {
            dihedral_apply<D>(gd, A, id[n6.a], id[n6.b], id[n6.c], id[n6.d], Rl(0.15) * wt, nat);
        }
        if (A.err) atomicOr(&d.rs[r].err, A.err);
    }
}

template <bool D, bool EN, class Bar>
__device__ __forceinline__ void stack2_unit(const Dev &d, int unit, int w, int lane, Real<D> *q, Bar bar)
{
    using Rl = Real<D>;
    const int item = unit * 32 + lane;
    const bool on = item < d.nst2;
    const int *id = d.st2_idx + 7 * item;  // k_10 k00 k01 k10 k20 k21 k30
    int r = 0;
    BondGeom<D> gb;
    DihedralGeom<D> gd;
    Rl nat = Rl(0), val = Rl(0);
    if (on) {
        r = d.rep_of[id[0]];
        const Pos<D> P = make_pos<D>(d, d.rp + r);
        if (w == 0) {
            gb = bond_geom<D>(P, id[2], id[5]);
            nat = (Rl)d.st2_r0[item];
            val = Rl(1.4) * (gb.r - nat) * (gb.r - nat);
        } else if (w <= 2) {
            gd = dihedral_geom<D>(P, id[w == 1 ? 0 : 6], id[w == 1 ? 1 : 4], id[3], id[w == 1 ? 4 : 1]);
            nat = w == 1 ? Rl(-2.58684) : Rl(3.07135);
            nat = psi_shift<Rl>(nat, psi_branch<Rl>(gd.psi, nat));
            val = Rl(4) * (gd.psi - nat) * (gd.psi - nat);
        } else {
            val = stack2_off<D>(d, P, item) ? Rl(1) : Rl(0);
        }
        q[w * 32 + lane] = val;
    }
    bar();
    if (on && w < 3 && q[3 * 32 + lane] == Rl(0)) {
        Rl Dn = Rl(1) + q[lane];
        Dn += q[32 + lane];
        Dn += q[64 + lane];
        const Rl E = (Rl)d.st2_E[item] / Dn, wt = -E / Dn;
        Acc<D> A = force_acc<D>(d);
        if (w == 0) {
            bond_apply<D>(gb, A, id[2], id[5], Rl(1.4) * wt, nat);
            atomicAdd(EN ? d.eterm + r * kNE + 6 : &d.rs[r].e2st_acc, (double)E);
        } else {
            dihedral_apply<D>(gd, A, id[w == 1 ? 0 : 6], id[w == 1 ? 1 : 4], id[3], id[w == 1 ? 4 : 1], Rl(4) * wt, nat);
        }
        if (A.err) atomicOr(&d.rs[r].err, A.err);
    }
}

// item t of the handle's bonded terms, tertiary and secondary stacks, by one thread (the
// fused step kernel's form)
template <bool D>
__device__ __forceinline__ void topo_item(const Dev &d, int t)
{
    using Rl = Real<D>;
    if (t < d.nbt) {
        bonded_item<D, false>(d, t, 1);
        return;
    }
    const bool tert = t < d.nbt + d.nst3;
    const int item = tert ? t - d.nbt : t - d.nbt - d.nst3;
    const int *id = tert ? d.st3_idx + 6 * item : d.st2_idx + 7 * item;
    const int r = d.rep_of[id[0]];
    const Pos<D> P = make_pos<D>(d, d.rp + r);
    Acc<D> A = force_acc<D>(d);
    if (tert) {
        const double *nat = d.st3_nat + 6 * item;
        const Rl rdev = distance<D>(P, id[1], id[4]) - (Rl)nat[0];
        int code;
        const Rl Dn = six_q<D>(P, id, nat, rdev, Rl(1), code);
        const Rl E = (Rl)d.st3_E[item] / Dn;
        six_force<D>(P, A, id, nat, code, -E / Dn);
        d.st_energy[item] = (double)E;
        atomicAdd(&d.rs[r].e3st_acc, (double)E);
    } else {
        if (stack2_off<D>(d, P, item)) return;
        const Rl rr = distance<D>(P, id[2], id[5]);
        const Rl p1 = dihedral_of<D>(P, id[0], id[1], id[3], id[4]);
        const Rl p2 = dihedral_of<D>(P, id[6], id[4], id[3], id[1]);
        const Rl p10 = psi_shift<Rl>(Rl(-2.58684), psi_branch<Rl>(p1, Rl(-2.58684)));
        const Rl p20 = psi_shift<Rl>(Rl(3.07135), psi_branch<Rl>(p2, Rl(3.07135)));
        const Rl r0 = (Rl)d.st2_r0[item];
        Rl Dn = Rl(1) + Rl(1.4) * (rr - r0) * (rr - r0);
        Dn += Rl(4) * (p1 - p10) * (p1 - p10);
        Dn += Rl(4) * (p2 - p20) * (p2 - p20);
        const Rl E = (Rl)d.st2_E[item] / Dn;
        const Rl w = -E / Dn;
        bond_force<D>(P, A, id[2], id[5], Rl(1.4) * w, r0);
        dihedral_force<D>(P, A, id[0], id[1], id[3], id[4], Rl(4) * w, p10);
        dihedral_force<D>(P, A, id[6], id[4], id[3], id[1], Rl(4) * w, p20);
        atomicAdd(&d.rs[r].e2st_acc, (double)E);
    }
    if (A.err) atomicOr(&d.rs[r].err, A.err);
}

// Block b of the topology blocks (topo_plan): units of tertiary stacks (two per block of
// kForceThreads), units of secondary stacks (four per block), bonded terms, then the
// Gaussian pairs of every replica (noise: 1500 and kNoiseSpare / 2 more each, from the
// replica's draw counter on; the H-bond Monte Carlo's draws of the step come first, so
// the step's Gaussians start as many draws later in this table).
template <bool D, bool EN>
__device__ __forceinline__ void topo_block(const Dev &d, const TopoPlan &tp, int b, int mask, int excl_in_list,
                                           Real<D> *q /* 16 x 32 */)
{
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    if (b < tp.n3) {
        if (mask & 8) stack3_unit<D, EN>(d, 2 * b + (w >> 3), w & 7, lane, q + (w >> 3) * 8 * 32, NamedBar{1 + (w >> 3), 256});
        return;
    }
    b -= tp.n3;
    if (b < tp.n2) {
        if (mask & 8) stack2_unit<D, EN>(d, 4 * b + (w >> 2), w & 3, lane, q + (w >> 2) * 4 * 32, NamedBar{1 + (w >> 2), 128});
        return;
    }
    b -= tp.n2;
    if (b < tp.nb) {
        const int item = b * tp.per + tid;
        if ((mask & 4) && tid < tp.per && item < d.nbt) bonded_item<D, EN>(d, item, excl_in_list);
        return;
    }
    b -= tp.nb;
    constexpr int kPairs = (kNoise + kNoiseSpare) / 2, kPer = noise_blocks(kPairs);
    const int item = b * tp.per + tid;
    if (tid < tp.per && item < d.R * kPer) {
        const int r = item / kPer;
        noise_block<D>(d.rp[r].seed, d.rs[r].ctr, kPairs, item - r * kPer, d.gnoise + (size_t)r * kNoiseStride);
    }
}

template <bool D, bool EN>
__global__ void __launch_bounds__(kForceThreads) k_topo(Dev d, TopoPlan tp, int mask, int excl_in_list)
{
    __shared__ Real<D> s_q[16 * 32];
    topo_block<D, EN>(d, tp, blockIdx.x, mask, excl_in_list, s_q);
}

__device__ __forceinline__ unsigned long long global_ns_hb()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------
// hydrogen bonds of one replica per block: energies, the valence-limited Monte
// Carlo, forces; then (fused step) this step's Gaussians
// ---------------------------------------------------------------------------
// Working arrays of one replica's H-bonds, indexed by the replica's local bond
// and over-valence atom numbers: in shared memory when they fit (Dev::hb_smem),
// else in global scratch.  status starts as the list build left it (0: live,
// -1: out of range) and every live bond is back to 0 when the kernel ends, so
// the shared copy is never written back.
template <bool D>
struct HbWork {
    Real<D> *en;   // energy of each live bond this step
    Real<D> *term; // its six restraint terms (six per bond)
    int *st;       // status: 0 formed, 1 broken this step, -1 out of range
    signed char *br;  // per bond: the imaging branches of its three dihedrals; 1 when its distance breaks it
    int *exc;      // excess valence of each over-valence atom
    int *al;       // a bit per over-valence atom: positive excess (the reference's A list)
    int *kl;       // candidate bonds of the chosen atom (the reference's K list)
    const int *ca_off, *ca_idx;  // candidates of each over-valence atom: ca_idx[ca_off[i] ..]
    const int *hb_off, *hb_pos;  // over-valence atoms of each bond: hb_pos[hb_off[k] ..]
};

constexpr int kHbThreads = 512;

// n ints to shared memory by bd threads, landing by copy_async_wait
__device__ __forceinline__ void copy_async(int *dst, const int *src, int n, int tid, int bd)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    for (int i = tid; i < n; i += bd)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s + 4u * (unsigned)i), "l"(src + i) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// rand() draws vbase .. vbase + 63 of a replica into v[], by 17 lanes of one warp
// (one Philox block of four draws each; the same words rand_value returns)
__device__ inline void fill_draws(uint32_t *v, unsigned long long seed, unsigned long long vbase, int lane)
{
    const unsigned long long b = (vbase >> 2) + (unsigned long long)lane;
    if (lane < 17) {
        uint32_t c[4] = {(uint32_t)b, (uint32_t)(b >> 32), 0u, 0u};
        philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
        for (int w = 0; w < 4; ++w) {
            const long long idx = (long long)(4 * b + (unsigned long long)w) - (long long)vbase;
            if (idx >= 0 && idx < 64) {
                const uint32_t x = c[w] >> 1;
                v[idx] = x ? x : 1u;
            }
        }
    }
    __syncwarp();
}

// One block per replica.  The restraint energies and forces of the live bonds run
// as (chunk of 32 bonds, term) warp tasks, so that the lanes of a warp evaluate
// the same term; the Monte Carlo runs on one warp.  make_noise: 1 the block then draws the
// step's Gaussians itself; 2 they are being made beside it (topo_block), and the Monte
// Carlo's draw count is left for control_step to book with them.
template <bool D, bool EN, class Bar>
__device__ __forceinline__ void hbond_block(const Dev &d, int r, int do_hb, int make_noise, int tid, int bd, Bar bar)
{
    using Rl = Real<D>;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ uint32_t s_v[64];  // draws vbase .. vbase + 63 of the replica's rand() stream
    __shared__ unsigned long long s_ctr;
    const RepParams *R = d.rp + r;
    RepState *S = d.rs + r;
    const Pos<D> P = make_pos<D>(d, R);
    Acc<D> A = force_acc<D>(d);
    const unsigned long long c0 = S->ctr;
    double e2hb = 0, e3hb = 0;
    const int hb0 = R->hb0, nhb = R->hb1 - R->hb0, ca0 = R->ca0, nca = R->ca1 - R->ca0;
    const int warp = tid >> 5, nwarp = bd >> 5, lane = tid & 31;
    // sub-phase times of the fused kernel's phase timer (tis_profile_fused), by tid 0
    unsigned long long *prof = (d.fprof && tid == 0) ? d.fprof + (size_t)r * kFusedPhases : nullptr;
    unsigned long long tlap = prof ? global_ns_hb() : 0ull;
    auto lap = [&](int k) {
        if (prof) {
            const unsigned long long t = global_ns_hb();
            atomicAdd(prof + k, t - tlap);
            tlap = t;
        }
    };
    HbWork<D> w;
    const int nact = do_hb ? S->n_active : 0;

    // ---- hydrogen_bonds_interactions (E:2145-2350) ----
    if (do_hb) {
        const int c_base = d.ca_coff[ca0], n_cidx = d.ca_coff[R->ca1] - c_base;
        const int h_base = d.hb_coff[hb0], n_cpos = d.hb_coff[R->hb1] - h_base;
        int off_c = 0, off_h = 0;  // what the offsets below start from
        if (d.hb_smem) {
            const HbLayout L = hb_layout(d.hb_nmax, d.ca_nmax, d.k_nmax, d.cidx_max, d.cpos_max, D);
            w.en = (Rl *)(s_dyn + L.en);
            w.term = (Rl *)(s_dyn + L.term);
            w.st = (int *)(s_dyn + L.st);
            w.br = (signed char *)(s_dyn + L.br);
            w.exc = (int *)(s_dyn + L.exc);
            w.al = (int *)(s_dyn + L.al);
            w.kl = (int *)(s_dyn + L.kl);
            int *cao = (int *)(s_dyn + L.ca_off), *cai = (int *)(s_dyn + L.ca_idx);
            int *hbo = (int *)(s_dyn + L.hb_off), *hbp = (int *)(s_dyn + L.hb_pos);
            // the replica's tables travel to shared memory while the terms are evaluated
            copy_async(w.st, d.hb_status + hb0, nhb, tid, bd);
            copy_async(cao, d.ca_coff + ca0, nca + 1, tid, bd);
            copy_async(cai, d.ca_cidx + c_base, n_cidx, tid, bd);
            copy_async(hbo, d.hb_coff + hb0, nhb + 1, tid, bd);
            copy_async(hbp, d.hb_cpos + h_base, n_cpos, tid, bd);
            off_c = c_base;
            off_h = h_base;
            w.ca_off = cao; w.ca_idx = cai; w.hb_off = hbo; w.hb_pos = hbp;
        } else {
            w.en = (Rl *)(d.hb_energy + hb0);
            w.term = (Rl *)(d.hb_term + 6 * (size_t)hb0);
            w.st = d.hb_status + hb0;
            w.br = (signed char *)(d.hb_code + hb0);
            w.exc = d.ca_exc + ca0;
            w.al = d.hb_A + ca0;
            w.kl = d.hb_K + R->kscr0;
            w.ca_off = d.ca_coff + ca0; w.ca_idx = d.ca_cidx;
            w.hb_off = d.hb_coff + hb0; w.hb_pos = d.hb_cpos;
        }
        for (int i = tid; i < nca; i += bd) w.exc[i] = d.hb_excess[d.ca_list[ca0 + i]];
        // the restraint terms: warp task (chunk of 32 live bonds, term 0..5)
        const int nchunk = (nact + 31) >> 5;
        for (int task = warp; task < 6 * nchunk; task += nwarp) {
            const int s = task % 6, t = (task / 6) * 32 + lane;
            if (t < nact) {
                const int k = d.hb_active[hb0 + t], kl = k - hb0;
                int br;
                Rl rdev = Rl(0);
                if (s == 0) {
                    rdev = distance<D>(P, d.hb_idx[6 * k + 1], d.hb_idx[6 * k + 4]) - (Rl)d.hb_nat[6 * k];
                    w.br[4 * kl + 3] = fabs(rdev) > Rl(2);
                }
                w.term[6 * kl + s] = six_term<D>(P, d.hb_idx + 6 * k, d.hb_nat + 6 * k, s, rdev, br);
                if (s >= 3) w.br[4 * kl + s - 3] = (signed char)br;
            }
        }
        copy_async_wait();
        bar();
        for (int t = tid; t < nact; t += bd) {
            const int k = d.hb_active[hb0 + t], kl = k - hb0;
            if (w.br[4 * kl + 3]) {  // a live bond whose central distance strays more than 2 A from native breaks (E:2165-2175)
                w.st[kl] = 1;
                for (int u = w.hb_off[kl] - off_h; u < w.hb_off[kl + 1] - off_h; ++u) atomicSub(w.exc + w.hb_pos[u], 1);
                w.en[kl] = Rl(0);
                continue;
            }
            Rl q = Rl(0);
            for (int s = 0; s < 6; ++s) q += w.term[6 * kl + s];
            w.en[kl] = (Rl)d.hb_E[k] * exp_(-q);
        }
        bar();
        lap(8);
        if (tid < 32) {  // valence-limited Monte Carlo (E:2239-2315), one warp
            const unsigned lt = (1u << lane) - 1u;
            unsigned long long ctr = c0, vbase = ctr;
            bool filled = false;
            const double T = R->T;
            const float inv_t = 1.0f / R->Tf;
            // A: atoms with positive excess, in atom order: a bit each, kept up as they lose it
            const int nword = (nca + 31) >> 5;
            int nA = 0;
            for (int v = 0; v < nword; ++v) {
                const int i = 32 * v + lane;
                const unsigned m = __ballot_sync(kFull, i < nca && w.exc[i] > 0);
                if (lane == 0) w.al[v] = (int)m;
                nA += __popc(m);
            }
            __syncwarp();
            int guard = nact + 2;
            while (nA > 0 && guard-- > 0) {
                // draws ctr, ctr+1, ...: the atom, the K shuffle, the acceptances; u[i] is draw ctr + i
                if (!filled || ctr - vbase > 32) {
                    vbase = ctr;
                    fill_draws(s_v, R->seed, vbase, lane);
                    filled = true;
                }
                const uint32_t *u = s_v + (ctr - vbase);
                const int nu = 64 - (int)(ctr - vbase);  // draws held from u[0] on (at least 32)
                int nth = pick_index(u[0], nA), atom = 0;
                for (int v0 = 0; v0 < nword; v0 += 32) {  // the nth set bit
                    const unsigned m = v0 + lane < nword ? (unsigned)w.al[v0 + lane] : 0u;
                    const int c = __popc(m);
                    int incl = c;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(kFull, incl, o);
                        if (lane >= o) incl += t;
                    }
                    const unsigned at = __ballot_sync(kFull, incl >= nth);
                    if (at) {
                        const int src = __ffs((int)at) - 1;
                        unsigned mm = __shfl_sync(kFull, m, src);
                        for (int i = nth - __shfl_sync(kFull, incl - c, src); i > 1; --i) mm &= mm - 1u;
                        atom = 32 * (v0 + src) + __ffs((int)mm) - 1;
                        break;
                    }
                    nth -= __shfl_sync(kFull, incl, 31);
                }
                // K: the atom's candidates still formed, in candidate order
                const int k0 = w.ca_off[atom] - off_c, nc = w.ca_off[atom + 1] - off_c - k0;
                int nK = 0;
                for (int base = 0; base < nc; base += 32) {
                    const int t = base + lane;
                    const int k = t < nc ? w.ca_idx[k0 + t] : 0;
                    const bool ok = t < nc && w.st[k] == 0;
                    const unsigned m = __ballot_sync(kFull, ok);
                    if (ok) w.kl[nK + __popc(m & lt)] = k;
                    nK += __popc(m);
                }
                __syncwarp();
                if (nK == 0) {
                    ctr += 1;
                    A.err |= kErrRange;
                    break;
                }
                int chosen;
                if (nK * nK <= 32) {
                    // lane l holds entry l of the list; the swaps in draw order
                    int kl = w.kl[min(lane, nK - 1)];
                    const int jj = pick_index(u[min(lane + 1, nK)], nK) - 1;
                    for (int i = 0; i < nK; ++i) {
                        const int J = __shfl_sync(kFull, jj, i), ka = __shfl_sync(kFull, kl, i), kb = __shfl_sync(kFull, kl, J);
                        kl = lane == i ? kb : lane == J ? ka : kl;
                    }
                    // Metropolis walk over the shuffled K (draws nK+1 .. 2nK-1): lane a*nK+b
                    // decides whether candidate a replaces candidate b
                    const Rl en = w.en[kl];
                    const int a = lane / nK, b = lane - a * nK;
                    const Rl ea = __shfl_sync(kFull, en, a), eb = __shfl_sync(kFull, en, b);
                    const bool acc = lane < nK * nK && a >= 1 && accept_move(u[nK + a], ea, eb, T, inv_t);
                    const unsigned dm = __ballot_sync(kFull, acc);
                    int kc = 0;
                    for (int a2 = 1; a2 < nK; ++a2)
                        if ((dm >> (a2 * nK + kc)) & 1u) kc = a2;
                    chosen = __shfl_sync(kFull, kl, kc);
                } else {
                    int kc = 0;
                    if (lane == 0) {
                        for (int i = 1; i <= nK; ++i) {
                            const int jj = pick_index(i < nu ? u[i] : rand_value(R->seed, ctr + i), nK);
                            const int tmp = w.kl[i - 1];
                            w.kl[i - 1] = w.kl[jj - 1];
                            w.kl[jj - 1] = tmp;
                        }
                        for (int i = 2; i <= nK; ++i) {
                            const int di = nK + i - 1;
                            const uint32_t v = di < nu ? u[di] : rand_value(R->seed, ctr + di);
                            if (accept_move(v, w.en[w.kl[i - 1]], w.en[w.kl[kc]], T, inv_t)) kc = i - 1;
                        }
                        kc = w.kl[kc];
                    }
                    chosen = __shfl_sync(kFull, kc, 0);
                }
                if (lane == 0) w.st[chosen] = 1;
                const int h0 = w.hb_off[chosen] - off_h, nh = w.hb_off[chosen + 1] - off_h - h0;
                for (int t0 = 0; t0 < nh; t0 += 32) {
                    bool gone = false;
                    if (t0 + lane < nh) {
                        const int i = w.hb_pos[h0 + t0 + lane];
                        gone = atomicSub(w.exc + i, 1) == 1;
                        if (gone) atomicAnd(w.al + (i >> 5), ~(1 << (i & 31)));
                    }
                    nA -= __popc(__ballot_sync(kFull, gone));
                }
                ctr += 2 * nK;
                __syncwarp();
            }
            if (lane == 0) s_ctr = ctr;
        }
        bar();
        lap(9);
        if (warp == nwarp - 1) {  // the energies
            for (int t = lane; t < nact; t += 32) {
                const int k = d.hb_active[hb0 + t], kl = k - hb0;
                if (w.st[kl] != 1) {
                    if (d.hb_dode[k]) e3hb += (double)w.en[kl];
                    else e2hb += (double)w.en[kl];
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                e2hb += __shfl_down_sync(kFull, e2hb, o);
                e3hb += __shfl_down_sync(kFull, e3hb, o);
            }
            if (lane == 0) {
                S->e2hb = e2hb;
                S->e3hb = e3hb;
                if (EN) {
                    double *e = d.eterm + r * kNE;
                    e[8] += e2hb; e[9] += e3hb;
                }
            }
        }
        // forces of the bonds still formed: warp task (chunk of 32 live bonds, term 0..5)
        for (int task = warp; task < 6 * nchunk; task += nwarp) {
            const int s = task % 6, t = (task / 6) * 32 + lane;
            if (t < nact) {
                const int k = d.hb_active[hb0 + t], kl = k - hb0;
                if (w.st[kl] != 1) {
                    const Rl wk = -(Rl)w.en[kl];
                    six_force_term<D>(P, A, d.hb_idx + 6 * k, d.hb_nat + 6 * k, s >= 3 ? w.br[4 * kl + s - 3] : 0, wk, s);
                }
            }
        }
    }
    if (do_hb && d.hb_rec)  // the bonds formed after the Monte Carlo (status 0; 1 broken, -1 out of range)
        for (int i = tid; i < nhb; i += bd) d.hb_rec[hb0 + i] = w.st[i] == 0 ? 1 : 0;
    lap(10);
    // ---- full_forces: the step's Gaussians follow the Monte Carlo draws ----
    const unsigned long long c1 = do_hb ? s_ctr : c0;
    double *noise = d.gnoise + (size_t)r * kNoiseStride;
    if (make_noise == 1) gen_noise<D>(d, r, c1, noise, tid, bd);
    if (make_noise == 2 && c1 - c0 > (unsigned long long)kNoiseSpare)  // past the table's end: all of them here
        gen_noise<D>(d, r, c1, noise + kNoise + kNoiseSpare, tid, bd);
    if (d.fprof) {  // the Gaussians of every thread are done (timer runs only)
        bar();
        lap(11);
    }

    if (do_hb && !d.hb_smem) {
        bar();  // every warp has read the statuses
        for (int t = tid; t < nact; t += bd) {  // every live bond is formed again for the next step
            const int kl = d.hb_active[hb0 + t] - hb0;
            if (w.st[kl] == 1) w.st[kl] = 0;
        }
    }
    if (tid == 0) {
        if (make_noise == 2) S->pending = 1u + (unsigned)(c1 - c0);
        else S->ctr = make_noise ? c1 + kNoise : c1;
    }
    if (A.err) atomicOr(&S->err, A.err);
}

template <bool D, bool EN>
__global__ void __launch_bounds__(kHbThreads) k_hbond(Dev d, int do_hb, int make_noise)
{
    hbond_block<D, EN>(d, blockIdx.x, do_hb, make_noise, (int)threadIdx.x, (int)blockDim.x, CtaBar{});
}

// deterministic_forces_MPI (E:2524-2586) with the step's Gaussians, of every replica of the
// group in one launch: blocks [0, R) the H-bonds of a replica each (the longest chain, so
// first), then the topology blocks, then the pairs, kForceThreads / TS sub-blocks of PB
// particles per block.
// One launch instead of four on forked streams and one for the shift: a step is a chain of
// kernels of a few microseconds, so each launch, fork and join in it counts (step of one
// 346-nt replica 32.1 -> 24.7 us, of one 76-nt replica in FP64 96 -> 35 us), and an LR launch
// with nothing due waited for room beside the other groups' work (64 replicas: 114 -> 107 us).
// Blocks end without a word to one another: a count of ended blocks, whose last one formed
// the recentring shift here, held every block for its fence (the integrator forms it now).
// Two blocks of 512 threads per SM; FP64 needs the registers of one.
template <bool D, int PB, int TS>
__global__ void __launch_bounds__(kForceThreads, D ? 1 : 2) k_forces(Dev d, TopoPlan tp, int noise)
{
    wait_prior_grid();
    extern __shared__ __align__(16) unsigned char s_dyn[];
    const int tid = threadIdx.x;
    int b = blockIdx.x;
    if (b < d.R) {
        hbond_block<D, false>(d, b, 1, noise ? 2 : 0, tid, kForceThreads, CtaBar{});
    } else if ((b -= d.R) < tp.blocks()) {
        topo_block<D, false>(d, tp, b, 4 | 8, 1, (Real<D> *)s_dyn);
    } else {
        constexpr int kSub = kForceThreads / TS;
        const int sub = tid / TS, pb = (b - tp.blocks()) * kSub + sub;
        if (pb * PB < d.P)
            pair_tasks<D, false, true, PB, TS>(d, pb, 1, 1, tid - sub * TS, ((PairSmem<D, PB> *)s_dyn)[sub],
                                               NamedBar{1 + sub, TS});
    }
}

__device__ void control_step(const Dev &d, int r);

// x < 0 and x > L (L > 0) on the bit patterns, as IEEE comparisons decide them for
// finite x (-0.0 is not below zero): integer instructions instead of FP64 compares
__device__ inline bool below_zero(double x)
{
    const long long b = __double_as_longlong(x);
    return b < 0 && b != (long long)0x8000000000000000ull;
}
__device__ inline bool above(double x, double L) { return __double_as_longlong(x) > __double_as_longlong(L); }

// |x| < 2^20 and finite, from the exponent field
__device__ inline bool bounded(double x)
{
    return ((unsigned)(__double_as_longlong(x) >> 52) & 0x7ffu) < 1023u + 20u;
}

// The five Energies-file values of replica r (E:6308-6312: E2_HB, E3_HB, E2_STACK,
// E3_STACK of the last step, Rg of the RNA at the current positions) into out[0..4],
// by threads tid = 0 .. nthr-1 (written by tid 0)
template <class Bar>
__device__ void energies_block(const Dev &d, int r, double *out, int tid, int nthr, Bar bar)
{
    const RepParams *R = d.rp + r;
    __shared__ double s_red[3 * 32];
    __shared__ double s_c[3];
    double c[3] = {0, 0, 0};
    for (int i = tid; i < R->nrna; i += nthr) {
        c[0] += d.x[R->p0 + i];
        c[1] += d.y[R->p0 + i];
        c[2] += d.z[R->p0 + i];
    }
    block_sum_t<3>(c, s_red, tid, nthr, bar);
    if (tid == 0)
        for (int k = 0; k < 3; ++k) s_c[k] = c[k] / R->nrna;
    bar();
    double sq[1] = {0};
    for (int i = tid; i < R->nrna; i += nthr) {
        const double a = d.x[R->p0 + i] - s_c[0], b = d.y[R->p0 + i] - s_c[1], e = d.z[R->p0 + i] - s_c[2];
        sq[0] += a * a + b * b + e * e;
    }
    block_sum_t<1>(sq, s_red, tid, nthr, bar);
    if (tid == 0) {
        const RepState *S = d.rs + r;
        out[0] = S->e2hb;
        out[1] = S->e3hb;
        out[2] = S->e2st;
        out[3] = S->e3st;
        out[4] = sqrt(sq[0] / R->nrna);
    }
}

// The frame of replica r after step klok into its slot of the frame ring (d.fr),
// by threads tid = 0 .. nthr-1 of one block: positions, then the five energies,
// then, after a system-scope fence, the step number that marks the slot complete.
template <class Bar>
__device__ void write_frame(const Dev &d, int r, long long klok, int tid, int nthr, Bar bar)
{
    const FrameRing &F = d.fr;
    const RepParams *R = d.rp + r;
    const long long slot = (klok / F.every) % F.depth;
    const long long base = F.pk_base + R->pk0;
    double *px = F.pos + slot * 3 * F.n_total;
    for (int i = tid; i < R->n; i += nthr) {
        px[base + i] = d.x[R->p0 + i];
        px[F.n_total + base + i] = d.y[R->p0 + i];
        px[2 * F.n_total + base + i] = d.z[R->p0 + i];
    }
    __shared__ double s_e5[5];
    energies_block(d, r, s_e5, tid, nthr, bar);
    bar();
    if (tid < 5) F.en[(slot * F.R_total + F.rep_base + r) * 5 + tid] = s_e5[tid];
    __threadfence_system();
    bar();
    if (tid == 0) {
        __threadfence_system();
        *(volatile long long *)(F.done + slot * F.R_total + F.rep_base + r) = klok;
    }
}

// move_rigid_units for particle p of replica r after its leap-frog (xn, vn; the recentring
// shift sh, the ions' periodic wrap, the new fixed-point position,
// its force sum zeroed); xo: its old position, moved alike.  The centre bead's new state goes to `hold` when given
// (a replica's place in Dev::centre) instead of the arrays, from which other blocks still
// form the shift.
template <bool D, bool I>
__device__ __forceinline__ void move_particle(const Dev &d, const RepParams *R, int p, int4 q, const Shift<I> &sh,
                                              double xn[3], const double vn[3], double xo[3], double *hold, int &err)
{
    xo[0] = d.x[p];
    xo[1] = d.y[p];
    xo[2] = d.z[p];
    for (int c = 0; c < 3; ++c) {
        xn[c] = axis_add<I>(R, c, xn[c], sh);
        xo[c] = axis_add<I>(R, c, xo[c], sh);
    }
    if (p - R->p0 >= R->nrna) {  // periodic wrap of the ions (E:2676-2731)
        for (int c = 0; c < 3; ++c) {
            if (below_zero(xn[c])) { xn[c] += R->box[c]; xo[c] += R->box[c]; }
            if (above(xn[c], R->box[c])) { xn[c] -= R->box[c]; xo[c] -= R->box[c]; }
        }
    }
    // a runaway or non-finite particle (|x| or |v| component >= 2^20) stops the run
    bool ok = true;
    for (int c = 0; c < 3; ++c) ok = ok && bounded(xn[c]) && bounded(vn[c]);
    if (!ok) err |= kErrNonFinite;
    q.x = fix_position(R, 0, xn[0]);
    q.y = fix_position(R, 1, xn[1]);
    q.z = fix_position(R, 2, xn[2]);
    if (hold && p == R->center) {
        for (int c = 0; c < 3; ++c) {
            hold[c] = xn[c];
            hold[3 + c] = xo[c];
            hold[6 + c] = vn[c];
        }
        *(int4 *)(hold + 10) = q;
        return;
    }
    d.x[p] = xn[0]; d.y[p] = xn[1]; d.z[p] = xn[2];
    d.xo[p] = xo[0]; d.yo[p] = xo[1]; d.zo[p] = xo[2];
    d.vx[p] = vn[0]; d.vy[p] = vn[1]; d.vz[p] = vn[2];
    d.f[p] = 0ull;  // consumed: the next step's force kernels accumulate from zero
    d.f[d.P + p] = 0ull;
    d.f[2 * d.P + p] = 0ull;
    d.q[p] = q;
}

// the centre bead's held state into the arrays, by one thread, once every block has read them
__device__ __forceinline__ void release_centre(const Dev &d, const RepParams *R, const double *hold)
{
    const int p = R->center;
    double v[9];
    for (int c = 0; c < 9; ++c) v[c] = __ldcg(hold + c);
    const int4 q = __ldcg((const int4 *)(hold + 10));
    d.x[p] = v[0]; d.y[p] = v[1]; d.z[p] = v[2];
    d.xo[p] = v[3]; d.yo[p] = v[4]; d.zo[p] = v[5];
    d.vx[p] = v[6]; d.vy[p] = v[7]; d.vz[p] = v[8];
    d.f[p] = 0ull;
    d.f[d.P + p] = 0ull;
    d.f[2 * d.P + p] = 0ull;
    d.q[p] = q;
}

// component c of the recentring shift of adjust_box (E:2632-2656), the centre bead's new
// position moved to the box centre, by lane c of three (all lanes of the warp call): the
// leap-frog of leap_frog with a lane per component, so that a warp issues a third of it
template <bool D>
__device__ __forceinline__ double shift_lane(const Dev &d, const RepParams *R, int r, int lane)
{
    const int c = min(lane, 2), p = R->center, P = d.P;
    const int t = d.q[p].w & 0xff, k = (p - R->p0 + 1) % 1000;
    const double *xs = c == 0 ? d.x : c == 1 ? d.y : d.z, *os = c == 0 ? d.xo : c == 1 ? d.yo : d.zo,
                 *vs = c == 0 ? d.vx : c == 1 ? d.vy : d.vz;
    const double x0 = xs[p], o0 = os[p], v0 = vs[p], g = step_noise(d, r)[k + 1000 * c];
    double vn, xn;
    if (D) {
        double f = total_force<D>(d, p, c);
        if (d.noise == 0) f = __dadd_rn(f, __dmul_rn(g, R->sigma[t]));
        vn = __dadd_rn(__dmul_rn(R->k1[t], v0), __dmul_rn(R->k2[t], f));
    } else {
        const double kg = d.noise == 0 ? R->k2sig[t] : 0.0;
        const long long fx = (long long)(__ldcg(d.f + c * P + p) + __ldcg(d.flr + c * P + p));
        vn = fma(kg, g, fma(R->k2fix[t], fix_to_double(fx), R->k1[t] * v0));
    }
    const int hv = __reduce_max_sync(kFull, __double2hiint(vn) & 0x7fffffff);
    if (hv >= R->vcut[t]) {
        const double v[3] = {__shfl_sync(kFull, vn, 0), __shfl_sync(kFull, vn, 1), __shfl_sync(kFull, vn, 2)};
        double vsq = R->vcap[t] * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        if (vsq > 1.0) {
            vsq = 1.0 / sqrt(vsq);
            vn *= vsq;
        }
    }
    if (D) xn = __dadd_rn(__dsub_rn(__dmul_rn(2.0, x0), o0), __dmul_rn(__dsub_rn(vn, v0), R->h));
    else xn = fma(vn - v0, R->h, x0 + (x0 - o0));
    return R->hbox[c] - xn;
}

// |xn - xo|^2 as a bit pattern (non-negative doubles order as integers)
__device__ __forceinline__ unsigned long long shift_bits(const double xn[3], const double xo[3])
{
    double e2 = 0.0;
    for (int c = 0; c < 3; ++c) {
        const double e = xn[c] - xo[c];
        e2 += e * e;
    }
    return (unsigned long long)__double_as_longlong(e2);
}

// move_rigid_units (E:2660-2731) of one particle per thread, T threads per block: leap-frog,
// the recentring shift, which a warp of every block forms from the centre bead, the
// periodic wrap of the ions.  The centre bead's new state and the skin check wait until every
// block is done: the cell kernel begins with them in a step (k_cells); with `tail` (the
// drop-in routine, after which a caller may look at anything) the replica's last block to
// finish does both.  A count of finished blocks in every step held each block for a fence, an
// atomic and two barriers: step of one 346-nt replica 19.2 -> 18.0 us, of 7 replicas of 203 nt
// 31.6 -> 30.6 us, of 64 replicas 84.6 -> 83.8 us.
// Bound by the FP64 pipe (a warp instruction takes it 16 cycles or more, 64 issue slots):
// everything but the update itself runs on integers or FP32.  Of the largest
// displacement, which check_shifts needs exactly, an FP32 estimate finds the block's
// candidates and only those form it in FP64.  Measured (one launch for all replicas): 64
// replicas, 344,903 particles, 51.3 -> 38.9 us; 16 replicas, 782,384 particles, 96 -> 70 us.
// Handles of few particles for the GPU (Dev::wide) take blocks of 64 threads, so that the
// FP64 work spreads over more SMs; with more they would only add blocks to schedule.
// The shift costs a block a twelfth of its FP64 work and the centre bead a detour through
// Dev::centre; formed at the end of the force launch it held that launch's blocks for a
// fence and an atomic: step of 64 replicas 95.3 -> 92.7 us, of one 23.7 -> 21.4 us.
// E: threads of a further warp that forms the shift beside the others' leap-frog (wide handles:
// the block's FP64 chain is what takes the time; step of one 346-nt replica 19.8 -> 18.8 us, of 7
// replicas of 203 nt 32.1 -> 31.2 us, FP64 step 32.1 -> 31.2 us).  Full blocks have their first warp
// do both: a fifth warp takes registers of blocks that would run beside (85.5 against 84.7 us).
template <bool D, int T, int E>
__global__ void __launch_bounds__(T + E) k_integrate(Dev d, int tail)
{
    wait_prior_grid();
    const int p = blockIdx.x * T + (int)threadIdx.x;
    const int r = d.blk_rep[blockIdx.x * T / kBlock];
    const RepParams *R = d.rp + r;
    __shared__ int s_est;
    __shared__ int s_last;
    constexpr bool I = T == kBlock;  // axis_fix
    __shared__ Shift<I> s_shift;
    if (threadIdx.x == 0) s_est = 0;
    int err = 0;
    float2 est = make_float2(0.0f, 0.0f);
    double xn[3], vn[3], xo[3];
    int4 q = make_int4(0, 0, 0, 0);
    if (E == 0 || threadIdx.x < T) q = d.q[p];
    const bool on = (q.w >> 16) & 1;
    // padding particles too (their state is zero and nothing of it is kept): the loads then
    // need not wait for the type's (step of 64 replicas 83.9 -> 83.6 us, one 18.0 -> 17.9 us)
    if (E == 0 || threadIdx.x < T) leap_frog<D, I>(d, R, r, p, xn, vn, &est);
    if (E == 0 ? threadIdx.x < 32 : threadIdx.x >= T) {
        const int lane = (int)threadIdx.x & 31;
        const double s = shift_lane<D>(d, R, r, lane);
        if (lane < 3) s_shift.set(R, lane, s);
    }
    __syncthreads();
    double *hold = d.centre + (size_t)r * kCentre;
    if (on) move_particle<D, I>(d, R, p, q, s_shift, xn, vn, xo, hold, err);
    // check_shifts (E:1745-1762): max |x - x_old|^2 over the block (a NaN estimate orders above all)
    const int wm = __reduce_max_sync(kFull, on ? __float_as_int(est.x) & 0x7fffffff : 0);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_est, wm);
    __syncthreads();
    // within 512 units in the last place, 3e-5 to 6e-5, of the block's largest estimate
    if (on && (__float_as_int(est.y) & 0x7fffffff) >= s_est - 512) atomicMax(&d.rs[r].maxd2, shift_bits(xn, xo));
    if (err) atomicOr(&d.rs[r].err, err);
    if (!tail) return;  // of the whole block
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        // the replica's last block to finish runs the skin check for it
        const unsigned done = atomicAdd(&d.rs[r].blocks_done, 1u);
        s_last = (done == (unsigned)(R->npad / T) - 1u);
        if (s_last) d.rs[r].blocks_done = 0u;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        if (threadIdx.x == 32) release_centre(d, R, hold);  // beside control_step's thread
        control_step(d, r);
        if (d.fr.every > 0) {  // a frame step: this block writes the replica's frame (all its blocks are done)
            __syncthreads();
            const long long kl = *(volatile long long *)&d.rs[r].klok;
            if (kl % d.fr.every == 0) write_frame(d, r, kl, (int)threadIdx.x, (int)blockDim.x, CtaBar{});
        }
    }
}

// check_shifts (E:1741-1776) and the LR gate of deterministic_forces_MPI (E:2550)
// for replica r, by thread 0.  RepState::rebuild stays as decided here until the
// next step's decision: the rebuild kernels that follow read it.
__device__ void control_step(const Dev &d, int r)
{
    const RepParams *R = d.rp + r;
    RepState *S = d.rs + r;
    if (threadIdx.x == 0) {
        const double d2 = __longlong_as_double((long long)__ldcg(&S->maxd2));  // every block of the step has added its own
        const unsigned pending = __ldcg(&S->pending);
        const long long kl = __ldcg(&S->klok) + 1;
        const double e2 = __ldcg(&S->e2st_acc), e3 = __ldcg(&S->e3st_acc);
        const unsigned long long ctr = __ldcg(&S->ctr);
        double progress = __ldcg(&S->progress);
        const double sh = sqrt(d2);
        progress += (sh + sh);
        const int reb = progress > R->skin;
        if (reb) progress = 0.0;
        S->maxd2 = 0ull;
        S->progress = progress;
        S->klok = kl;
        S->rebuild = reb;
        S->lr_now = (R->lr_interval <= 1) || ((kl + 1) % R->lr_interval == 1) || (progress == 0.0);
        if (pending) {  // the step's Monte Carlo draws and Gaussians (hbond_block)
            S->ctr = ctr + (pending - 1u) + (unsigned long long)kNoise;
            S->pending = 0u;
        }
        S->e2st = e2;  // stacking energies of the step just finished (E2_STACK, E3_STACK)
        S->e3st = e3;
        S->e2st_acc = 0.0;
        S->e3st_acc = 0.0;
    }
}

__global__ void k_force_rebuild(Dev d)
{
    RepState *S = d.rs + blockIdx.x;
    if (threadIdx.x == 0) {
        S->rebuild = 1;
        S->progress = 0.0;
        S->lr_now = 1;
        S->maxd2 = 0ull;
    }
}

// ---------------------------------------------------------------------------
// list rebuild (populate_lists, E:1546-1737)
// ---------------------------------------------------------------------------
// separate_in_cells (E:1461-1542): single periodic wrap then ceil(tmp / l)
__device__ inline int cell_axis(double v, double side, double l)
{
    double t = v;
    if (t < 0) t = __dadd_rn(t, side);
    else if (t > side) t = __dsub_rn(t, side);
    return (int)ceil(__ddiv_rn(t, l));
}

// cell_axis decided in FP32 from the fixed-point coordinate q = floor(v 2^32 / side)
// mod 2^32, for v in [0, side] (no wrap): c = q m / 2^32 approximates v / l (l = side
// / m) within 2e-7 m; when c lies farther than 4e-7 m + 1e-6 from an integer, ceil(c)
// is the FP64 result, else the FP64 form decides.
__device__ inline int cell_axis_q(double v, unsigned q, double side, double l, int m)
{
    const long long b = __double_as_longlong(v);
    if (b >= 0 && b <= __double_as_longlong(side)) {
        const float c = (float)q * ((float)m * 2.3283064365386963e-10f);
        const float fr = c - floorf(c), band = 4.0e-7f * (float)m + 1.0e-6f;
        if (fr > band && fr < 1.0f - band) return (int)c + 1;
    }
    return cell_axis(v, side, l);
}

// populate_lists' cell binning (separate_in_cells, E:1461-1542) and hydrogen-bond
// candidate status (E:1698-1736) of one rebuilding replica per block.  Counting
// and filling run on shared-memory cell counters when the replica's cells fit
// (Dev::cell_smem), else on the global ones.  In FP64 mode each cell's particles
// are put in index order, as the reference appends them (E:1536-1540), so that
// list order and FP64 summation order are reproducible; mixed-precision sums are
// exact in fixed point and need no order.  The packed positions are copied in cell
// order, so the pair search reads each cell's candidates contiguously.
constexpr int kCellThreads = 1024;

template <bool D>
__device__ __forceinline__ void cells_block(const Dev &d, int r)
{
    extern __shared__ int s_cells[];
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    RepState *S = d.rs + r;
    if (!S->rebuild) return;
    const RepParams *R = d.rp + r;
    const int nc = R->nc, tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, w = tid >> 5, nw = bd >> 5;
    // per cell: particle count, first slot (in place of the count in shared memory), fill counter
    int *cnt = d.cell_smem ? s_cells : d.cell_count + R->c0;
    int *first = d.cell_smem ? s_cells : d.cell_start + R->c0;
    int *fill = d.cell_smem ? s_cells + d.nc_max : d.cell_fill + R->c0;
    for (int c = tid; c < nc; c += bd) {
        cnt[c] = 0;
        fill[c] = 0;
    }
    if (tid == 0) s_carry = 0;
    __syncthreads();
    constexpr int kF = 4;  // particles of a thread whose loads are in flight together
    for (int i0 = tid; i0 < R->npad; i0 += kF * bd) {
        int4 qv[kF];
        double xv[kF][3];
#pragma unroll
        for (int u = 0; u < kF; ++u) {
            const int i = i0 + u * bd, p = R->p0 + i;
            qv[u] = make_int4(0, 0, 0, 0);
            if (i < R->npad) {
                qv[u] = d.q[p];
                xv[u][0] = d.x[p];
                xv[u][1] = d.y[p];
                xv[u][2] = d.z[p];
            }
        }
#pragma unroll
        for (int u = 0; u < kF; ++u) {
            const int i = i0 + u * bd;
            if (i >= R->npad) break;
            int c = -1;
            const int4 qp = qv[u];
            if ((qp.w >> 16) & 1) {
                const int i1 = cell_axis_q(xv[u][0], (unsigned)qp.x, R->box[0], R->lcell[0], R->mc[0]);
                const int i2 = cell_axis_q(xv[u][1], (unsigned)qp.y, R->box[1], R->lcell[1], R->mc[1]);
                const int i3 = cell_axis_q(xv[u][2], (unsigned)qp.z, R->box[2], R->lcell[2], R->mc[2]);
                if (i1 < 1 || i1 > R->mc[0] || i2 < 1 || i2 > R->mc[1] || i3 < 1 || i3 > R->mc[2]) {
                    atomicOr(&S->err, kErrRange);
                } else {
                    c = (i1 - 1) * R->mc[1] * R->mc[2] + (i2 - 1) * R->mc[2] + (i3 - 1);
                    atomicAdd(cnt + c, 1);
                }
            }
            d.cell_of[R->p0 + i] = c;
        }
    }
    __syncthreads();
    // exclusive scan of the counts: first slot of every cell
    for (int base = 0; base < nc; base += bd) {
        const int c = base + tid;
        const int v = c < nc ? cnt[c] : 0;
        int incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[w] = incl;
        __syncthreads();
        if (w == 0) {
            int t = lane < nw ? s_warp[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(kFull, t, o);
                if (lane >= o) t += u;
            }
            if (lane < nw) s_warp[lane] = t;
        }
        __syncthreads();
        const int excl = s_carry + (w > 0 ? s_warp[w - 1] : 0) + incl - v;
        if (c < nc) {
            first[c] = excl;
            d.cell_start[R->c0 + c] = excl;
            d.cell_count[R->c0 + c] = v;
        }
        __syncthreads();
        if (tid == bd - 1) s_carry = excl + v;
        __syncthreads();
    }
    const int nslots = s_carry;
    for (int i0 = tid; i0 < R->npad; i0 += kF * bd) {
        int cv[kF];
        int4 qv[kF];
#pragma unroll
        for (int u = 0; u < kF; ++u) {
            const int i = i0 + u * bd;
            cv[u] = -1;
            if (i < R->npad) {
                cv[u] = d.cell_of[R->p0 + i];
                if (!D) qv[u] = d.q[R->p0 + i];
            }
        }
#pragma unroll
        for (int u = 0; u < kF; ++u)
            if (cv[u] >= 0) {
                const int slot = R->p0 + first[cv[u]] + atomicAdd(fill + cv[u], 1);
                d.cell_list[slot] = R->p0 + i0 + u * bd;
                if (!D) d.qs[slot] = qv[u];
            }
    }
    __syncthreads();
    if (D)  // one warp per cell: rank sort (at most 8 particles per lane), or insertion sort by one lane
        for (int c = w; c < nc; c += nw) {
            const int n = d.cell_count[R->c0 + c];
            int *seg = d.cell_list + R->p0 + first[c];
            if (n > 1 && n <= 256) {
                int v[8], rk[8];
                int m = 0;
                for (int i = lane; i < n; i += 32, ++m) {
                    v[m] = seg[i];
                    int k = 0;
                    for (int u = 0; u < n; ++u) k += seg[u] < v[m];
                    rk[m] = k;
                }
                __syncwarp();
                for (int t = 0; t < m; ++t) seg[rk[t]] = v[t];
                __syncwarp();
            } else if (n > 256) {
                if (lane == 0)
                    for (int i = 1; i < n; ++i) {
                        const int v = seg[i];
                        int j = i - 1;
                        while (j >= 0 && seg[j] > v) {
                            seg[j + 1] = seg[j];
                            --j;
                        }
                        seg[j + 1] = v;
                    }
                __syncwarp();
            }
        }
    if (D) {
        __syncthreads();
        for (int i = tid; i < nslots; i += bd) d.qs[R->p0 + i] = d.q[d.cell_list[R->p0 + i]];
    }

    // hydrogen-bond candidates: live (0) when the central pair is within the SR radius
    for (int a = R->hba0 + tid; a < R->hba1; a += bd) d.hb_excess[a] = d.hba_n[a] - d.hba_val[a];
    __syncthreads();
    for (int k = R->hb0 + tid; k < R->hb1; k += bd) {
        const int a = d.hb_idx[6 * k + 1], b = d.hb_idx[6 * k + 4];
        const int st = (a != b && exact_r2(d, R, a, b) <= R->r2sr) ? 0 : -1;
        d.hb_status[k] = st;
        if (st != 0)
            for (int u = d.hb_aoff[k]; u < d.hb_aoff[k + 1]; ++u) atomicSub(d.hb_excess + d.hb_aidx[u], 1);
    }
    if (tid == 0) s_carry = 0;
    __syncthreads();
    // ordered compaction of the live candidates
    const int nh = R->hb1 - R->hb0;
    for (int base = 0; base < nh; base += bd) {
        const int k = R->hb0 + base + tid;
        const bool live = (base + tid < nh) && d.hb_status[k] == 0;
        const unsigned m = __ballot_sync(kFull, live);
        if (lane == 0) s_warp[w] = __popc(m);
        __syncthreads();
        int off = s_carry;
        for (int t = 0; t < w; ++t) off += s_warp[t];
        if (live) d.hb_active[R->hb0 + off + __popc(m & ((1u << lane) - 1u))] = k;
        __syncthreads();
        if (tid == 0) {
            int tot = 0;
            for (int t = 0; t < nw; ++t) tot += s_warp[t];
            s_carry += tot;
        }
        __syncthreads();
    }
    if (tid == 0) {
        S->n_active = s_carry;
        S->rebuilds += 1;
    }
}

template <bool D>
__global__ void __launch_bounds__(kCellThreads) k_cells(Dev d, int control)
{
    wait_prior_grid();
    const int r = blockIdx.x;
    if (control) {
        if (threadIdx.x == 32) release_centre(d, d.rp + r, d.centre + (size_t)r * kCentre);
        control_step(d, r);
        __syncthreads();
        if (d.fr.every > 0) {
            const long long kl = *(volatile long long *)&d.rs[r].klok;
            if (kl % d.fr.every == 0) write_frame(d, r, kl, (int)threadIdx.x, (int)blockDim.x, CtaBar{});
        }
    }
    cells_block<D>(d, r);
}

// how far, in cells, the cell d (-1, 0, 1) from cell i of m along an axis is from
// fixed-point coordinate q, which lies in cell i up to rounding at its faces
__device__ __forceinline__ float cell_gap(unsigned q, int m, int i, int d)
{
    const unsigned long long u = (unsigned long long)q * (unsigned)m;
    float f = (float)((int)(u >> 32) - i) + (float)(unsigned)u * 2.3283064365386963e-10f;  // from the lower face
    // a bead on the box's face may be binned on its other side
    f = f > 0.5f * (float)m + 0.5f ? f - (float)m : f < 0.5f - 0.5f * (float)m ? f + (float)m : f;
    const float below = fmaxf(0.0f, f), above = fmaxf(0.0f, 1.0f - f);
    if (d == 0 || m == 1) return 0.0f;
    return m == 2 ? fminf(below, above) : d < 0 ? below : above;  // of two cells, the other one is on both sides
}

// SR and LR neighbour lists (E:1576-1694).  A pair is SR when r^2 <= (sr+skin)^2,
// else LR when r^2 <= (rc+skin)^2 and neither bead is a sugar or a base.  The FP32
// distance from the exact integer differences decides outside a narrow band
// around each threshold; inside it the FP64 distance with the reference's
// rounding and image rule decides, so the lists are the reference's sets.
// One warp per particle.  Its up to 27 neighbour cells (a lane each) are those the sphere
// it looks in reaches: the LR list radius, or, for a bead without charge and pruned lists,
// its widest LJ range plus the skin (of 35 A cells, 18 and 3 on average, where all 27 were
// scanned before).  The cells' candidates, contiguous in cell order, are scanned end to end,
// 32 kU at a time, and hits appended in candidate order by ballot: the reference's order.
// Bound by instructions and the latency of the candidates' loads.  Alone, per step and 64
// replicas in one launch: 88 -> 49 us; 16 large ones: 200 -> 113 us.
// populate_lists' pair search for particle `off` of replica r by one warp; seg: the warp's
// 32 ints of shared memory
template <bool D>
__device__ __forceinline__ void search_particle(const Dev &d, int r, int off, int lane, int *seg)
{
    const unsigned lt = (1u << lane) - 1u;
    const int P = d.P;
    const RepParams *R = d.rp + r;
    const int p = R->p0 + off;
    const int c = d.cell_of[p];
    if (c < 0) {
        if (lane == 0) { d.n_sr[p] = 0; d.n_lr[p] = 0; }
        return;
    }
    const float sx = R->qstep[0], sy = R->qstep[1], sz = R->qstep[2];
    const float sr_lo = R->r2srf * (1.0f - kBand), sr_hi = R->r2srf * (1.0f + kBand);
    const float lr_lo = R->r2lrf * (1.0f - kBand), lr_hi = R->r2lrf * (1.0f + kBand);
    const int4 qp = d.q[p];
    const int nex = d.n_excl[p];
    const bool chp = is_charged((qp.w >> 8) & 0xff);
    // the lane's cell of the 3 x 3 x 3 block, in the reference's cell order
    int cnt = 0, start = 0;
    if (lane < 27) {
        const int m1 = R->mc[0], m2 = R->mc[1], m3 = R->mc[2];
        const int i1 = c / (m2 * m3), i2 = (c / m3) % m2, i3 = c % m3;
        const int d1 = lane / 9 - 1, d2 = (lane / 3) % 3 - 1, d3 = lane % 3 - 1;
        // an axis of one or two cells repeats them: each cell once, where the reference meets it first
        const bool rep = d1 > min(m1, 3) - 2 || d2 > min(m2, 3) - 2 || d3 > min(m3, 3) - 2;
        const float reach = chp ? R->reach_lr : d.full_lists ? R->reach_sr : R->reach_lj[qp.w & 0xff];
        const float g1 = cell_gap((unsigned)qp.x, m1, i1, d1) * R->lcellf[0], g2 = cell_gap((unsigned)qp.y, m2, i2, d2) * R->lcellf[1],
                    g3 = cell_gap((unsigned)qp.z, m3, i3, d3) * R->lcellf[2];
        if (!rep && g1 * g1 + g2 * g2 + g3 * g3 <= reach) {
            int a = i1 + d1, b = i2 + d2, e = i3 + d3;
            a += a < 0 ? m1 : a >= m1 ? -m1 : 0;
            b += b < 0 ? m2 : b >= m2 ? -m2 : 0;
            e += e < 0 ? m3 : e >= m3 ? -m3 : 0;
            const int cc = R->c0 + (a * m2 + b) * m3 + e;
            start = R->p0 + d.cell_start[cc];
            cnt = d.cell_count[cc];
        }
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(kFull, incl, 31), first = incl - cnt;
    const unsigned has = __ballot_sync(kFull, cnt > 0);
    __syncwarp();  // the previous particle's reads of seg are done
    if (cnt > 0) seg[__popc(has & lt)] = start - first;  // slot of candidate t of the n-th such cell: seg[n] + t
    __syncwarp();
    int exl[kExcl];
#pragma unroll
    for (int k = 0; k < kExcl; ++k) exl[k] = k < nex ? d.excl[(size_t)k * P + p] : -1;
    int nsr = 0, nlr = 0, before = 0;
    constexpr int kU = 4;  // candidate chunks of 32 whose loads are issued together
    for (int t0 = 0; t0 < total; t0 += 32 * kU) {
        int jv[kU];
        int4 qv[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int t = t0 + 32 * u + lane;
            // bit i: a cell's candidates begin at the chunk's i-th
            const unsigned rel = (unsigned)(first - (t0 + 32 * u));
            const unsigned begins = __reduce_or_sync(kFull, cnt > 0 && rel < 32u ? 1u << rel : 0u);
            jv[u] = -1;
            qv[u] = make_int4(0, 0, 0, 0);
            if (t < total) {
                const int slot = seg[before + __popc(begins & (lt | (1u << lane))) - 1] + t;
                jv[u] = d.cell_list[slot];
                qv[u] = d.qs[slot];
            }
            before += __popc(begins);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (t0 + 32 * u >= total) break;
            const int j = jv[u];
            const int4 qj = qv[u];
            int cls = 0;  // 0 none, 1 SR, 2 LR
            if (j >= 0 && j != p) {
                const bool ch = chp && is_charged((qj.w >> 8) & 0xff);
                const float dx = (float)(int)((unsigned)qp.x - (unsigned)qj.x) * sx;
                const float dy = (float)(int)((unsigned)qp.y - (unsigned)qj.y) * sy;
                const float dz = (float)(int)((unsigned)qp.z - (unsigned)qj.z) * sz;
                const float r2f = dx * dx + dy * dy + dz * dz;
                if (D) {
                    const double r2 = exact_r2(d, R, p, j);
                    cls = r2 <= R->r2sr ? 1 : ((ch && r2 <= R->r2lr) ? 2 : 0);
                } else {
                    if (r2f < sr_lo) cls = 1;
                    else if (r2f > sr_hi && (!ch || r2f > lr_hi)) cls = 0;
                    else if (r2f > sr_hi && r2f < lr_lo) cls = 2;
                    else {
                        const double e2 = exact_r2(d, R, p, j);
                        cls = e2 <= R->r2sr ? 1 : ((ch && e2 <= R->r2lr) ? 2 : 0);
                    }
                }
                // pruned list: a pair with an uncharged bead can only exert LJ, which
                // vanishes beyond D_LJ; the skin keeps it exact until the next rebuild
                if (cls == 1 && !d.full_lists && !ch && r2f > R->ljkeep2[jn12(qp.w & 0xff, qj.w & 0xff)]) cls = 0;
            }
            const unsigned bs = __ballot_sync(kFull, cls == 1), bl = __ballot_sync(kFull, cls == 2);
            if (cls == 1) {
                int m = 0;  // how often the reference subtracts this pair's LJ again
                if (nex)
#pragma unroll
                    for (int k = 0; k < kExcl; ++k) m += exl[k] == j;
                const int pos = nsr + __popc(bs & lt);
                if (pos < d.cap_sr) d.nbr_sr[nb_idx(pos, p, P)] = j | (m << kExclShift);
            } else if (cls == 2) {
                const int pos = nlr + __popc(bl & lt);
                if (pos < d.cap_lr) d.nbr_lr[nb_idx(pos, p, P)] = j;
            }
            nsr += __popc(bs);
            nlr += __popc(bl);
        }
    }
    if (lane == 0) {
        if (nsr > d.cap_sr || nlr > d.cap_lr) atomicOr(&d.rs[r].err, kErrCapacity);
        d.n_sr[p] = min(nsr, d.cap_sr);
        d.n_lr[p] = min(nlr, d.cap_lr);
    }
}

// the warps stride over the particles of the replicas that rebuild this step, laid end to end
template <bool D>
__global__ void __launch_bounds__(128) k_pair_search(Dev d)
{
    wait_prior_grid();
    __shared__ int s_seg[4][32];
    const int lane = threadIdx.x & 31, warps = d.search_warps;
    int next = (blockIdx.x * 4 + (threadIdx.x >> 5));  // this warp's next particle, counted from the replica's first
    for (int base = 0; base < d.R; base += 32) {
        unsigned m = __ballot_sync(kFull, base + lane < d.R && d.rs[min(base + lane, d.R - 1)].rebuild);
        for (; m; m &= m - 1u) {
            const int r = base + __ffs((int)m) - 1, npad = d.rp[r].npad;
            for (; next < npad; next += warps) search_particle<D>(d, r, next, lane, s_seg[threadIdx.x >> 5]);
            next -= npad;
        }
    }
}

// ---------------------------------------------------------------------------
// persistent fused step kernel: one thread-block cluster per replica runs `steps`
// whole steps (the sequence of E:6380-6386) without leaving the kernel
// ---------------------------------------------------------------------------
// A replica's cluster of C CTAs (cluster dimension C, grid R x C) shares its work;
// phases are separated by the cluster's hardware barrier (all CTAs of a cluster are
// resident together, so no wait depends on another cluster).  Per step:
//   forces   warps 0-7 of the first CTA: H-bond terms, the valence-limited Monte
//            Carlo and the step's Gaussians (hbond_block on a named barrier); all
//            other threads: SR pairs (one thread per particle), LR pairs when due
//            (four per particle), bonded terms and stacks (one thread per item)
//   shift    every CTA forms the recentring shift from the centre bead
//   move     each CTA integrates its share of the particles; max |x - x_old|^2
//   control  check_shifts and the LR gate (control_step) by the first CTA
//   rebuild  when due: cell binning by the first CTA, pair search by every warp
// Data the kernel rewrites while it runs is read through L2 (__ldcg).
constexpr int kFusedThreads = 512;
constexpr int kFusedHbThreads = 256;
constexpr int kFusedWarps = kFusedThreads / 32;

__device__ __forceinline__ int cluster_rank()
{
    unsigned v;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    return (int)v;
}
__device__ __forceinline__ int cluster_ctas()
{
    unsigned v;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
    return (int)v;
}
// every thread of the cluster; writes before it (global and shared) are visible to
// every thread of the cluster after it
__device__ __forceinline__ void cluster_barrier()
{
    __threadfence();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <bool D>
__global__ void __launch_bounds__(kFusedThreads, 1) k_step_fused(Dev d, int steps)
{
    const int cs = cluster_ctas(), rank = cluster_rank();
    const int r = blockIdx.x / cs;
    const RepParams *R = d.rp + r;
    RepState *S = d.rs + r;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ float s_dlj2[46], s_dm[46], s_flj[46], s_qclb[46];
    __shared__ int s_seg[kFusedWarps][32];
    __shared__ double s_shift[3];
    __shared__ unsigned long long s_max;
    for (int t = tid; t < 46; t += kFusedThreads) {
        s_dlj2[t] = R->dlj2[t];
        s_dm[t] = R->dm[t];
        s_flj[t] = R->flj[t];
        s_qclb[t] = R->qclb[t];
    }
    __syncthreads();
    const PairTables tb{s_dlj2, s_dm, s_flj, s_qclb};
    const bool hbt = rank == 0 && tid < kFusedHbThreads;  // the H-bond threads
    const int nwk = cs * kFusedThreads - kFusedHbThreads;  // pair workers (a multiple of 32)
    const int wk = rank * kFusedThreads + tid - kFusedHbThreads;  // this thread's worker index (when !hbt)
    const int npad = R->npad, p0 = R->p0;
    const int nb = R->bt1 - R->bt0, n3 = R->s31 - R->s30, n2 = R->s21 - R->s20;
    const int per = (npad / kBlock + cs - 1) / cs * kBlock;  // particles integrated per CTA
    int err = 0;
    // phase times (tis_profile_fused): the first thread of the cluster's first CTA
    const bool timer = d.fprof && rank == 0 && tid == 0;
    unsigned long long ph[8] = {0, 0, 0, 0, 0, 0, 0, 0}, t0 = timer ? global_ns() : 0ull, t1;
    auto lap = [&](int k) {
        if (timer) {
            t1 = global_ns();
            ph[k] += t1 - t0;
            t0 = t1;
        }
    };
    for (int step = 0; step < steps; ++step) {
        const int lr_now = __ldcg(&S->lr_now);
        if (hbt) {
            hbond_block<D, false>(d, r, 1, 1, tid, kFusedHbThreads, NamedBar{1, kFusedHbThreads});
            if (timer) ph[1] += global_ns() - t0;
        } else {
            for (int i = wk; i < npad; i += nwk) pair_particle<D, false, 1>(d, R, p0 + i, 0, tb, err);
            if (lr_now)  // groups of four workers per particle (every group of a warp runs the same passes)
                for (int i = wk >> 2; i < npad; i += nwk >> 2)
                    pair_particle<D, true, 4>(d, R, p0 + i, wk & 3, tb, err);
            for (int i = wk; i < nb + n3 + n2; i += nwk) {
                const int t = i < nb ? R->bt0 + i
                                     : (i < nb + n3 ? d.nbt + R->s30 + (i - nb) : d.nbt + d.nst3 + R->s20 + (i - nb - n3));
                topo_item<D>(d, t);
            }
        }
        cluster_barrier();
        lap(0);
        ph[6] += lr_now ? 1 : 0;
        if (warp == 0) {  // adjust_box's shift (E:2632-2656) from the centre bead's new position
            const double s = shift_lane<D>(d, R, r, lane);
            if (lane < 3) s_shift[lane] = s;
            if (lane == 0) s_max = 0ull;
        }
        cluster_barrier();  // no CTA moves the centre bead before every CTA has read it
        lap(2);
        {
            const Shift<false> sh = {{s_shift[0], s_shift[1], s_shift[2]}};
            unsigned long long bits = 0ull;
            const int i1 = min(npad, (rank + 1) * per);
            for (int i = rank * per + tid; i < i1; i += kFusedThreads) {
                const int4 q = d.q[p0 + i];
                if (!((q.w >> 16) & 1)) continue;
                double xn[3], vn[3], xo[3];
                leap_frog<D, false>(d, R, r, p0 + i, xn, vn);
                move_particle<D, false>(d, R, p0 + i, q, sh, xn, vn, xo, nullptr, err);
                bits = max(bits, shift_bits(xn, xo));
            }
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long b = __shfl_down_sync(kFull, bits, o);
                bits = b > bits ? b : bits;
            }
            if (lane == 0) atomicMax(&s_max, bits);
            __syncthreads();
            if (tid == 0) atomicMax(&S->maxd2, s_max);
        }
        cluster_barrier();
        lap(3);
        if (rank == 0) control_step(d, r);  // thread 0: check_shifts, the next step's LR gate
        cluster_barrier();
        lap(4);
        if (d.fr.every > 0 && rank == 0) {  // a frame step: the first CTA writes the replica's frame
            const long long kl = __ldcg(&S->klok);
            if (kl % d.fr.every == 0) write_frame(d, r, kl, tid, kFusedThreads, CtaBar{});
        }
        if (__ldcg(&S->rebuild)) {  // populate_lists (E:1546-1737)
            if (rank == 0) cells_block<D>(d, r);
            cluster_barrier();
            for (int off = rank * kFusedWarps + warp; off < npad; off += cs * kFusedWarps)
                search_particle<D>(d, r, off, lane, s_seg[warp]);
            cluster_barrier();
            lap(5);
            ph[7] += 1;
        }
    }
    if (err) atomicOr(&S->err, err);
    if (timer)
        for (int k = 0; k < 8; ++k) atomicAdd(d.fprof + (size_t)r * kFusedPhases + k, ph[k]);
}

// radius_of_gyration (E:2844-2876) of the RNA beads of one replica
__global__ void k_rg(Dev d, int r, double *out)
{
    const RepParams *R = d.rp + r;
    __shared__ double s_red[3 * 32];
    double c[3] = {0, 0, 0};
    for (int i = threadIdx.x; i < R->nrna; i += blockDim.x) {
        c[0] += d.x[R->p0 + i];
        c[1] += d.y[R->p0 + i];
        c[2] += d.z[R->p0 + i];
    }
    block_sum<3>(c, s_red);
    __shared__ double s_c[3];
    if (threadIdx.x == 0)
        for (int k = 0; k < 3; ++k) s_c[k] = c[k] / R->nrna;
    __syncthreads();
    double s[1] = {0};
    for (int i = threadIdx.x; i < R->nrna; i += blockDim.x) {
        const double a = d.x[R->p0 + i] - s_c[0], b = d.y[R->p0 + i] - s_c[1], e = d.z[R->p0 + i] - s_c[2];
        s[0] += a * a + b * b + e * e;
    }
    block_sum<1>(s, s_red);
    if (threadIdx.x == 0) *out = sqrt(s[0] / R->nrna);
}

// Ions of one kind within sqrt(r2cut) of each phosphate of replica r, from the SR
// lists (complete within the SR radius between rebuilds): count[i] for RNA bead i
// (-1 for sugars and bases), hit[j] = 1 for every ion j within range of some P.  A warp
// per bead, its lanes over the list.
__global__ void k_ion_counts(Dev d, int r, int kind, double r2cut, int *count, int *hit)
{
    const RepParams *R = d.rp + r;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= R->nrna) return;
    const int p = R->p0 + i;
    int c = -1;
    if (((d.q[p].w >> 8) & 0xff) == 0) {
        const int n = d.n_sr[p];
        c = 0;
        for (int k = lane; k < n; k += 32) {
            const int j = d.nbr_sr[nb_idx(k, p, d.P)] & kIdxMask;
            if (((d.q[j].w >> 8) & 0xff) == kind && exact_r2(d, R, p, j) <= r2cut) {
                ++c;
                hit[j - R->p0] = 1;
            }
        }
        c = __reduce_add_sync(kFull, c);
    }
    if (lane == 0) count[i] = c;
}

// the total force of particles p0 .. p0 + n - 1 as (x, y, z) triples
__global__ void k_get_forces(Dev d, int p0, int n, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int c = 0; c < 3; ++c) out[3 * i + c] = d.fp64 ? total_force<true>(d, p0 + i, c) : total_force<false>(d, p0 + i, c);
}

// clears every replica's device-side error flags
__global__ void k_clear_err(Dev d)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < d.R; r += gridDim.x * blockDim.x) d.rs[r].err = 0;
}

// the largest SR and LR neighbour counts of the group (out[0], out[1]; zero on entry)
__global__ void k_list_peaks(Dev d, int *out)
{
    int a = 0, b = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.P; p += gridDim.x * blockDim.x) {
        a = max(a, d.n_sr[p]);
        b = max(b, d.n_lr[p]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = max(a, __shfl_down_sync(kFull, a, o));
        b = max(b, __shfl_down_sync(kFull, b, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, a);
        atomicMax(out + 1, b);
    }
}

// E2_HB, E3_HB, E2_STACK, E3_STACK and Rg of every replica (one block each)
__global__ void k_energies(Dev d, double *out)
{
    energies_block(d, blockIdx.x, out + 5 * blockIdx.x, (int)threadIdx.x, (int)blockDim.x, CtaBar{});
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void launch_quantize(const Dev &d, cudaStream_t s) { k_quantize<<<d.nblk, kBlock, 0, s>>>(d); }

void launch_put_state(const Dev &d, cudaStream_t s, const double *stage, int n)
{
    k_put_state<<<d.nblk, kBlock, 0, s>>>(d, stage, n);
}

void launch_get_state(const Dev &d, cudaStream_t s, double *stage, int n, unsigned mask)
{
    k_get_state<<<d.nblk, kBlock, 0, s>>>(d, stage, n, mask);
}

void launch_energies(const Dev &d, cudaStream_t s, double *out) { k_energies<<<d.R, 256, 0, s>>>(d, out); }

void launch_get_forces(const Dev &d, cudaStream_t s, int p0, int n, double *out)
{
    k_get_forces<<<(n + 127) / 128, 128, 0, s>>>(d, p0, n, out);
}

void launch_clear_err(const Dev &d, cudaStream_t s) { k_clear_err<<<1, 256, 0, s>>>(d); }

void launch_list_peaks(const Dev &d, cudaStream_t s, int *out) { k_list_peaks<<<d.sm_count, 256, 0, s>>>(d, out); }

void launch_ion_counts(const Dev &d, cudaStream_t s, int r, int nrna, int kind, double r2cut, int *count, int *hit)
{
    k_ion_counts<<<(nrna + 3) / 4, 128, 0, s>>>(d, r, kind, r2cut, count, hit);
}

void launch_pair(const Dev &d, cudaStream_t s, bool en, int sr, int lr)
{
    const int nb = d.P / 32;
    if (d.fp64) {
        if (en) k_pair<true, true><<<nb, kPairAlone, 0, s>>>(d, sr, lr);
        else k_pair<true, false><<<nb, kPairAlone, 0, s>>>(d, sr, lr);
    } else {
        if (en) k_pair<false, true><<<nb, kPairAlone, 0, s>>>(d, sr, lr);
        else k_pair<false, false><<<nb, kPairAlone, 0, s>>>(d, sr, lr);
    }
}

namespace {

TopoPlan topo_plan(const Dev &d, bool noise)
{
    TopoPlan tp;
    tp.per = d.wide ? 64 : kForceThreads;
    tp.n3 = (d.nst3 + 63) / 64;
    tp.n2 = (d.nst2 + 127) / 128;
    tp.nb = (d.nbt + tp.per - 1) / tp.per;
    tp.nn = noise && d.noise == 0 ? (d.R * noise_blocks((kNoise + kNoiseSpare) / 2) + tp.per - 1) / tp.per : 0;
    return tp;
}

// a launch that may begin before the previous kernel on the stream has finished
// (the kernel waits in wait_prior_grid).  All four of a step: the force kernel launched this
// way as well took the step of 64 replicas 83.6 -> 82.9 us, the drop-in step 49.2 -> 47.7 us.
// An early trigger in them (griddepcontrol.launch_dependents) is worth nothing on one small
// replica (17.4 us either way) and costs where groups share the GPU (7 replicas 30.1 -> 33.2 us),
// as the waiting blocks hold room that running kernels would take.
template <class K, class... A>
void launch_pdl(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t s, const Dev &d, A... a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, d, a...);
}

template <bool D, int PB, int TS>
size_t forces_smem(const Dev &d)
{
    const size_t pair = sizeof(PairSmem<D, PB>) * (kForceThreads / TS), topo = sizeof(Real<D>) * 16 * 32;
    size_t m = pair > topo ? pair : topo;
    return m > (size_t)d.hb_smem ? m : (size_t)d.hb_smem;
}

template <bool D, int PB, int TS>
void launch_forces_t(const Dev &d, cudaStream_t s, bool noise)
{
    const TopoPlan tp = topo_plan(d, noise);
    constexpr int per = PB * (kForceThreads / TS);  // particles per pair block
    const dim3 grid((unsigned)(d.R + tp.blocks() + (d.P + per - 1) / per));
    launch_pdl(k_forces<D, PB, TS>, grid, dim3(kForceThreads), forces_smem<D, PB, TS>(d), s, d, tp, noise ? 1 : 0);
}

}  // namespace

void launch_forces(const Dev &d, cudaStream_t s, bool noise)
{
    if (d.fp64) {
        if (d.wide) launch_forces_t<true, 32, 512>(d, s, noise);
        else launch_forces_t<true, 32, 128>(d, s, noise);
    } else {
        if (d.wide) launch_forces_t<false, 32, 128>(d, s, noise);
        else launch_forces_t<false, 128, 128>(d, s, noise);
    }
}

void launch_topology(const Dev &d, cudaStream_t s, int mask, bool en, bool make_noise, bool ex)
{
    const int xl = ex ? 1 : 0;
    const TopoPlan tp = topo_plan(d, false);
    if ((mask & (4 | 8)) && tp.blocks() > 0) {
        if (d.fp64) {
            if (en) k_topo<true, true><<<tp.blocks(), kForceThreads, 0, s>>>(d, tp, mask, xl);
            else k_topo<true, false><<<tp.blocks(), kForceThreads, 0, s>>>(d, tp, mask, xl);
        } else {
            if (en) k_topo<false, true><<<tp.blocks(), kForceThreads, 0, s>>>(d, tp, mask, xl);
            else k_topo<false, false><<<tp.blocks(), kForceThreads, 0, s>>>(d, tp, mask, xl);
        }
    }
    const int hb = (mask & 16) ? 1 : 0, mn = make_noise ? 1 : 0;
    const size_t sm = hb ? (size_t)d.hb_smem : 0;
    if (hb || mn) {
        if (d.fp64) {
            if (en) k_hbond<true, true><<<d.R, kHbThreads, sm, s>>>(d, hb, mn);
            else k_hbond<true, false><<<d.R, kHbThreads, sm, s>>>(d, hb, mn);
        } else {
            if (en) k_hbond<false, true><<<d.R, kHbThreads, sm, s>>>(d, hb, mn);
            else k_hbond<false, false><<<d.R, kHbThreads, sm, s>>>(d, hb, mn);
        }
    }
}

// Every kernel with dynamic shared memory may take as much as a block can have: the
// limit belongs to the function, not to a handle, so no handle's size is set.
int configure_kernels(const Dev &)
{
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (const void *k : {(const void *)k_step_fused<true>, (const void *)k_step_fused<false>, (const void *)k_cells<true>,
                          (const void *)k_cells<false>, (const void *)k_hbond<true, true>, (const void *)k_hbond<true, false>,
                          (const void *)k_hbond<false, true>, (const void *)k_hbond<false, false>,
                          (const void *)k_forces<true, 32, 512>, (const void *)k_forces<true, 32, 128>,
                          (const void *)k_forces<false, 32, 128>, (const void *)k_forces<false, 128, 128>}) {
        cudaFuncAttributes a;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
    }
    return (int)e;
}

void launch_noise(const Dev &d, cudaStream_t s)
{
    if (d.fp64) launch_pdl(k_noise<true>, d.R, kNoiseThreads, 0, s, d);
    else launch_pdl(k_noise<false>, d.R, kNoiseThreads, 0, s, d);
}

void launch_move(const Dev &d, cudaStream_t s, int tail)
{
    if (d.wide) {
        if (d.fp64) launch_pdl(k_integrate<true, 64, 32>, d.P / 64, 64 + 32, 0, s, d, tail);
        else launch_pdl(k_integrate<false, 64, 32>, d.P / 64, 64 + 32, 0, s, d, tail);
    } else {
        if (d.fp64) launch_pdl(k_integrate<true, kBlock, 0>, d.nblk, kBlock, 0, s, d, tail);
        else launch_pdl(k_integrate<false, kBlock, 0>, d.nblk, kBlock, 0, s, d, tail);
    }
}

void launch_cells(const Dev &d, cudaStream_t s, int control)
{
    if (d.fp64) launch_pdl(k_cells<true>, d.R, d.cell_threads, d.cell_smem, s, d, control);
    else launch_pdl(k_cells<false>, d.R, d.cell_threads, d.cell_smem, s, d, control);
}

void launch_search(const Dev &d, cudaStream_t s)
{
    if (d.fp64) launch_pdl(k_pair_search<true>, d.search_warps / 4, 128, 0, s, d);
    else launch_pdl(k_pair_search<false>, d.search_warps / 4, 128, 0, s, d);
}

void launch_rebuild(const Dev &d, cudaStream_t s, int control)
{
    launch_cells(d, s, control);
    launch_search(d, s);
}

void launch_force_all_rebuild(const Dev &d, cudaStream_t s) { k_force_rebuild<<<d.R, 128, 0, s>>>(d); }

void launch_rg(const Dev &d, cudaStream_t s, int replica, double *out) { k_rg<<<1, 256, 0, s>>>(d, replica, out); }

// forces (+ Gaussians), integrate (+ recentring shift), cells (+ skin check), pair search
int kernel_launches_per_step() { return 4; }

size_t fused_smem(const Dev &d) { return (size_t)max(d.hb_smem, d.cell_smem); }

int launch_step_fused(const Dev &d, cudaStream_t s, int steps, int ctas)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(d.R * ctas));
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = fused_smem(d);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)(d.fp64 ? cudaLaunchKernelEx(&cfg, k_step_fused<true>, d, steps)
                        : cudaLaunchKernelEx(&cfg, k_step_fused<false>, d, steps));
}

}  // namespace tis
