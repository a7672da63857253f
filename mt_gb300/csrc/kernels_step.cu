// kernels_step.cu - per-bead forces, the fused force + Euler-Maruyama step,
// energies, and the state <-> Coord conversions.
//
// One thread per bead (k_step_plain, k_forces), or in small batches four threads
// by role (k_split), or one CTA per trajectory for a whole list period
// (k_period_split, k_step_period).  A bead's neighbours are read from the current frame
// buffer (16 B gathers of precomputed lab-frame site vectors, L2-resident for
// the batch sizes of interest); the moving bead writes its new state and new
// site vectors to the other buffer, so forces and integration fuse into one
// launch per step without a race.
#include "mtg_internal.cuh"

namespace mtg {

struct Acc {
    float fx, fy, fz, ffi, fpsi, fth, tx, ty, tz;
};

// The force arithmetic below is written with explicitly rounded operations
// wherever a product meets a sum, so that every kernel it is inlined into
// (per-step, persistent, forces only) gives the same bits.

// Adds a pair term with radial factor dUdr = U'(r)/r along d = site_j - site_i
// and its torque dUdr * (w_i x d) about the bead centre.
__device__ __forceinline__ float cross1(float a, float b, float c, float d) {   // a b - c d
    return __fmaf_rn(a, b, -__fmul_rn(c, d));
}
__device__ __forceinline__ void acc_pair(Acc &A, float dUdr, float3 d, float3 wi) {
    A.fx = __fmaf_rn(dUdr, d.x, A.fx);
    A.fy = __fmaf_rn(dUdr, d.y, A.fy);
    A.fz = __fmaf_rn(dUdr, d.z, A.fz);
    A.tx = __fmaf_rn(dUdr, cross1(wi.y, d.z, wi.z, d.y), A.tx);
    A.ty = __fmaf_rn(dUdr, cross1(wi.z, d.x, wi.x, d.z), A.ty);
    A.tz = __fmaf_rn(dUdr, cross1(wi.x, d.y, wi.y, d.x), A.tz);
}

// sin(x) without the library's large-argument code in line: x = k pi + r, three
// fused steps with pi in three parts, then an odd polynomial fitted to sin on
// [-pi/2, pi/2] (minimax in the relative error: 1e-8 with these coefficients before
// rounding), and the sign of (-1)^k.  Largest relative error over the angles up to 1000 rad,
// every 13th float: 1.2e-7 (1.4e-6 next to multiples of pi without the third part), inside
// the two units in the last place of sinf.  Larger angles go to sinf.
static __device__ __noinline__ float sin_far(float x) { return sinf(x); }
__device__ __forceinline__ float sin_fit(float x) {
    if (!(fabsf(x) < 1000.0f)) return sin_far(x);
    const float t = __fmaf_rn(x, 0.318309886f, 12582912.0f), k = __fsub_rn(t, 12582912.0f);
    const float r = __fmaf_rn(k, 3.43019883e-15f, __fmaf_rn(k, 8.74227766e-8f, __fmaf_rn(k, -3.14159274f, x)));
    const float u = __fmul_rn(r, r);
    float p = __fmaf_rn(2.605780537e-6f, u, -1.980960224e-4f);
    p = __fmaf_rn(p, u, 8.333066478e-3f);
    p = __fmaf_rn(p, u, -1.666665971e-1f);
    const float s = __fmaf_rn(__fmul_rn(r, u), p, r);
    return __int_as_float(__float_as_int(s) ^ (__float_as_int(t) << 31));
}

// Bending terms of a harmonic/longitudinal partner (src/compute_cuda.cu:142-180,
// :265-298): sign by the site side, theta0 chosen by the caller.
__device__ __forceinline__ void acc_bend(const KParams &P, Acc &A, float rmon, float dpsi, float dfi, float dth,
                                         float th0) {
    // rmon > 0: + B sin(d - d0); rmon < 0: - B sin(-d - d0)
    const float sg = rmon > 0.0f ? 1.0f : -1.0f;
    A.fpsi = __fmaf_rn(__fmul_rn(sg, P.B_psi), sin_fit(__fmaf_rn(sg, dpsi, -P.psi_0)), A.fpsi);
    A.ffi = __fmaf_rn(__fmul_rn(sg, P.B_fi), sin_fit(__fmaf_rn(sg, dfi, -P.fi_0)), A.ffi);
    A.fth = __fmaf_rn(__fmul_rn(sg, P.B_theta), sin_fit(__fmaf_rn(sg, dth, -th0)), A.fth);
}

// r and 1/r from r^2: the hardware reciprocal square root with one correction each, so r is
// as a rounded root and 1/r as a rounded division give them (the approximation alone is 2e-7 off).
// Error of the forces against FP64, rms over 24 systems, forces and torques: 2.927e-5 and 8.615e-5
// (2.931e-5 and 8.623e-5 without the corrections; 3.089e-5 and 8.819e-5 with rounded roots,
// divisions and the library's sine, and LJ from the root).
// Squares past the largest float count as that one: the exponentials of r are 0 there.
struct Dist {
    float r, rinv;
};
__device__ __forceinline__ Dist dist_of(float r2) {
    const float x = fminf(r2, 3.402823466e38f), y = rsqrt_hw(x);
    float r = __fmul_rn(x, y);
    r = __fmaf_rn(__fmaf_rn(-r, r, x), __fmul_rn(0.5f, y), r);
    return {r, __fmaf_rn(__fmaf_rn(-r, y, 1.0f), y, y)};
}
// U'(r)/r of a Morse bond.  Squares below the smallest normal float count as touching sites
// (no force), as r = 0 does.
__device__ __forceinline__ float dmorse_over_r(float D, float a, float r, float rinv) {
    const float e = expf(__fmul_rn(-a, r));
    return __fmul_rn(__fmul_rn(__fmul_rn(2.0f * a, D), __fmul_rn(__fsub_rn(1.0f, e), e)), rinv);
}
__device__ __forceinline__ float norm2(float3 d) {
    return __fmaf_rn(d.x, d.x, __fmaf_rn(d.y, d.y, __fmul_rn(d.z, d.z)));
}
constexpr float kTouch2 = 1.17549435e-38f;

// Where a bead's neighbours' frames and flags are read: plane k of local bead
// j at fr[k * stride + base + j], its flags at fl[base + j].  The per-step
// kernels read the global frame buffer (stride nb, base = the trajectory's
// first bead); the persistent kernel reads its trajectory's copy in shared
// memory (stride = trajectory size, base 0).  Same arithmetic either way.
struct NbrView {
    const float4 *fr;
    const int *fl;
    int stride, base;
};

// What a bead's force loops start from, requested together at the head of a
// kernel so that no list's chain count -> entry -> neighbour waits for
// another's (entries past a count are in bounds and ignored).
struct ListHead {
    int nl, nt, nlj;
    int e_h0, e_l0, e_t0;
    int jj[4];
};
__device__ __forceinline__ ListHead list_head(const KParams &P, const DevBuffers &B, int g) {
    ListHead H;
    H.nl = P.maxLong > 0 ? B.lonc[g] : 0;
    H.nt = P.maxLat > 0 ? B.latc[g] : 0;
    H.nlj = P.lj_on ? B.ljc[g] : 0;
    H.e_h0 = B.harm[g * P.maxH];
    H.e_l0 = P.maxLong > 0 ? B.lon[g] : 0;
    H.e_t0 = P.maxLat > 0 ? B.lat[g] : 0;
#pragma unroll
    for (int u = 0; u < 4; u++) H.jj[u] = (P.lj_on && u < P.maxLJ) ? B.lj[u * P.nb + g] : 0;
    return H;
}

// LJ r^-6 repulsion with the hard 6 nm force cutoff (src/compute_cuda.cu:470-495):
// 6 pref / r^8 along the difference.  Four neighbours a round; while a round is
// summed, the indices of the next are in flight.
// Even and odd list entries have sums of their own, added at the end.
__device__ __forceinline__ float3 lj_force(const KParams &P, const DevBuffers &B, const NbrView &V, int g,
                                           float4 p0, const ListHead &H) {
    const int nb = P.nb;
    const float4 *fr = V.fr + V.base;
    float3 s[2] = {make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
    int jj[4] = {H.jj[0], H.jj[1], H.jj[2], H.jj[3]};
    const int *next = B.lj + g;
    const float c = 6.0f * P.lj_pref;
#pragma unroll 1
    for (int k0 = 0; k0 < H.nlj; k0 += 4) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) q[u] = k0 + u < H.nlj ? fr[jj[u]] : make_float4(3.0e18f, 0.f, 0.f, 0.f);
        next += 4 * nb;
        if (k0 + 4 < H.nlj) {
#pragma unroll
            for (int u = 0; u < 4; u++) jj[u] = k0 + 4 + u < P.maxLJ ? next[u * nb] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float dx = __fsub_rn(p0.x, q[u].x), dy = __fsub_rn(p0.y, q[u].y), dz = __fsub_rn(p0.z, q[u].z);
            const float r2 = norm2(make_float3(dx, dy, dz));
            if (r2 < 36.0f) {
                const float i2 = rcp_hw(r2), i4 = __fmul_rn(i2, i2), f = __fmul_rn(c, __fmul_rn(i4, i4));
                float3 &S = s[u & 1];
                S.x = __fmaf_rn(f, dx, S.x);
                S.y = __fmaf_rn(f, dy, S.y);
                S.z = __fmaf_rn(f, dz, S.z);
            }
        }
    }
    return make_float3(__fadd_rn(s[0].x, s[1].x), __fadd_rn(s[0].y, s[1].y), __fadd_rn(s[0].z, s[1].z));
}

// Bonds along the protofilament axis of bead g (src/compute_cuda.cu:69-301):
// harmonic + bending inside the dimer, then Morse longitudinal + bending and
// barrier, in one loop.  (Force, bending and torque sums from zero.)
__device__ __forceinline__ Acc axial_force(const KParams &P, const DevBuffers &B, const NbrView &V, int g, int flags,
                                           float4 p0, float4 p1, float theta, const ListHead &H) {
    const int nb = P.nb;          // list layout (k-major over all beads)
    const int ps = V.stride;      // plane stride of the neighbour frames
    const float4 *fr = V.fr + V.base;
    Acc A = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const bool off_tub = (flags & kFlagOnTubule) == 0;
    const int hc = (flags >> kHarmShift) & 7;
#pragma unroll 1
    for (int k = 0; k < hc + H.nl; k++) {
        const bool harm = k < hc;
        int e;
        if (harm)
            e = k == 0 ? H.e_h0 : B.harm[g * P.maxH + k];
        else
            e = k == hc ? H.e_l0 : B.lon[(k - hc) * nb + g];
        const float rmon = e < 0 ? 2.0f : -2.0f;
        const int pj = e < 0 ? -e : e;
        const float4 rj = fr[pj], uj = fr[ps + pj];
        const float thj = fr[2 * ps + pj].w;
        const int fj = V.fl[V.base + pj];
        const float3 wi = make_float3(p1.x * rmon, p1.y * rmon, p1.z * rmon);
        const float3 wj = make_float3(-uj.x * rmon, -uj.y * rmon, -uj.z * rmon);
        const float3 d = site_delta(p0, rj, wi, wj);
        const float r2 = norm2(d);
        float dUdr = P.C;
        int gl = flags;   // whose nucleotide sets theta0: the bead's own, or (longitudinal) the
                          // bead's nearer the plus end (:282-283)
        if (!harm) {
            const Dist q = dist_of(r2);
            dUdr = dmorse_over_r(P.D_long, P.A_long, q.r, q.rinv);
            if (P.barrier && off_tub && (fj & kFlagOnTubule) == 0)
                dUdr = __fmaf_rn(dbarr(P.a_bl, P.r_bl, P.w_bl, q.r), q.rinv, dUdr);
            if (r2 < kTouch2) dUdr = 0.f;
            if (!(p0.z > rj.z)) gl = fj;
        }
        acc_pair(A, dUdr, d, wi);
        if (r2 < 1.0f)
            acc_bend(P, A, rmon, uj.w - p1.w, rj.w - p0.w, thj - theta, (gl & kFlagGtp) ? P.th0_gtp : P.th0_gdp);
    }
    return A;
}

// Morse lateral bonds of bead g (src/compute_cuda.cu:303-467) with seam
// coefficient and barrier; l1, l2: the bead's own sites.
__device__ __forceinline__ Acc lateral_force(const KParams &P, const DevBuffers &B, const NbrView &V, int g, int flags,
                                             float4 p0, float3 l1, float3 l2, const ListHead &H) {
    const int nb = P.nb, ps = V.stride;
    const float4 *fr = V.fr + V.base;
    Acc A = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const bool off_tub = (flags & kFlagOnTubule) == 0;
#pragma unroll 1
    for (int k = 0; k < H.nt; k++) {
        const int e = k == 0 ? H.e_t0 : B.lat[k * nb + g];
        const bool neg = e <= 0;
        int pj = e < 0 ? -e : e;
        if (pj == kZeroCode) pj = 0;
        const float4 rj = fr[pj];
        const float4 sj = neg ? fr[3 * ps + pj] : fr[2 * ps + pj];
        const int fj = V.fl[V.base + pj];
        const float3 wi = neg ? l1 : l2;
        const float3 d = site_delta(p0, rj, wi, f3(sj));
        const float r2 = norm2(d);
        const Dist q = dist_of(r2);
        float dUdr = dmorse_over_r(((flags ^ fj) & kFlagBeta) ? P.D_lat_seam : P.D_lat, P.A_lat, q.r, q.rinv);
        if (P.barrier && off_tub && (fj & kFlagOnTubule) == 0)
            dUdr = __fmaf_rn(dbarr(P.a_bt, P.r_bt, P.w_bt, q.r), q.rinv, dUdr);
        if (r2 < kTouch2) dUdr = 0.f;
        acc_pair(A, dUdr, d, wi);
    }
    return A;
}

// sin and cos of psi and theta: the Euler axes of the torque.
struct Euler {
    float sp, cp, st, ct;
};
__device__ __forceinline__ Euler euler(float psi, float theta) {
    Euler E;
    sincosf(psi, &E.sp, &E.cp);
    sincosf(theta, &E.st, &E.ct);
    return E;
}
// The generalised force from its parts, which are summed in this order in
// every kernel: axial bonds A, lateral bonds T, LJ L; then the cylindrical
// walls (src/compute_cuda.cu:497-517), and the bending terms plus the torque
// projected on the Euler axes (psi about z, theta about Rz(psi) y, fi about
// R x).  out = (fx, fy, fz, ffi, ftheta, fpsi).
__device__ __forceinline__ void force_out(const KParams &P, const Acc &A, const Acc &T, float3 L, const float *zs,
                                          float4 p0, const Euler &E, float out[6]) {
    float fx = __fadd_rn(__fadd_rn(A.fx, T.fx), L.x), fy = __fadd_rn(__fadd_rn(A.fy, T.fy), L.y),
          fz = __fadd_rn(__fadd_rn(A.fz, T.fz), L.z);
    const float tx = __fadd_rn(A.tx, T.tx), ty = __fadd_rn(A.ty, T.ty), tz = __fadd_rn(A.tz, T.tz);
    if (P.is_wall) {
        const float z = p0.z, top = __fadd_rn(*zs, P.lb);
        if (z < P.lb)
            fz = __fmaf_rn(P.rep_eps, fabsf(z - P.lb), fz);
        else if (z > top)
            fz = __fmaf_rn(-P.rep_eps, fabsf(z - top), fz);
        const float rad2 = __fmaf_rn(p0.x, p0.x, __fmul_rn(p0.y, p0.y));
        if (rad2 > P.rep_r * P.rep_r) {
            const float rad = __fsqrt_rn(rad2);
            const float coeff = __fdiv_rn(__fmul_rn(-P.rep_eps, __fsub_rn(rad, P.rep_r)), rad);
            fx = __fmaf_rn(p0.x, coeff, fx);
            fy = __fmaf_rn(p0.y, coeff, fy);
        }
    }
    out[0] = fx;
    out[1] = fy;
    out[2] = fz;
    const float tf =
        __fmaf_rn(__fmul_rn(E.cp, E.ct), tx, __fmaf_rn(__fmul_rn(E.sp, E.ct), ty, -__fmul_rn(E.st, tz)));
    out[3] = __fadd_rn(A.ffi, tf);
    out[4] = __fadd_rn(A.fth, __fmaf_rn(E.cp, ty, -__fmul_rn(E.sp, tx)));
    out[5] = __fadd_rn(A.fpsi, tz);
}

// Generalised force on bead g (compute_kernel, src/compute_cuda.cu:32-525).
__device__ __forceinline__ void bead_forces(const KParams &P, const DevBuffers &B, const NbrView &V, int g,
                                            const float *zs, int flags, const Frame &Fi, const ListHead &H,
                                            float out[6]) {
    const float3 L = lj_force(P, B, V, g, Fi.p0, H);
    const Acc T = lateral_force(P, B, V, g, flags, Fi.p0, f3(Fi.p2), f3(Fi.p3), H);
    const Acc A = axial_force(P, B, V, g, flags, Fi.p0, Fi.p1, Fi.p2.w, H);
    force_out(P, A, T, L, zs, Fi.p0, euler(Fi.p1.w, Fi.p2.w), out);
}

__device__ __forceinline__ Frame load_frame(const float4 *planes, int nb, int g) {
    Frame F;
    F.p0 = planes[g];
    F.p1 = planes[nb + g];
    F.p2 = planes[2 * nb + g];
    F.p3 = planes[3 * nb + g];
    return F;
}

// Euler-Maruyama update of one moving bead (integrate_kernel,
// src/compute_cuda.cu:955-963): xyz from normals gx, angles from ga.
// Explicitly rounded, like make_frame, so that every kernel gets the same bits.
__device__ __forceinline__ float em_rn(float x, float k, float f, float v, float g) {
    return __fadd_rn(x, __fadd_rn(__fmul_rn(k, f), __fmul_rn(v, g)));
}
__device__ __forceinline__ Frame em_update(const KParams &P, const Frame &Fi, const float f[6], float4 gx,
                                           float4 ga) {
    const float x = em_rn(Fi.p0.x, P.kr, f[0], P.varR, gx.x);
    const float y = em_rn(Fi.p0.y, P.kr, f[1], P.varR, gx.y);
    const float z = em_rn(Fi.p0.z, P.kr, f[2], P.varR, gx.z);
    const float fi = em_rn(Fi.p0.w, P.kfi, f[3], P.nfi, ga.x);
    const float psi = em_rn(Fi.p1.w, P.kfi, f[5], P.nfi, ga.y);
    const float th = em_rn(Fi.p2.w, P.kth, f[4], P.varTheta, ga.z);
    return make_frame(P, x, y, z, fi, th, psi);
}

// One MD step of one bead per thread.  Bound by the latency of the chain list
// entry -> neighbour frame -> force, so everything that does not depend on
// another bead (list heads, noise states) is requested first and the noise is
// drawn while the neighbours are on their way.  AHEAD: the state and lists of the beads that an
// SM takes next but for one CTA are asked into L2; from kAheadBeads beads on, where they
// (250 bytes a bead) do not stay there from step to step: 1024 uneven trajectories
// of up to 3560 beads 138 -> 134 us a step, 512 x 1520 beads 65.3 -> 64.0; 486,000 beads 42.2
// and 42.6.
// kAheadBy: the beads of one CTA of the default block on each of a GB300's SMs (a distance, not a bound: another
// block or device asks a little earlier or later).
constexpr int kAheadBeads = 500000, kAheadBy = 152 * 128;
template <bool KEEP_FORCES, bool AHEAD>
__global__ void __launch_bounds__(256, 4) k_step_plain(KParams P, DevBuffers B) {
    chain_wait();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const int nb = P.nb;
    if (AHEAD) {
        const int a = min(g + kAheadBy, nb - 1);
        auto ask = [](const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); };
#pragma unroll
        for (int k = 0; k < 4; k++) ask(B.frame_in + (size_t)k * nb + a);
        ask(B.seeds + a);
        ask(B.seeds + nb + a);
        ask(B.flags + a);
        ask(B.base + a);
        ask(B.lonc + a);
        ask(B.latc + a);
        ask(B.ljc + a);
        ask(B.harm + (size_t)a * P.maxH);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k < P.maxLJ) ask(B.lj + (size_t)k * nb + a);
    }
    const int flags = B.flags[g];
    const NbrView V = {B.frame_in, B.flags, nb, B.base[g]};
    Frame Fi = load_frame(B.frame_in, nb, g);
    float f[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (!(flags & kFlagExtra)) {
        const bool moving = !(flags & kFlagFixed);
        if (moving || KEEP_FORCES) {
            const ListHead H = list_head(P, B, g);
            float4 gx, ga;
            if (moving) {
                uint4 s1 = B.seeds[g], s2 = B.seeds[nb + g];
                gx = gauss4(s1);
                ga = gauss4(s2);
                B.seeds[g] = s1;
                B.seeds[nb + g] = s2;
            }
            const float *zs = P.is_wall ? B.zs + B.traj[g] : B.zs;
            bead_forces(P, B, V, g, zs, flags, Fi, H, f);
            if (moving) Fi = em_update(P, Fi, f, gx, ga);
        }
    }
    store_frame(B.frame_out, nb, g, Fi);
    if (KEEP_FORCES) {
        B.force[g] = make_float4(f[0], f[1], f[2], 0.f);
        B.force[nb + g] = make_float4(f[3], f[4], f[5], 0.f);
    }
}

// ------------------------------------------------------- persistent period
// A whole run of plain steps between two pair-list rebuilds in one launch, for
// trajectories too large for k_period_split: one CTA per trajectory keeps the trajectory's frames (the four planes) and
// flags in shared memory across the steps, so every neighbour gather of the
// force loop is a shared-memory load; the pair lists and noise streams stay
// in global memory (L2).  Each step is a force phase over the CTA's beads, a
// barrier, the Euler-Maruyama update of every moving bead into shared
// memory, and a barrier; trajectories never interact, so no grid-wide
// synchronisation is needed.  The arithmetic is bead_forces / em_update, as in
// k_step_plain: the result equals that of nsteps launches of k_step_plain bit
// for bit.  At the end the frames go to the buffer the engine's step parity
// expects (frame_out for an odd number of steps, frame_in otherwise).
template <bool KEEP_FORCES>
__global__ void __launch_bounds__(kPeriodThreads, 2) k_step_period(KParams P, DevBuffers B, int nsteps, int nmax,
                                                                   int rebuild) {
    extern __shared__ float4 s_dyn[];
    const int traj = blockIdx.x;
    const int base = B.off[traj], n = B.off[traj + 1] - base;
    const int nb = P.nb, nt = blockDim.x;
    float4 *sf = s_dyn;                                       // plane k of bead j at sf[k * n + j]
    int *sfl = reinterpret_cast<int *>(s_dyn + 4 * (size_t)nmax);
    for (int j = threadIdx.x; j < n; j += nt) {
        const int g = base + j;
        sf[j] = B.frame_in[g];
        sf[n + j] = B.frame_in[nb + g];
        sf[2 * n + j] = B.frame_in[2 * nb + g];
        sf[3 * n + j] = B.frame_in[3 * nb + g];
        sfl[j] = B.flags[g];
    }
    __syncthreads();
    if (rebuild) {
        // the pair lists of this state first, from the frames in shared
        // memory: every bead against the trajectory in ascending j, the
        // decisions of k_rebuild (the same lists)
        // beads farther apart than every cutoff (plus a margin over the
        // rounding of the distance) are skipped before the full decisions
        const float reach = fmaxf(P.lj_on ? P.ljcut : 0.f, P.is_assembly ? kPairPrefilter : 0.f) + 0.05f;
        const float reach2 = reach * reach;
        for (int il = threadIdx.x; il < n; il += nt) {
            const int g = base + il;
            const ListSite I = list_site(P, sf[il], sf[n + il], sf[2 * n + il], sf[3 * n + il], sfl[il], il,
                                         B.harm[g * P.maxH]);
            int nlj = 0, nlo = 0, nla = 0;
            bool overflow = false;
            if (I.do_lj || I.do_pairs)
                for (int jl = 0; jl < n; jl++) {
                    const float4 q = sf[jl];
                    const float dx = q.x - I.p.x, dy = q.y - I.p.y, dz = q.z - I.p.z;
                    if (dx * dx + dy * dy + dz * dz > reach2) continue;
                    const unsigned bits = list_bits(P, I, jl, q, sf[n + jl], sf[2 * n + jl], sf[3 * n + jl], sfl[jl]);
                    list_append(P, B, g, I, bits, jl, nlj, nlo, nla, overflow);
                }
            if (P.lj_on) B.ljc[g] = min(nlj, P.maxLJ);
            if (P.is_assembly) {
                B.lonc[g] = min(nlo, P.maxLong);
                B.latc[g] = min(nla, P.maxLat);
            }
            if (overflow) atomicOr(B.err, kErrOverflow);
        }
        __syncthreads();
    }
    const NbrView V = {sf, sfl, n, 0};
    float f[kPeriodBeads][6];
    for (int step = 0; step < nsteps; step++) {
#pragma unroll
        for (int q = 0; q < kPeriodBeads; q++) {
            const int j = threadIdx.x + q * nt;
#pragma unroll
            for (int c = 0; c < 6; c++) f[q][c] = 0.f;
            if (j < n) {
                const int fl = sfl[j];
                if (!(fl & kFlagExtra) && (KEEP_FORCES || !(fl & kFlagFixed))) {
                    Frame Fi;
                    Fi.p0 = sf[j];
                    Fi.p1 = sf[n + j];
                    Fi.p2 = sf[2 * n + j];
                    Fi.p3 = sf[3 * n + j];
                    bead_forces(P, B, V, base + j, B.zs + traj, fl, Fi, list_head(P, B, base + j), f[q]);
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kPeriodBeads; q++) {
            const int j = threadIdx.x + q * nt;
            if (j >= n) continue;
            const int fl = sfl[j], g = base + j;
            if (!(fl & (kFlagExtra | kFlagFixed))) {
                Frame Fi;
                Fi.p0 = sf[j];
                Fi.p1 = sf[n + j];
                Fi.p2 = sf[2 * n + j];
                Fi.p3 = sf[3 * n + j];
                uint4 s1 = B.seeds[g], s2 = B.seeds[nb + g];
                const float4 gx = gauss4(s1), ga = gauss4(s2);
                B.seeds[g] = s1;
                B.seeds[nb + g] = s2;
                Fi = em_update(P, Fi, f[q], gx, ga);
                sf[j] = Fi.p0;
                sf[n + j] = Fi.p1;
                sf[2 * n + j] = Fi.p2;
                sf[3 * n + j] = Fi.p3;
            }
            if (KEEP_FORCES && step == nsteps - 1) {
                B.force[g] = make_float4(f[q][0], f[q][1], f[q][2], 0.f);
                B.force[nb + g] = make_float4(f[q][3], f[q][4], f[q][5], 0.f);
            }
        }
        __syncthreads();
    }
    float4 *out = (nsteps & 1) ? B.frame_out : B.frame_in;
    for (int j = threadIdx.x; j < n; j += nt) {
        const int g = base + j;
        out[g] = sf[j];
        out[nb + g] = sf[n + j];
        out[2 * nb + g] = sf[2 * n + j];
        out[3 * nb + g] = sf[3 * n + j];
    }
}

// The random force of bead g for TEA from stream g, scaled by sqrt(2 kB T gammaR /
// dt) (integrateTea_prepare, src/bdhitea_kernel.cu:16-36).
__device__ __forceinline__ float4 tea_random(const KParams &P, const DevBuffers &B, int g) {
    uint4 s = B.seeds[g];
    float4 r = gauss4(s);
    B.seeds[g] = s;
    r.x *= P.tea_var;
    r.y *= P.tea_var;
    r.z *= P.tea_var;
    B.tea_r[g] = r;
    return r;
}

// Forces only (for output and the TEA path).  With TEA_PREPARE it also draws
// the random force of every bead and lays the bead out for the all-pairs pass.
template <bool TEA_PREPARE>
__global__ void __launch_bounds__(256) k_forces(KParams P, DevBuffers B) {
    chain_wait();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const int nb = P.nb;
    const int flags = B.flags[g];
    float f[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const Frame Fi = load_frame(B.frame_in, nb, g);
    if (!(flags & kFlagExtra)) {
        const NbrView V = {B.frame_in, B.flags, nb, B.base[g]};
        const ListHead H = list_head(P, B, g);
        bead_forces(P, B, V, g, P.is_wall ? B.zs + B.traj[g] : B.zs, flags, Fi, H, f);
    }
    B.force[g] = make_float4(f[0], f[1], f[2], 0.f);
    B.force[nb + g] = make_float4(f[3], f[4], f[5], 0.f);
    if (TEA_PREPARE) {
        const float4 r = tea_random(P, B, g);
        tea_pack_bead(B, g, (flags & kFlagExtra) != 0, Fi.p0, f[0], f[1], f[2], r);
    }
}

// ------------------------------------------------ four warps for 32 beads
// k_step_plain and k_forces for batches that leave most of the GPU idle, where a
// step lasts as long as one bead's serial chain: a CTA of four warps serves 32
// beads, warp 0 their axial bonds, warp 1 the lateral bonds, warp 2 the LJ
// neighbours, warp 3 the noise and the Euler axes; the parts meet in shared
// memory and warp 3 sums them (force_out) and moves the beads.  The same
// functions and order of sums as the one-thread form: the same bits.
constexpr int kSplitBeads = 32, kSplitThreads = 128;
enum { kPartA = 0, kPartT = 9, kPartL = 15, kParts = 18 };
__device__ __forceinline__ void put_axial(float (*s)[kSplitBeads], int l, const Acc &A) {
    const float v[9] = {A.fx, A.fy, A.fz, A.ffi, A.fpsi, A.fth, A.tx, A.ty, A.tz};
#pragma unroll
    for (int c = 0; c < 9; c++) s[kPartA + c][l] = v[c];
}
__device__ __forceinline__ void put_lateral(float (*s)[kSplitBeads], int l, const Acc &T) {
    const float v[6] = {T.fx, T.fy, T.fz, T.tx, T.ty, T.tz};
#pragma unroll
    for (int c = 0; c < 6; c++) s[kPartT + c][l] = v[c];
}
__device__ __forceinline__ void get_parts(float (*s)[kSplitBeads], int l, Acc &A, Acc &T, float3 &L) {
    A = {s[0][l], s[1][l], s[2][l], s[3][l], s[4][l], s[5][l], s[6][l], s[7][l], s[8][l]};
    T = {s[9][l], s[10][l], s[11][l], 0.f, 0.f, 0.f, s[12][l], s[13][l], s[14][l]};
    L = make_float3(s[15][l], s[16][l], s[17][l]);
}
// STEP: the Euler-Maruyama step of k_step_plain; otherwise the forces (TEA:
// with the random force of every bead).
template <bool STEP, bool KEEP_FORCES, bool TEA>
__global__ void __launch_bounds__(kSplitThreads) k_split(KParams P, DevBuffers B) {
    __shared__ float s_part[kParts][kSplitBeads];
    const int role = threadIdx.x >> 5, l = threadIdx.x & 31, g = blockIdx.x * kSplitBeads + l;
    const int nb = P.nb;
    const bool valid = g < nb;
    const int base = valid && role < 3 ? B.base[g] : 0;
    chain_wait();   // no kernel writes what was read so far
    const int flags = valid ? B.flags[g] : kFlagExtra;
    const bool moving = !(flags & (kFlagExtra | kFlagFixed));
    const bool work = STEP && !KEEP_FORCES ? moving : !(flags & kFlagExtra);
    float4 gx, ga, rt;
    Frame Fi;
    Euler E;
    NbrView V;
    ListHead H;
    if (role < 3) {
        if (work) {
            V = {B.frame_in, B.flags, nb, base};
            H = list_head(P, B, g);
            const float4 p0 = B.frame_in[g];
            if (role == 0) {
                put_axial(s_part, l, axial_force(P, B, V, g, flags, p0, B.frame_in[nb + g], B.frame_in[2 * nb + g].w, H));
            } else if (role == 1) {
                put_lateral(s_part, l,
                            lateral_force(P, B, V, g, flags, p0, f3(B.frame_in[2 * nb + g]), f3(B.frame_in[3 * nb + g]), H));
            } else {
                const float3 L = lj_force(P, B, V, g, p0, H);
                s_part[kPartL][l] = L.x;
                s_part[kPartL + 1][l] = L.y;
                s_part[kPartL + 2][l] = L.z;
            }
        }
    } else if (valid) {
        Fi = load_frame(B.frame_in, nb, g);
        if (STEP && moving) {
            uint4 s1 = B.seeds[g], s2 = B.seeds[nb + g];
            gx = gauss4(s1);
            ga = gauss4(s2);
            B.seeds[g] = s1;
            B.seeds[nb + g] = s2;
        }
        if (TEA) rt = tea_random(P, B, g);
        if (work) E = euler(Fi.p1.w, Fi.p2.w);
    }
    __syncthreads();
    if (role < 3 || !valid) return;
    float f[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (work) {
        Acc A, T;
        float3 L;
        get_parts(s_part, l, A, T, L);
        force_out(P, A, T, L, P.is_wall ? B.zs + B.traj[g] : B.zs, Fi.p0, E, f);
    }
    if (STEP) {
        if (moving) Fi = em_update(P, Fi, f, gx, ga);
        store_frame(B.frame_out, nb, g, Fi);
    }
    if (!STEP || KEEP_FORCES) {
        B.force[g] = make_float4(f[0], f[1], f[2], 0.f);
        B.force[nb + g] = make_float4(f[3], f[4], f[5], 0.f);
    }
    if (TEA) tea_pack_bead(B, g, (flags & kFlagExtra) != 0, Fi.p0, f[0], f[1], f[2], rt);
}

// --------------------------------------- persistent period, four warps a bead group
// k_step_period for trajectories of up to kPeriodSplitBeads beads: the roles of
// k_split inside one CTA per trajectory that keeps the frames (two buffers) in
// shared memory across the steps.  A step is the serial chain of one bead, so it is
// cut by role: three groups of warps take the axial bonds, the lateral bonds and
// the LJ neighbours while the fourth takes the Euler axes; after a barrier the fourth sums
// the parts and moves the beads while the lateral and LJ groups draw the noise of
// the next step; list heads and noise states stay in registers.  The pair lists are rebuilt
// first when due, a quarter of the trajectory for each of a bead's four threads.
// The same functions, order of sums and list order as the other forms: the same bits.
// One 156-bead seed: 7.1 us a step with one thread a bead, 3.1 us so (10 steps and
// a rebuild a launch).
constexpr int kPeriodSplitBeads = 192;   // 768 threads of 80 registers (256 beads would leave 64 and spill)
struct PeriodSplitSmem {   // offsets in bytes; s: beads rounded up to a warp
    int frames, noise, parts, flags, total;
    __host__ __device__ explicit PeriodSplitSmem(int s) {
        frames = 0;
        noise = frames + 2 * 4 * 16 * s;
        parts = noise + 2 * 2 * 16 * s;
        flags = parts + kParts * 4 * s;
        total = flags + 4 * s;
    }
};
template <bool KEEP_FORCES>
__global__ void __launch_bounds__(4 * kPeriodSplitBeads) k_period_split(KParams P, DevBuffers B, int nsteps,
                                                                        int rebuild, ListCuts cut) {
    chain_wait();
    extern __shared__ float4 s_dyn[];
    char *smem = reinterpret_cast<char *>(s_dyn);
    const int S = blockDim.x >> 2, role = threadIdx.x / S, l = threadIdx.x % S;
    const PeriodSplitSmem at(S);
    const int traj = blockIdx.x, base = B.off[traj], n = B.off[traj + 1] - base, nb = P.nb, g = base + l;
    float4 *s_fr = reinterpret_cast<float4 *>(smem + at.frames);     // plane k of bead j of buffer b at [(4 b + k) S + j]
    float4 *s_noise = reinterpret_cast<float4 *>(smem + at.noise);   // [2 parity + (xyz, angles)][S]
    float *s_part = reinterpret_cast<float *>(smem + at.parts);      // [kParts][S]
    int *s_fl = reinterpret_cast<int *>(smem + at.flags);
    const bool valid = l < n;
    if (valid) {   // role k copies plane k, into both buffers (beads that never move stay as they are)
        const float4 p = B.frame_in[role * nb + g];
        s_fr[role * S + l] = p;
        s_fr[(4 + role) * S + l] = p;
        if (role == 0) s_fl[l] = B.flags[g];
    }
    __syncthreads();
    const int flags = valid ? s_fl[l] : kFlagExtra;
    if (rebuild) {
        // exact decisions on squared distances (sq_below): the near ones of a
        // quarter first, as a mask, then their lists, four bits each
        const int quarter = (n + 3) / 4, j0 = min(n, role * quarter), j1 = min(n, j0 + quarter);   // at most 48 beads
        int *s_cnt = reinterpret_cast<int *>(s_part);   // [3][4][S]
        ListSite I;
        unsigned long long near = 0, got[3] = {0, 0, 0};
        int c[3] = {0, 0, 0};
        bool overflow = false;
        if (valid) {
            I = list_site(P, s_fr[l], s_fr[S + l], s_fr[2 * S + l], s_fr[3 * S + l], flags, l, B.harm[g * P.maxH]);
            const float t_near = fmaxf(I.do_lj ? cut.lj : 0.f, I.do_pairs ? cut.pair : 0.f);
            unsigned lo = 0, hi = 0;
#pragma unroll 4
            for (int j = j0; j < j1; j++) {
                const unsigned bit = dist2_rn(I.p, s_fr[j]) < t_near ? 1u << ((j - j0) & 31) : 0u;
                if (j - j0 < 32)
                    lo |= bit;
                else
                    hi |= bit;
            }
            near = (unsigned long long)hi << 32 | lo;
            int k = 0;
            for (unsigned long long m = near; m; m &= m - 1, k++) {
                const int j = j0 + __ffsll((long long)m) - 1;
                const unsigned bits = list_bits_sq(I, j, s_fr[j], s_fr[S + j], s_fr[2 * S + j], s_fr[3 * S + j],
                                                   s_fl[j], cut);
                c[0] += bits & 1u;
                c[1] += (bits >> 1) & 1u;
                c[2] += ((bits >> 2) & 1u) + (bits >> 3);
                const unsigned long long at16 = (unsigned long long)bits << (4 * (k & 15));
                got[0] |= k < 16 ? at16 : 0;   // 48 beads, 16 a word
                got[1] |= k >= 16 && k < 32 ? at16 : 0;
                got[2] |= k >= 32 ? at16 : 0;
            }
        }
#pragma unroll
        for (int k = 0; k < 3; k++) s_cnt[(4 * k + role) * S + l] = c[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; k++) {
            c[k] = 0;
            for (int r = 0; r < role; r++) c[k] += s_cnt[(4 * k + r) * S + l];
        }
        if (valid) {
            int k = 0;
            for (unsigned long long m = near; m; m &= m - 1, k++) {
                const unsigned bits = (unsigned)((k < 16 ? got[0] : k < 32 ? got[1] : got[2]) >> (4 * (k & 15))) & 15u;
                list_append(P, B, g, I, bits, j0 + __ffsll((long long)m) - 1, c[0], c[1], c[2], overflow);
            }
            if (role == 3) {   // the last quarter ends with the totals
                if (P.lj_on) B.ljc[g] = min(c[0], P.maxLJ);
                if (P.is_assembly) {
                    B.lonc[g] = min(c[1], P.maxLong);
                    B.latc[g] = min(c[2], P.maxLat);
                }
            }
            if (overflow) atomicOr(B.err, kErrOverflow);
        }
        __syncthreads();
    }
    const bool moving = !(flags & (kFlagExtra | kFlagFixed));
    const bool work = KEEP_FORCES ? !(flags & kFlagExtra) : moving;
    ListHead H = {};
    if (role < 3 && work) H = list_head(P, B, g);
    // the noise of the lateral (angles) and LJ (xyz) groups' beads
    uint4 seed = make_uint4(0u, 0u, 0u, 0u);
    const bool draws = (role == 1 || role == 2) && moving;
    uint4 *my_seed = B.seeds + (role == 1 ? nb + g : g);
    if (draws) {
        seed = *my_seed;
        s_noise[(role == 1 ? S : 0) + l] = gauss4(seed);
    }
    float f[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int step = 0; step < nsteps; step++) {
        const float4 *fr = s_fr + 4 * S * (step & 1);
        const NbrView V = {fr, s_fl, S, 0};
        Euler E;
        if (work) {
            const float4 p0 = fr[l];
            if (role == 0) {
                const Acc A = axial_force(P, B, V, g, flags, p0, fr[S + l], fr[2 * S + l].w, H);
                const float v[9] = {A.fx, A.fy, A.fz, A.ffi, A.fpsi, A.fth, A.tx, A.ty, A.tz};
#pragma unroll
                for (int k = 0; k < 9; k++) s_part[(kPartA + k) * S + l] = v[k];
            } else if (role == 1) {
                const Acc T = lateral_force(P, B, V, g, flags, p0, f3(fr[2 * S + l]), f3(fr[3 * S + l]), H);
                const float v[6] = {T.fx, T.fy, T.fz, T.tx, T.ty, T.tz};
#pragma unroll
                for (int k = 0; k < 6; k++) s_part[(kPartT + k) * S + l] = v[k];
            } else if (role == 2) {
                const float3 L = lj_force(P, B, V, g, p0, H);
                s_part[kPartL * S + l] = L.x;
                s_part[(kPartL + 1) * S + l] = L.y;
                s_part[(kPartL + 2) * S + l] = L.z;
            } else {
                E = euler(fr[S + l].w, fr[2 * S + l].w);
            }
        }
        __syncthreads();
        if (role == 3 && work) {
            Frame Fi;
            Fi.p0 = fr[l];
            Fi.p1 = fr[S + l];
            Fi.p2 = fr[2 * S + l];
            float v[kParts];
#pragma unroll
            for (int k = 0; k < kParts; k++) v[k] = s_part[k * S + l];
            const Acc A = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]};
            const Acc T = {v[9], v[10], v[11], 0.f, 0.f, 0.f, v[12], v[13], v[14]};
            force_out(P, A, T, make_float3(v[15], v[16], v[17]), B.zs + traj, Fi.p0, E, f);
            if (moving) {
                const float4 *noise = s_noise + 2 * S * (step & 1);
                Fi = em_update(P, Fi, f, noise[l], noise[S + l]);
                float4 *to = s_fr + 4 * S * ((step & 1) ^ 1);
                to[l] = Fi.p0;
                to[S + l] = Fi.p1;
                to[2 * S + l] = Fi.p2;
                to[3 * S + l] = Fi.p3;
            }
        } else if (draws && step + 1 < nsteps) {
            s_noise[2 * S * ((step & 1) ^ 1) + (role == 1 ? S : 0) + l] = gauss4(seed);
        }
        __syncthreads();
    }
    if (draws) *my_seed = seed;
    if (!valid) return;
    float4 *out = (nsteps & 1) ? B.frame_out : B.frame_in;
    out[role * nb + g] = s_fr[(4 * (nsteps & 1) + role) * S + l];
    if (KEEP_FORCES && role == 3) {
        B.force[g] = make_float4(f[0], f[1], f[2], 0.f);
        B.force[nb + g] = make_float4(f[3], f[4], f[5], 0.f);
    }
}

// ------------------------------------------------------------- energies
// energy_kernel (src/compute_cuda.cu:676-911): per-bead FP32 terms, halved;
// block partial sums in FP64 over one trajectory chunk.
__global__ void __launch_bounds__(kTile) k_energy(KParams P, DevBuffers B, const int2 *work, double *per_bead,
                                                  double *partials) {
    const int2 w = work[blockIdx.x];
    const int traj = w.x, base = B.off[traj], end = B.off[traj + 1];
    const int g = w.y + threadIdx.x;
    const int nb = P.nb;
    const float4 *fr = B.frame_in;
    float U[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (g < end) {
        const int flags = B.flags[g];
        if (!(flags & kFlagExtra)) {
            const Frame Fi = load_frame(fr, nb, g);
            const float3 uzi = f3(Fi.p1);
            const bool off_tub = (flags & kFlagOnTubule) == 0;
            const int hc = (flags >> kHarmShift) & 7;
            for (int k = 0; k < hc; k++) {
                const int e = B.harm[g * P.maxH + k];
                const float rmon = e < 0 ? 2.0f : -2.0f;
                const int pj = base + (e < 0 ? -e : e);
                const float4 rj = fr[pj], uj = fr[nb + pj];
                const float3 d = site_delta(Fi.p0, rj, make_float3(uzi.x * rmon, uzi.y * rmon, uzi.z * rmon),
                                            make_float3(-uj.x * rmon, -uj.y * rmon, -uj.z * rmon));
                const float dr = norm3_rn(d);
                U[0] += (P.C / 2.0f) * dr * dr;
                if (dr < 1.0f) {
                    // psi_ij, fi_ij, theta_ji (src/compute_cuda.cu:751-756)
                    const float th0 = (flags & kFlagGtp) ? P.th0_gtp : P.th0_gdp;
                    U[3] += P.B_psi * (1.0f - cosf((Fi.p1.w - uj.w) - P.psi_0));
                    U[4] += P.B_fi * (1.0f - cosf((Fi.p0.w - rj.w) - P.fi_0));
                    U[5] += P.B_theta * (1.0f - cosf((fr[2 * nb + pj].w - Fi.p2.w) - th0));
                }
            }
            const int nl = B.lonc[g];
            for (int k = 0; k < nl; k++) {
                const int e = B.lon[k * nb + g];
                const float rmon = e < 0 ? 2.0f : -2.0f;
                const int pj = base + (e < 0 ? -e : e);
                const float4 rj = fr[pj], uj = fr[nb + pj];
                const float3 d = site_delta(Fi.p0, rj, make_float3(uzi.x * rmon, uzi.y * rmon, uzi.z * rmon),
                                            make_float3(-uj.x * rmon, -uj.y * rmon, -uj.z * rmon));
                const float dr = norm3_rn(d);
                U[1] += morse_en(P.D_long, P.A_long, dr);
                const int fj = B.flags[pj];
                if (P.barrier && off_tub && (fj & kFlagOnTubule) == 0) U[1] += barr(P.a_bl, P.r_bl, P.w_bl, dr);
                if (dr < 1.0f) {
                    const int glast = (Fi.p0.z > rj.z) ? flags : fj;
                    const float th0 = (glast & kFlagGtp) ? P.th0_gtp : P.th0_gdp;
                    U[3] += P.B_psi * (1.0f - cosf((Fi.p1.w - uj.w) - P.psi_0));
                    U[4] += P.B_fi * (1.0f - cosf((Fi.p0.w - rj.w) - P.fi_0));
                    U[5] += P.B_theta * (1.0f - cosf((Fi.p2.w - fr[2 * nb + pj].w) - th0));
                }
            }
            const int nt = B.latc[g];
            for (int k = 0; k < nt; k++) {
                const int e = B.lat[k * nb + g];
                const bool neg = e <= 0;
                int j = e < 0 ? -e : e;
                if (j == kZeroCode) j = 0;
                const int pj = base + j;
                const float4 rj = fr[pj];
                const float4 sj = neg ? fr[3 * nb + pj] : fr[2 * nb + pj];
                const float3 d = site_delta(Fi.p0, rj, neg ? f3(Fi.p2) : f3(Fi.p3), f3(sj));
                const float dr = norm3_rn(d);
                const int fj = B.flags[pj];
                U[2] += morse_en(((flags ^ fj) & kFlagBeta) ? P.D_lat_seam : P.D_lat, P.A_lat, dr);
                if (P.barrier && off_tub && (fj & kFlagOnTubule) == 0) U[2] += barr(P.a_bt, P.r_bt, P.w_bt, dr);
            }
            if (P.lj_on) {
                const int n = B.ljc[g];
                for (int k = 0; k < n; k++) {
                    const float4 rj = fr[base + B.lj[k * nb + g]];
                    const float dx = Fi.p0.x - rj.x, dy = Fi.p0.y - rj.y, dz = Fi.p0.z - rj.z;
                    const float dr2 = dx * dx + dy * dy + dz * dz;
                    if (sqrtf(dr2) < 6.0f) U[6] += P.lj_pref / (dr2 * dr2 * dr2);
                }
            }
        }
        if (per_bead) {
            for (int c = 0; c < 7; c++) per_bead[7 * (size_t)g + c] = (double)(U[c] / 2.0f);
        }
    }
    // FP64 block reduction: warp shuffles, then one warp over the warp sums.
    __shared__ double red[kTile / 32][7];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c = 0; c < 7; c++) {
        double v = (double)(U[c] / 2.0f);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[wid][c] = v;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double v = 0.0;
        for (int w2 = 0; w2 < kTile / 32; w2++) v += red[w2][threadIdx.x];
        partials[7 * (size_t)blockIdx.x + threadIdx.x] = v;
    }
}

// Per-trajectory totals: fixed-order sum of the trajectory's block partials, one
// thread for each term, eight partials requested at a time.  (One thread for a
// trajectory waited for memory at every block: 97 trajectories of up to 2684
// beads 16 us, 5 us so.)
constexpr int kEnergyTerms = 7;
__global__ void k_energy_totals(int nt, const double *partials, const int *work_first, double *per_traj,
                                int *err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, t = k / kEnergyTerms, c = k % kEnergyTerms;
    if (t >= nt) return;
    const int last = work_first[t + 1];
    double s = 0;
    for (int w = work_first[t]; w < last; w += 8) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = w + u < last ? partials[kEnergyTerms * (size_t)(w + u) + c] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (w + u < last) s += v[u];
    }
    per_traj[kEnergyTerms * (size_t)t + c] = s;
    // the terms the reference checks (src/updater.cpp:27)
    if (c != 3 && c != 4 && c != 5 && !isfinite(s)) atomicOr(err, kErrNonFinite);
}

// ----------------------------------------------------------- conversions
__global__ void k_frames_from_coords(KParams P, const float *c7, float4 *planes) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const float *c = c7 + 7 * (size_t)g;
    store_frame(planes, P.nb, g, make_frame(P, c[0], c[1], c[2], c[3], c[4], c[5]));
}

__global__ void k_coords_from_frames(int nb, const float4 *planes, float *c7) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nb) return;
    const float4 a = planes[g];
    float *c = c7 + 7 * (size_t)g;
    c[0] = a.x;
    c[1] = a.y;
    c[2] = a.z;
    c[3] = a.w;
    c[4] = planes[2 * nb + g].w;
    c[5] = planes[nb + g].w;
    c[6] = 0.f;
}

__global__ void k_forces_to_coords(int nb, const float4 *force, float *c7) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nb) return;
    const float4 a = force[g], b = force[nb + g];
    float *c = c7 + 7 * (size_t)g;
    c[0] = a.x;
    c[1] = a.y;
    c[2] = a.z;
    c[3] = b.x;
    c[4] = b.y;
    c[5] = b.z;
    c[6] = 0.f;
}

__global__ void k_set_flags(int nb, const uint8_t *extra, const int *gtp, const int *ontub, int *flags) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nb) return;
    int f = flags[g];
    if (extra) f = extra[g] ? (f | kFlagExtra) : (f & ~kFlagExtra);
    if (gtp) f = gtp[g] == 1 ? (f | kFlagGtp) : (f & ~kFlagGtp);
    if (ontub) f = ontub[g] != 0 ? (f | kFlagOnTubule) : (f & ~kFlagOnTubule);
    flags[g] = f;
}

// --------------------------------------------------------------- launchers
static inline int blocks(int n, int t) { return (n + t - 1) / t; }

void launch_frames_from_coords(const KParams &P, const float *c7, float4 *frame, cudaStream_t s) {
    k_frames_from_coords<<<blocks(P.nb, 256), 256, 0, s>>>(P, c7, frame);
}
void launch_coords_from_frames(const KParams &P, const float4 *frame, float *c7, cudaStream_t s) {
    k_coords_from_frames<<<blocks(P.nb, 256), 256, 0, s>>>(P.nb, frame, c7);
}
void launch_forces_to_coords(const KParams &P, const float4 *force, float *c7, cudaStream_t s) {
    k_forces_to_coords<<<blocks(P.nb, 256), 256, 0, s>>>(P.nb, force, c7);
}
void launch_step_plain(const KParams &P, const DevBuffers &B, bool keep_forces, cudaStream_t s) {
    if (P.nb <= kSplitMaxBeads) {
        const int n = blocks(P.nb, kSplitBeads);
        if (keep_forces)
            launch_chained(P, k_split<true, true, false>, n, kSplitThreads, 0, s, P, B);
        else
            launch_chained(P, k_split<true, false, false>, n, kSplitThreads, 0, s, P, B);
        return;
    }
    const int t = P.step_block > 0 ? P.step_block : 128;
    const bool ahead = P.nb >= kAheadBeads;
    const auto kernel = keep_forces ? (ahead ? k_step_plain<true, true> : k_step_plain<true, false>)
                                    : (ahead ? k_step_plain<false, true> : k_step_plain<false, false>);
    launch_chained(P, kernel, blocks(P.nb, t), t, 0, s, P, B);
}
size_t period_smem_bytes(int nmax) { return (size_t)nmax * (4 * sizeof(float4) + sizeof(int)); }
bool period_fits(int nmax) {
    return nmax > 0 && nmax <= kPeriodThreads * kPeriodBeads && period_smem_bytes(nmax) <= kPeriodMaxSmem;
}
int period_prepare(int) {   // the limits of the largest trajectory: engines share the kernels
    const int whole = (int)kPeriodMaxSmem, split = PeriodSplitSmem(kPeriodSplitBeads).total;
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (cudaFuncSetAttribute(k_step_period<false>, attr, whole) != cudaSuccess ||
        cudaFuncSetAttribute(k_step_period<true>, attr, whole) != cudaSuccess ||
        cudaFuncSetAttribute(k_period_split<false>, attr, split) != cudaSuccess ||
        cudaFuncSetAttribute(k_period_split<true>, attr, split) != cudaSuccess)
        return -1;
    return 0;
}
bool period_rebuilds(int nmax) { return nmax <= kPeriodRebuildMax; }
void launch_step_period(const KParams &P, const DevBuffers &B, bool keep_forces, int nsteps, int nmax, bool rebuild,
                        cudaStream_t s) {
    int t = ((nmax + 31) / 32) * 32;
    if (t <= kPeriodSplitBeads) {
        const size_t bytes = PeriodSplitSmem(t).total;
        const ListCuts cut = list_cuts(P);
        if (keep_forces)
            launch_chained(P, k_period_split<true>, P.nt, 4 * t, bytes, s, P, B, nsteps, rebuild ? 1 : 0, cut);
        else
            launch_chained(P, k_period_split<false>, P.nt, 4 * t, bytes, s, P, B, nsteps, rebuild ? 1 : 0, cut);
        return;
    }
    if (t > kPeriodThreads) t = kPeriodThreads;
    const size_t bytes = period_smem_bytes(nmax);
    if (keep_forces)
        k_step_period<true><<<P.nt, t, bytes, s>>>(P, B, nsteps, nmax, rebuild ? 1 : 0);
    else
        k_step_period<false><<<P.nt, t, bytes, s>>>(P, B, nsteps, nmax, rebuild ? 1 : 0);
}

void launch_forces(const KParams &P, const DevBuffers &B, bool tea_prepare, cudaStream_t s) {
    if (P.nb <= kSplitMaxBeads) {
        const int n = blocks(P.nb, kSplitBeads);
        if (tea_prepare)
            launch_chained(P, k_split<false, false, true>, n, kSplitThreads, 0, s, P, B);
        else
            launch_chained(P, k_split<false, false, false>, n, kSplitThreads, 0, s, P, B);
        return;
    }
    if (tea_prepare)
        launch_chained(P, k_forces<true>, blocks(P.nb, 128), 128, 0, s, P, B);
    else
        launch_chained(P, k_forces<false>, blocks(P.nb, 128), 128, 0, s, P, B);
}
void launch_energy(const KParams &P, const DevBuffers &B, double *per_bead, double *partials, const int2 *work,
                   int nwork, cudaStream_t s) {
    k_energy<<<nwork, kTile, 0, s>>>(P, B, work, per_bead, partials);
}
void launch_energy_totals(const KParams &P, const double *partials, const int *work_first, double *per_traj,
                          int *err, cudaStream_t s) {
    k_energy_totals<<<blocks(P.nt * kEnergyTerms, 128), 128, 0, s>>>(P.nt, partials, work_first, per_traj, err);
}
void launch_set_flags(int nb, const uint8_t *extra, const int *gtp, const int *ontub, int *flags, cudaStream_t s) {
    k_set_flags<<<blocks(nb, 256), 256, 0, s>>>(nb, extra, gtp, ontub, flags);
}

}  // namespace mtg
