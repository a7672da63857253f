// kernels_tea.cu - TEA hydrodynamics (Geyer & Winter 2009): the all-pairs
// epsilon / C_i pass, the FP64 epsilon -> beta reduction, and the all-pairs
// RPY mobility product fused with the position update; below them the far
// field of the learned mode.
//
// Both O(N^2) passes are one kernel template, k_tea_pass (k_tea_small for small
// systems, which are bound by latency).  They are bound by
// the FP32 pipe (about 45 FLOP per ordered pair: 24 packed FP32x2 operations
// for two pairs, each pair visited from both its beads), so everything else is arranged to stay off its way:
//   * The beads j come from B.tea_pack, where the force kernel of the step has
//     laid every trajectory out in blocks of 32 beads = 16 pairs in the order the
//     loop reads them: the two lanes of a packed operation are two beads j, one
//     16-byte shared-memory broadcast feeds two operands of both.  A tile of
//     kTeaTileBlocks blocks is copied by cp.async two tiles ahead, one barrier a
//     tile.  Extra beads and padding sit at 1e18 nm with zero F and R: every term they give is zero or
//     below the rounding of the sums.
//   * A CTA of four warps serves 128 beads i, one a thread: 56 registers and nine
//     CTAs an SM (two beads a thread load half as many words but leave six CTAs:
//     1.82 against 1.76 ms).
//   * A bead's sums are cut by its trajectory alone (tea_fine, mtg_internal.cuh), so they have the
//     same bits in every batch and in both kernels.  A CTA takes one grain, a whole
//     node of that tree of sums, for its 128 beads; the grain's size fits the batch
//     (tea_grain_level).  Of a chunk of several grains each CTA leaves its sums, and the one
//     that comes last (an atomic count; nothing waits) adds them in the tree's order and
//     finishes the beads.  (Equal runs of units, cut where k/G of the batch's work is, are
//     2% faster in the product and 1% slower in the epsilon pass, but a bead's bits then depend on the batch.)
// The far-field formula runs for every pair; the few overlapping pairs
// (r <= 2a) are found through a running minimum of r^2 per block; in a block
// that holds one their distances are taken once more and only they get the near-field formula
// in place of the far one.  That one takes r >= 2a, so what is replaced is never larger than the
// sums (at r = 0.14 nm the row sums were 4e-3 off without it, 1e-7 so; 1% of the time).  In
// the block that holds a bead itself its own pair gets r^2 = 1e30: its term is
// then far below the rounding of the sums, and the correction skips it.
// Sums are kept in units of 0.75 a (T' = T / (0.75 a)).
// What the two kernels compute for a bead is written with explicitly rounded operations wherever a product
// meets a sum, so that both give the same bits.
// Measured (mobility product): 64 x 5600 beads 1.71 ms (53 TFLOP/s of the measured 80),
// 16 x 3300 beads 170 us; epsilon pass 1.58 ms and 154 us.
#include "mtg_internal.cuh"

namespace mtg {

constexpr int kTeaThreads = 128;
constexpr int kTeaI = kTeaChunk;            // beads i per CTA
static_assert(kTeaI == kTeaThreads, "one bead a thread");
constexpr int kTeaTileBlocks = 4;           // blocks of a tile
constexpr int kTeaStages = 3;               // tiles in shared memory
constexpr float kFarAway = kTeaFarAway;     // position of padding and extra beads j

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Scaled RPY coefficients (integrateTea_RPY, src/bdhitea_kernel.cu:38-58:
// T = cii I + crr u u^T, ra = r/a; ra > 2: cii = 0.75/ra (1 + 2/(3 ra^2)),
// crr = 0.75/ra (1 - 2/ra^2); otherwise cii = 1 - 9 ra/32, crr = 3 ra/32),
// divided by 0.75 a.  With rinv = 1/r, q = rinv^2, t = q rinv the far field
// is cii' = rinv + (2/3) a^2 t and crr' = rinv - 2 a^2 t.
struct TeaConst {
    float kap, two_a2, four_a2, inv_a, inv_c075a, c075a;
};
__device__ __forceinline__ TeaConst tea_const(float a) {
    return {(2.0f / 3.0f) * a * a, 2.0f * a * a, 4.0f * a * a, 1.0f / a, 1.0f / (0.75f * a), 0.75f * a};
}
// near branch (r <= 2a): scaled cii', crr'
__device__ __forceinline__ void rpy_near(const TeaConst &K, float r2, float rinv, float &cii, float &crr) {
    const float ra = r2 * rinv * K.inv_a;
    cii = __fmaf_rn(-(9.0f / 32.0f), ra, 1.0f) * K.inv_c075a;
    crr = (3.0f / 32.0f) * ra * K.inv_c075a;
}

// Scaled epsilon terms of one pair from cii', crr', q: the row sums of
// squares minus cii'^2 (Bc d_c^2 with Bc = (2 cii' + crr') crr' q), cii'^2, and
// the sum of all nine entries 3 cii' + crr' q (d_x + d_y + d_z)^2.
struct EpsTerms {
    float bx, by, bz, a2, w;
};
__device__ __forceinline__ EpsTerms eps_terms(float dx, float dy, float dz, float cii, float crr, float q) {
    const float crq = crr * q;
    const float bc = fmaf(2.0f, cii, crr) * crq;
    const float us = dx + dy + dz;
    return {__fmul_rn(__fmul_rn(bc, dx), dx), __fmul_rn(__fmul_rn(bc, dy), dy), __fmul_rn(__fmul_rn(bc, dz), dz),
            __fmul_rn(cii, cii), __fmaf_rn(__fmul_rn(crq, us), us, __fmul_rn(3.0f, cii))};
}

// Stores the epsilon-pass result of bead g from its scaled sums
// (x, y, z: row sums of squares; w: sum of all entries).
__device__ __forceinline__ void eps_store(const KParams &P, const DevBuffers &B, int g, bool active, float4 acc,
                                          const TeaConst &K) {
    const float c2 = K.c075a * K.c075a;
    if (!active) acc = make_float4(0.f, 0.f, 0.f, 0.f);
    B.tea_ci[g] = make_float4(acc.x * c2, acc.y * c2, acc.z * c2, 0.f);
    B.tea_eps[g] = acc.w * K.c075a;
}


// updateTea's reduction (src/bdhitea.cu:75-116), in FP64 on the device: one
// CTA per trajectory sums the bead epsilons and counts the non-extra beads N',
// eps = sum / (3N'(3N'-3)), clamped to 1; a = (3N'-1) eps^2 - (3N'-2) eps;
// beta = (1 - sqrt(1 - a)) / a, or 0.5 when |a| < 1e-7.  The reference's
// exits become the kErrTeaEps bit.
__global__ void __launch_bounds__(256) k_tea_beta(KParams P, DevBuffers B, int capricious, float epsmax,
                                                  const int *gate, int run_if) {
    chain_wait();
    if (gate && *gate != run_if) return;
    const int t = blockIdx.x;
    const int base = B.off[t], end = B.off[t + 1];
    double s = 0.0;
    int cnt = 0;
    for (int g = base + threadIdx.x; g < end; g += blockDim.x) {
        s += (double)B.tea_eps[g];
        cnt += (B.flags[g] & kFlagExtra) ? 0 : 1;
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    }
    __shared__ double ss[8];
    __shared__ int sc[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        ss[wid] = s;
        sc[wid] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double e = 0.0;
        int n = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
            e += ss[k];
            n += sc[k];
        }
        e /= 3.0 * n * (3.0 * n - 3.0);
        int bad = 0;
        if (e > 1.0) {
            if (capricious) bad = 1;
            e = 1.0;
        }
        if (e > (double)epsmax) bad = 1;
        const double a = (3.0 * n - 1.0) * e * e - (3.0 * n - 2.0) * e;
        float beta;
        if (fabs(a) < 1e-7) {
            beta = 0.5f;
            if (capricious && P.tea_a > 0.0f) bad = 1;
        } else {
            beta = (float)((1.0 - sqrt(1.0 - a)) / a);
        }
        B.tea_beta[t] = beta;
        B.tea_eps_t[t] = e;
        if (bad) atomicOr(B.err, kErrTeaEps);
    }
}

// Scaled far-field term of one pair in scalar arithmetic, the operations of
// one lane of the packed loop in the same order.
__device__ __forceinline__ float3 tea_far1(const TeaConst &K, float dx, float dy, float dz, float gx, float gy,
                                           float gz) {
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float rinv = rsqrt_hw(fmaxf(r2, K.four_a2)), q = rinv * rinv, tq = q * rinv;
    const float cii = fmaf(K.kap, tq, rinv);
    const float cr = tq * fmaf(-K.two_a2, q, 1.0f);
    const float s = cr * fmaf(dx, gx, fmaf(dy, gy, dz * gz));
    return make_float3(fmaf(cii, gx, s * dx), fmaf(cii, gy, s * dy), fmaf(cii, gz, s * dz));
}
// Scaled term of one pair with both branches (r2 > 0).
__device__ __forceinline__ float3 tea_pair1(const TeaConst &K, float dx, float dy, float dz, float gx, float gy,
                                            float gz) {
    const float r2 = fmaxf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), 1e-6f);
    const float rinv = rsqrt_hw(r2), q = rinv * rinv, tq = q * rinv;
    float cii = fmaf(K.kap, tq, rinv);
    float cr = tq * fmaf(-K.two_a2, q, 1.0f);
    if (r2 <= K.four_a2) {
        float crr;
        rpy_near(K, r2, rinv, cii, crr);
        cr = crr * q;
    }
    const float s = cr * fmaf(dx, gx, fmaf(dy, gy, dz * gz));
    return make_float3(fmaf(cii, gx, s * dx), fmaf(cii, gy, s * dy), fmaf(cii, gz, s * dz));
}

// a / sqrt(1 + beta^2 C): C_i (a = 1) and beta C_i
__device__ __forceinline__ float tea_norm(float a, float b2, float c) { return a / sqrtf(__fmaf_rn(b2, c, 1.0f)); }

// What the update of bead g starts from; with FEFF its effective force only.
template <bool FEFF>
struct TeaBead {
    float4 ci, F, R, fa;   // fa: ffi, ftheta, fpsi
    Frame Fr;
    uint4 s2;
    int flags;
    __device__ __forceinline__ void load(const KParams &P, const DevBuffers &B, int g) {
        const int nb = P.nb;
        ci = B.tea_ci[g];
        F = B.force[g];
        R = B.tea_r[g];
        if (FEFF) return;
        fa = B.force[nb + g];
        flags = B.flags[g];
        Fr.p0 = B.frame_in[g];
        Fr.p1 = B.frame_in[nb + g];
        Fr.p2 = B.frame_in[2 * nb + g];
        Fr.p3 = B.frame_in[3 * nb + g];
        s2 = B.seeds[nb + g];
    }
};
// The update of bead g from its scaled mobility sums (sx, sy, sz): back to
// units of D_ii, plus the bead's own term F_i + C_i o R_i; FEFF stores f_i.
template <bool FEFF>
__device__ __forceinline__ void tea_bead_update(const KParams &P, const DevBuffers &B, int g, TeaBead<FEFF> &b, float sx,
                                                float sy, float sz, float b2, const TeaConst &K, float4 *feff) {
    const int nb = P.nb;
    sx = __fmaf_rn(K.c075a, sx, __fmaf_rn(b.R.x, tea_norm(1.0f, b2, b.ci.x), b.F.x));
    sy = __fmaf_rn(K.c075a, sy, __fmaf_rn(b.R.y, tea_norm(1.0f, b2, b.ci.y), b.F.y));
    sz = __fmaf_rn(K.c075a, sz, __fmaf_rn(b.R.z, tea_norm(1.0f, b2, b.ci.z), b.F.z));
    if (FEFF) {
        feff[g] = make_float4(sx, sy, sz, 0.f);
        return;
    }
    const float4 ga = gauss4(b.s2), fa = b.fa;
    B.seeds[nb + g] = b.s2;
    Frame Fr = b.Fr;
    if (!(b.flags & (kFlagExtra | kFlagFixed))) {
        const float x = __fmaf_rn(P.kr, sx, Fr.p0.x), y = __fmaf_rn(P.kr, sy, Fr.p0.y), z = __fmaf_rn(P.kr, sz, Fr.p0.z);
        const float fi = __fadd_rn(Fr.p0.w, __fmaf_rn(P.kfi, fa.x, __fmul_rn(P.nfi, ga.x)));
        const float psi = __fadd_rn(Fr.p1.w, __fmaf_rn(P.kfi, fa.z, __fmul_rn(P.nfi, ga.y)));
        const float th = __fadd_rn(Fr.p2.w, __fmaf_rn(P.kth, fa.y, __fmul_rn(P.varTheta, ga.z)));
        Fr = make_frame(P, x, y, z, fi, th, psi);
    }
    store_frame(B.frame_out, nb, g, Fr);
}
template <bool FEFF>
__device__ __forceinline__ void tea_bead_update(const KParams &P, const DevBuffers &B, int g, float sx, float sy,
                                                float sz, float b2, const TeaConst &K, float4 *feff) {
    TeaBead<FEFF> b;
    b.load(P, B, g);
    tea_bead_update<FEFF>(P, B, g, b, sx, sy, sz, b2, K, feff);
}

// ------------------------------------------------------- the all-pairs pass
// One block of beads j for the epsilon pass (integrateTea_epsilon_unlisted,
// src/bdhitea_kernel.cu:84-101): per bead i, sums over non-extra j != i of the
// row sums of squared entries and of all nine entries.  With T = cii I + crr u u^T
// the row sums of squares are cii^2 + (2 cii + crr) crr u_c^2 and the sum of
// all entries is 3 cii + crr (u_x + u_y + u_z)^2.
struct EpsOp {
    static constexpr int kWords = 2 * kTeaPairSlots;   // float4 of a block that it reads: positions
    float2 nx, ny, nz;
    float2 sx, sy, sz, sa, sw;
    __device__ __forceinline__ void start(const KParams &, const DevBuffers &, int, float4 p, int, bool) {
        nx = f2(-p.x);
        ny = f2(-p.y);
        nz = f2(-p.z);
        clear();
    }
    __device__ __forceinline__ void clear() { sx = sy = sz = sa = sw = f2(0.f); }
    template <bool SELF>
    __device__ __forceinline__ void pair(const TeaConst &K, const float4 *blk, int t, int sp, int se,
                                         float &rm) {
        const float2 vkap = f2(K.kap), vn2a2 = f2(-K.two_a2), two = f2(2.0f), three = f2(3.0f);
        const float4 a = blk[t], b = blk[kTeaPairSlots + t];
        const float2 dx = __fadd2_rn(lo2(a), nx), dy = __fadd2_rn(hi2(a), ny), dz = __fadd2_rn(lo2(b), nz);
        const float2 x2 = __fmul2_rn(dx, dx), y2 = __fmul2_rn(dy, dy), z2 = __fmul2_rn(dz, dz);
        float2 r2 = __fadd2_rn(x2, __fadd2_rn(y2, z2));
        if (SELF && t == sp) {
            if (se)
                r2.y = 1e30f;
            else
                r2.x = 1e30f;
        }
        rm = fmin3(rm, r2.x, r2.y);
        const float2 rinv = make_float2(rsqrt_hw(fmaxf(r2.x, K.four_a2)), rsqrt_hw(fmaxf(r2.y, K.four_a2)));
        const float2 q = __fmul2_rn(rinv, rinv);
        const float2 tq = __fmul2_rn(q, rinv);
        const float2 cii = __ffma2_rn(vkap, tq, rinv);
        const float2 crr = __ffma2_rn(vn2a2, tq, rinv);
        const float2 crq = __fmul2_rn(crr, q);
        const float2 bc = __fmul2_rn(__ffma2_rn(two, cii, crr), crq);
        sa = __ffma2_rn(cii, cii, sa);
        sx = __ffma2_rn(bc, x2, sx);
        sy = __ffma2_rn(bc, y2, sy);
        sz = __ffma2_rn(bc, z2, sz);
        const float2 us = __fadd2_rn(__fadd2_rn(dx, dy), dz);
        sw = __ffma2_rn(__fmul2_rn(crq, us), us, __ffma2_rn(three, cii, sw));
    }
    __device__ __forceinline__ float2 dist2(const float4 *blk, int t) const {
        const float4 a = blk[t], b = blk[kTeaPairSlots + t];
        const float2 dx = __fadd2_rn(lo2(a), nx), dy = __fadd2_rn(hi2(a), ny), dz = __fadd2_rn(lo2(b), nz);
        return __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    }
    // one overlapping pair: the far-field terms are replaced by the near ones
    __device__ __forceinline__ void near(const TeaConst &K, const float4 *blk, int t, int e) {
        const float4 a = blk[t], b = blk[kTeaPairSlots + t];
        const float dx = (e ? a.y : a.x) + nx.x, dy = (e ? a.w : a.z) + ny.x, dz = (e ? b.y : b.x) + nz.x;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float rc = rsqrt_hw(fmaxf(r2, K.four_a2)), qc = rc * rc, tq = qc * rc;
        const EpsTerms f = eps_terms(dx, dy, dz, fmaf(K.kap, tq, rc), fmaf(-K.two_a2, tq, rc), qc);
        const float rinv = rsqrt_hw(r2);
        float cn, rn;
        rpy_near(K, r2, rinv, cn, rn);
        const EpsTerms n = eps_terms(dx, dy, dz, cn, rn, rinv * rinv);
        sx.x += __fsub_rn(n.bx, f.bx);
        sy.x += __fsub_rn(n.by, f.by);
        sz.x += __fsub_rn(n.bz, f.bz);
        sa.x += __fsub_rn(n.a2, f.a2);
        sw.x += __fsub_rn(n.w, f.w);
    }
    __device__ __forceinline__ float4 sum() const {
        const float A = sa.x + sa.y;
        return make_float4(sx.x + sx.y + A, sy.x + sy.y + A, sz.x + sz.y + A, sw.x + sw.y);
    }
    struct Bead {
        int flags;
        __device__ __forceinline__ void load(const KParams &, const DevBuffers &B, int g) { flags = B.flags[g]; }
    };
    __device__ __forceinline__ void finish(const KParams &P, const DevBuffers &B, int g, Bead &b, int, float4 acc,
                                           const TeaConst &K, float4 *) const {
        eps_store(P, B, g, (b.flags & kFlagExtra) == 0, acc, K);
    }
};

// The mobility product (integrateTea_kernel_unlisted + integrateTea_force,
// src/bdhitea_kernel.cu:104-213): f_i = F_i + C_i o R_i + sum_{j != i, non-extra}
// T_ij (F_j + beta C_i o R_j), x_i += dt/gammaR f_i; angles by
// Euler-Maruyama from stream i + nb, which is drawn for every bead.  Reads the
// current frame, writes the next one.  With FEFF it stores f_i instead and moves nothing.
template <bool FEFF>
struct StepOp {
    static constexpr int kWords = kTeaBlockF4;
    float2 nx, ny, nz, cbx, cby, cbz;
    float2 ax, ay, az;
    __device__ __forceinline__ void start(const KParams &P, const DevBuffers &B, int traj, float4 p, int g,
                                          bool valid) {
        nx = f2(-p.x);
        ny = f2(-p.y);
        nz = f2(-p.z);
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) {
            const float beta = B.tea_beta[traj], b2 = beta * beta;
            const float4 ci = B.tea_ci[g];
            c = make_float4(tea_norm(beta, b2, ci.x), tea_norm(beta, b2, ci.y), tea_norm(beta, b2, ci.z), 0.f);
        }
        cbx = f2(c.x);
        cby = f2(c.y);
        cbz = f2(c.z);
        clear();
    }
    __device__ __forceinline__ void clear() { ax = ay = az = f2(0.f); }
    template <bool SELF>
    __device__ __forceinline__ void pair(const TeaConst &K, const float4 *blk, int t, int sp, int se,
                                         float &rm) {
        const float2 vkap = f2(K.kap), vn2a2 = f2(-K.two_a2), one = f2(1.0f);
        const float4 a = blk[t], b = blk[kTeaPairSlots + t], c = blk[2 * kTeaPairSlots + t], d = blk[3 * kTeaPairSlots + t];
        const float2 rz = reinterpret_cast<const float2 *>(blk + 4 * kTeaPairSlots)[t];
        const float2 dx = __fadd2_rn(lo2(a), nx), dy = __fadd2_rn(hi2(a), ny), dz = __fadd2_rn(lo2(b), nz);
        const float2 gx = __ffma2_rn(lo2(d), cbx, hi2(b)), gy = __ffma2_rn(hi2(d), cby, lo2(c)),
                     gz = __ffma2_rn(rz, cbz, hi2(c));
        float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        if (SELF && t == sp) {
            if (se)
                r2.y = 1e30f;
            else
                r2.x = 1e30f;
        }
        rm = fmin3(rm, r2.x, r2.y);
        const float2 rinv = make_float2(rsqrt_hw(fmaxf(r2.x, K.four_a2)), rsqrt_hw(fmaxf(r2.y, K.four_a2)));
        const float2 q = __fmul2_rn(rinv, rinv);
        const float2 tq = __fmul2_rn(q, rinv);
        const float2 cii = __ffma2_rn(vkap, tq, rinv);
        const float2 cr = __fmul2_rn(tq, __ffma2_rn(vn2a2, q, one));
        const float2 s = __fmul2_rn(cr, __ffma2_rn(dx, gx, __ffma2_rn(dy, gy, __fmul2_rn(dz, gz))));
        ax = __ffma2_rn(cii, gx, __ffma2_rn(s, dx, ax));
        ay = __ffma2_rn(cii, gy, __ffma2_rn(s, dy, ay));
        az = __ffma2_rn(cii, gz, __ffma2_rn(s, dz, az));
    }
    __device__ __forceinline__ float2 dist2(const float4 *blk, int t) const {
        const float4 a = blk[t], b = blk[kTeaPairSlots + t];
        const float2 dx = __fadd2_rn(lo2(a), nx), dy = __fadd2_rn(hi2(a), ny), dz = __fadd2_rn(lo2(b), nz);
        return __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    }
    __device__ __forceinline__ void near(const TeaConst &K, const float4 *blk, int t, int e) {
        const float4 a = blk[t], b = blk[kTeaPairSlots + t], c = blk[2 * kTeaPairSlots + t], d = blk[3 * kTeaPairSlots + t];
        const float2 rz = reinterpret_cast<const float2 *>(blk + 4 * kTeaPairSlots)[t];
        const float dx = (e ? a.y : a.x) + nx.x, dy = (e ? a.w : a.z) + ny.x, dz = (e ? b.y : b.x) + nz.x;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float gx = fmaf(e ? d.y : d.x, cbx.x, e ? b.w : b.z), gy = fmaf(e ? d.w : d.z, cby.x, e ? c.y : c.x),
                    gz = fmaf(e ? rz.y : rz.x, cbz.x, e ? c.w : c.z);
        const float3 fa = tea_far1(K, dx, dy, dz, gx, gy, gz);
        const float3 nr = tea_pair1(K, dx, dy, dz, gx, gy, gz);
        ax.x += nr.x - fa.x;
        ay.x += nr.y - fa.y;
        az.x += nr.z - fa.z;
    }
    __device__ __forceinline__ float4 sum() const {
        return make_float4(ax.x + ax.y, ay.x + ay.y, az.x + az.y, 0.f);
    }
    using Bead = TeaBead<FEFF>;
    __device__ __forceinline__ void finish(const KParams &P, const DevBuffers &B, int g, Bead &b, int traj, float4 acc,
                                           const TeaConst &K, float4 *feff) const {
        const float beta = B.tea_beta[traj];
        tea_bead_update<FEFF>(P, B, g, b, acc.x, acc.y, acc.z, beta * beta, K, feff);
    }
};

// The overlapping beads of a block (own: the slot of the bead itself, or -1): which they
// are, then their terms.
template <class Op>
__device__ __forceinline__ void tea_near_block(Op &X, const TeaConst &K, const float4 *blk, int own) {
    unsigned near = 0;
#pragma unroll 4
    for (int t = 0; t < kTeaPairSlots; t++) {
        const float2 r2 = X.dist2(blk, t);
        near |= (r2.x <= K.four_a2 ? 1u : 0u) << (2 * t) | (r2.y <= K.four_a2 ? 2u : 0u) << (2 * t);
    }
    if (own >= 0) near &= ~(1u << own);
    for (; near; near &= near - 1) {
        const int j = __ffs((int)near) - 1;
        X.near(K, blk, j >> 1, j & 1);
    }
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}

// Adds node v of an item's tree of sums (level lvl, first fine segment lo), of which the segments
// [s0, s1) of n are in hand: kTeaHold while its right sibling is to come (v is kept in node[lvl]),
// kTeaCut when its parent is not in hand (v is the sum of the largest node that is, from segment lo),
// kTeaGroup when v is that of a whole top node.
enum { kTeaHold, kTeaCut, kTeaGroup };
__device__ __forceinline__ int tea_carry(float4 &v, int &lo, int lvl, int s0, int s1, int n, float4 *node, int stride) {
#pragma unroll 1
    for (; lvl < kTeaLevels; lvl++) {
        const int plo = lo & ~((2 << lvl) - 1), pend = min(plo + (2 << lvl), n);
        if (plo < s0 || pend > s1) return kTeaCut;
        if (lo != plo) {
            v = add4(node[lvl * stride], v);
        } else if (lo + (1 << lvl) < n) {
            node[lvl * stride] = v;
            return kTeaHold;
        }   // else there is no right sibling
        lo = plo;
    }
    return kTeaGroup;
}

// The sum of a bead from the slots of its item's grains.  A call, once for an item, so that the
// pair loop keeps its registers.
static __device__ __noinline__ float4 tea_collect(const float4 *part, int ng, int level) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const int group = level < kTeaLevels ? (1 << kTeaLevels) >> level : 1;   // slots of a top node
    for (int j = 0; j < ng; j += 8) {   // eight requested at once
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (j + k < ng) v[k] = __ldcg(&part[(j + k) * kTeaI]);
#pragma unroll
        for (int h = 1; h < 8; h *= 2)
#pragma unroll
            for (int k = 0; k < 8; k += 2 * h)
                if (h < group && j + k + h < ng) v[k] = add4(v[k], v[k + h]);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k % group == 0 && j + k < ng) acc = add4(acc, v[k]);
    }
    return acc;
}

// One CTA for each grain of the work: 128 beads i and the blocks j of 2^tea_level fine segments
// (a fixed grid walks over them where a launch mostly finds its gate closed).  Runs
// while gate is null or *gate == run_if.
template <class Op>
__global__ void __launch_bounds__(kTeaThreads, kTeaOcc) k_tea_pass(KParams P, DevBuffers B, const int2 *work,
                                                                   int nwork, float4 *feff, const int *gate, int run_if) {
    constexpr int kW = Op::kWords;
    __shared__ float4 s_tile[kTeaStages][kTeaTileBlocks * kW];
    __shared__ float4 s_node[kTeaLevels + 1][kTeaThreads];   // each thread's own: nodes that wait, the sum
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int2 grain = work[blockIdx.x];   // chunk, first fine segment
    TeaItem w = B.tea_item[grain.x];
    chain_wait();   // no kernel writes the grains
    if (gate && *gate != run_if) return;
    const TeaConst K = tea_const(P.tea_a);
    for (int at = blockIdx.x;;) {
        const int nblk = (w.end - w.base + kTeaBlock - 1) / kTeaBlock, fine = tea_fine(nblk);
        const int nfine = (nblk + fine - 1) / fine, s0 = grain.y, s1 = min(nfine, s0 + (1 << P.tea_level));
        const int b0 = s0 * fine, b1 = min(nblk, s1 * fine);
        const int g = w.first + tid;
        const float4 *pack = B.tea_pack + (size_t)w.block * kTeaBlockF4;
        auto issue = [&](int tile) {
            const int q0 = b0 + tile * kTeaTileBlocks, nq = min(kTeaTileBlocks, b1 - q0);
            float4 *dst = s_tile[tile % kTeaStages];
            for (int c = tid; c < nq * kW; c += kTeaThreads)
                cp_async16(dst + c, pack + (size_t)(q0 + c / kW) * kTeaBlockF4 + c % kW);
        };
        const int ntiles = (b1 - b0 + kTeaTileBlocks - 1) / kTeaTileBlocks;
#pragma unroll
        for (int k = 0; k < kTeaStages - 1; k++) {
            if (k < ntiles) issue(k);
            cp_async_commit();
        }
        const bool valid = g < w.end;
        const float4 p = valid ? B.frame_in[g] : make_float4(0.f, 0.f, 0.f, 0.f);
        const bool act = __any_sync(0xffffffffu, valid && !(B.flags[g] & kFlagExtra));
        const bool split = s1 - s0 < nfine;
        float4 *node = &s_node[0][tid];
        node[kTeaLevels * kTeaThreads] = make_float4(0.f, 0.f, 0.f, 0.f);
        Op X;
        X.start(P, B, w.traj, p, g, valid);
        const int self = (w.first - w.base) / kTeaBlock + warp;   // the block that holds this warp's beads
        int left = fine, seg = s0;   // blocks of the fine segment still to come, its index
        for (int tile = 0; tile < ntiles; tile++) {
            cp_async_wait<kTeaStages - 2>();
            __syncthreads();
            if (tile + kTeaStages - 1 < ntiles) issue(tile + kTeaStages - 1);
            cp_async_commit();
            if (!act) continue;
            const int q0 = b0 + tile * kTeaTileBlocks, nq = min(kTeaTileBlocks, b1 - q0);
            for (int q = 0; q < nq; q++) {
                const float4 *blk = s_tile[tile % kTeaStages] + q * kW;
                const bool own = q0 + q == self;
                float rm = 3.4e38f;
                if (own) {
#pragma unroll 1
                    for (int t = 0; t < kTeaPairSlots; t++) X.template pair<true>(K, blk, t, lane >> 1, lane & 1, rm);
                } else {
#pragma unroll 8
                    for (int t = 0; t < kTeaPairSlots; t++) X.template pair<false>(K, blk, t, 0, 0, rm);
                }
                if (rm <= K.four_a2) tea_near_block(X, K, blk, own ? lane : -1);
                if (--left > 0 && q0 + q + 1 < nblk) continue;
                left = fine;
                float4 v = X.sum();
                X.clear();
                int lo = seg++;
                if (tea_carry(v, lo, 0, s0, s1, nfine, node, kTeaThreads) != kTeaHold)   // the grain, or a group of the item
                    node[kTeaLevels * kTeaThreads] = split ? v : add4(node[kTeaLevels * kTeaThreads], v);
            }
        }
        float4 acc = node[kTeaLevels * kTeaThreads];
        bool done = true;
        __syncthreads();   // the tiles are free again (and s_last)
        if (split) {
            float4 *part = B.tea_part + (size_t)w.slot * kTeaI + tid;   // of the item's grains
            const int ng = (nfine + (1 << P.tea_level) - 1) >> P.tea_level;
            part[(s0 >> P.tea_level) * kTeaI] = acc;
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(&B.tea_cnt[grain.x], 1) == ng - 1;
            __syncthreads();
            done = s_last;
            if (done) {
                __threadfence();
                acc = tea_collect(part, ng, P.tea_level);
                if (tid == 0) B.tea_cnt[grain.x] = 0;
            }
        }
        if (done && valid) {
            typename Op::Bead bead;
            bead.load(P, B, g);
            X.finish(P, B, g, bead, w.traj, acc, K, feff);
        }
        at += gridDim.x;
        if (at >= nwork) break;
        grain = work[at];
        w = B.tea_item[grain.x];
    }
}

// Positions of every bead into the pack (the force kernel of a TEA step does
// it with F and R; this one serves epsilon passes outside a step).
__global__ void k_tea_pack(KParams P, DevBuffers B) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const bool extra = (B.flags[g] & kFlagExtra) != 0;
    const float4 p = B.frame_in[g];
    tea_pack_position(B, g, extra ? make_float3(kTeaFarAway, kTeaFarAway, kTeaFarAway) : make_float3(p.x, p.y, p.z));
}
// An empty pack: every slot far away with zero F and R.
__global__ void k_tea_pack_clear(float4 *pack, int nblocks) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nblocks * kTeaBlockF4) return;
    const int w = k % kTeaBlockF4;
    const float a = w < 2 * kTeaPairSlots ? kTeaFarAway : 0.f, b = w < kTeaPairSlots ? kTeaFarAway : 0.f;
    pack[k] = make_float4(a, a, b, b);
}

// The same sums for systems too small to fill the GPU, where a pass lasts as long as its
// chain of waits: a CTA of eight warps serves eight beads, a thread one bead and one fine segment
// (eight lanes read the same words), the segments meet in shared memory, so
// no partial sum goes through global memory and no CTA waits for another's.
// The CTA copies its whole trajectory first, one word further for
// every block, so that the segments of a warp are in different banks.
constexpr int kSmallBeads = 8, kSmallThreads = 256, kSmallStride = kTeaBlockF4 + 1;
template <class Op>
__global__ void __launch_bounds__(kSmallThreads, 2) k_tea_small(KParams P, DevBuffers B, float4 *feff, const int *gate,
                                                                int run_if) {
    __shared__ float4 s_part[kTeaMaxFine][kSmallBeads];
    extern __shared__ float4 s_pack[];
    const int l = threadIdx.x % kSmallBeads;
    const int2 w = B.tea_small[blockIdx.x];   // trajectory, first bead
    const int traj = w.x, base = B.off[traj], end = B.off[traj + 1], n = end - base, g = w.y + l;
    const bool valid = g < end;
    const int gc = valid ? g : end - 1, slot0 = B.tea_slot[base];
    chain_wait();   // no kernel writes what was read so far
    if (gate && *gate != run_if) return;
    const int nblk = (n + kTeaBlock - 1) / kTeaBlock, fine = tea_fine(nblk), nfine = (nblk + fine - 1) / fine;
    const float4 *pack = B.tea_pack + (size_t)(slot0 / kTeaBlock) * kTeaBlockF4;
    for (int q = threadIdx.x / 32; q < nblk; q += kSmallThreads / 32)
        for (int c = threadIdx.x % 32; c < Op::kWords; c += 32) cp_async16(s_pack + q * kSmallStride + c, pack + q * kTeaBlockF4 + c);
    cp_async_commit();
    const float4 p = B.frame_in[gc];
    const TeaConst K = tea_const(P.tea_a);
    Op X;
    X.start(P, B, traj, p, gc, valid);
    const int self = (gc - base) / kTeaBlock, in = (gc - base) % kTeaBlock;
    typename Op::Bead bead;
    if (threadIdx.x < kSmallBeads) bead.load(P, B, gc);   // of the threads that finish the beads
    cp_async_wait<0>();
    __syncthreads();
    for (int f = threadIdx.x / kSmallBeads; f < nfine; f += kSmallThreads / kSmallBeads) {
        X.clear();
        const int last = min(nblk, (f + 1) * fine);
        for (int q = f * fine; q < last; q++) {
            const float4 *blk = s_pack + q * kSmallStride;
            const bool own = q == self;
            const int sp = own ? in >> 1 : -1;
            float rm = 3.4e38f;
#pragma unroll
            for (int t = 0; t < kTeaPairSlots; t++) X.template pair<true>(K, blk, t, sp, in & 1, rm);
            if (rm <= K.four_a2) tea_near_block(X, K, blk, own ? in : -1);
        }
        s_part[f][l] = X.sum();
    }
    __syncthreads();
    // the first warp adds them, a lane a bead and a group of the tree
    if (threadIdx.x >= 32) return;
    static_assert(kTeaLevels == 3 && kSmallBeads == 8, "four groups of eight a warp");
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 acc = zero;
    for (int f0 = 0; f0 < nfine; f0 += 32) {
        const int f = f0 + threadIdx.x / kSmallBeads * 8, m = nfine - f;
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = k < m ? s_part[f + k][l] : zero;
#pragma unroll
        for (int h = 1; h < 8; h *= 2)
#pragma unroll
            for (int k = 0; k < 8; k += 2 * h)
                if (k + h < m) v[k] = add4(v[k], v[k + h]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 t = make_float4(__shfl_sync(0xffffffffu, v[0].x, l + 8 * k), __shfl_sync(0xffffffffu, v[0].y, l + 8 * k),
                                         __shfl_sync(0xffffffffu, v[0].z, l + 8 * k), __shfl_sync(0xffffffffu, v[0].w, l + 8 * k));
            if (f0 + 8 * k < nfine) acc = add4(acc, t);
        }
    }
    if (threadIdx.x < kSmallBeads && valid) X.finish(P, B, g, bead, traj, acc, K, feff);
}
// Up to these CTAs for every SM and blocks of a trajectory the small form is used.  Steps with it and
// with k_tea_pass: 299 beads 9.4 and 13.5 us, 1520 beads 15.4 and 19.6, 2800 beads (350 CTAs) 28.6 and
// 29.1, 2 x 1520 beads (380) 22.2 and 23.5; but 3300 beads (104 blocks) 37.6 and 30.5, 4 x 1520 beads
// (760) 30.2 and 27.5, 20 x 299 beads (760) 20.0 and 18.3.
constexpr int kTeaSmallCtas = 3, kTeaSmallBlocks = 96;
int tea_small_prepare() {   // the limit of the largest trajectory: engines share the kernels
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int bytes = kTeaSmallBlocks * kSmallStride * (int)sizeof(float4);
    return cudaFuncSetAttribute(k_tea_small<EpsOp>, attr, bytes) == cudaSuccess &&
                   cudaFuncSetAttribute(k_tea_small<StepOp<false>>, attr, bytes) == cudaSuccess &&
                   cudaFuncSetAttribute(k_tea_small<StepOp<true>>, attr, bytes) == cudaSuccess
               ? 0
               : -1;
}
int tea_small_beads() { return kSmallBeads; }
// rare: a launch that mostly finds its gate closed, which should be short then.
template <class Op>
static void tea_launch(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, float4 *feff, const int *gate,
                       int run_if, cudaStream_t s) {
    if (P.tea_nsmall <= kTeaSmallCtas * (P.tea_wave / kTeaOcc) && P.tea_max_blocks <= kTeaSmallBlocks) {
        launch_chained(P, k_tea_small<Op>, P.tea_nsmall, kSmallThreads, sizeof(float4) * kSmallStride * P.tea_max_blocks,
                       s, P, B, feff, gate, run_if);
        return;
    }
    const bool rare = gate && run_if == 1;
    launch_chained(P, k_tea_pass<Op>, rare ? std::min(nwork, P.tea_wave) : nwork, kTeaThreads, 0, s, P, B, work, nwork, feff,
                   gate, run_if);
}
// The grain of a batch: of fine segments, pairs of them, and so on up to whole items the one with the
// least work a CTA slot plus a quarter of a grain at the end (a CTA alone on an SM is about four times as
// fast as one of nine), half a block a grain for its start and its partial sums.
int tea_grain_level(long long units, const long long *ngrains, const int *blocks, int wave) {
    int best = 0;
    double least = 1e300;
    for (int k = 0; k <= kTeaWhole; k++) {
        const double t = ((double)units + 0.5 * ngrains[k]) / wave + 0.25 * (blocks[k] + 0.5);
        if (t < least) {
            least = t;
            best = k;
        }
    }
    return best;
}
void launch_tea_pack(const KParams &P, const DevBuffers &B, cudaStream_t s) {
    k_tea_pack<<<(P.nb + 127) / 128, 128, 0, s>>>(P, B);
}
void launch_tea_pack_clear(float4 *pack, int nblocks, cudaStream_t s) {
    k_tea_pack_clear<<<(int)(((size_t)nblocks * kTeaBlockF4 + 255) / 256), 256, 0, s>>>(pack, nblocks);
}
void launch_tea_eps_gated(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, const int *gate,
                          int run_if, cudaStream_t s) {
    tea_launch<EpsOp>(P, B, work, nwork, nullptr, gate, run_if, s);
}
void launch_tea_eps(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, cudaStream_t s) {
    launch_tea_eps_gated(P, B, work, nwork, nullptr, 0, s);
}
void launch_tea_beta_gated(const KParams &P, const DevBuffers &B, int capricious, float epsmax, const int *gate,
                           int run_if, cudaStream_t s) {
    launch_chained(P, k_tea_beta, P.nt, 256, 0, s, P, B, capricious, epsmax, gate, run_if);
}
void launch_tea_beta(const KParams &P, const DevBuffers &B, int capricious, float epsmax, cudaStream_t s) {
    launch_tea_beta_gated(P, B, capricious, epsmax, nullptr, 0, s);
}
void launch_tea_step(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, cudaStream_t s) {
    tea_launch<StepOp<false>>(P, B, work, nwork, nullptr, nullptr, 0, s);
}
void launch_tea_step_gated(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, const int *gate,
                           cudaStream_t s) {
    tea_launch<StepOp<false>>(P, B, work, nwork, nullptr, gate, 1, s);
}
void launch_tea_feff(const KParams &P, const DevBuffers &B, const int2 *work, int nwork, float4 *feff,
                     const int *gate, cudaStream_t s) {
    tea_launch<StepOp<true>>(P, B, work, nwork, feff, gate, 0, s);
}

// ---------------------------------------------- far field of learned TEA
// The learned mode's approximation of sum_j T_ij (F_j + beta C_i o R_j) on a
// k-d tree per trajectory (tea_ff.cu): pairs of beads in near leaves are
// summed exactly (the packed pair loop of the all-pairs pass), and every far node J acts on a target node N through proxies: J's
// sources are spread onto the 8 points of a Chebyshev grid in its bounding box
// (P2M, trilinear Lagrange weights at nodes +-h/sqrt(2)), the RPY far field
// of those 8 charges is evaluated at the 8 grid points of N (M2L), brought
// down to the leaves under N (L2L) and interpolated to their beads (L2P).
// Because C_i weights R_j per component and per target, the proxies carry F
// and R separately and the targets receive A = T Q_F and B_k = T e_k Q_R,k
// (k = x, y, z); a bead adds A + sum_k beta C_ik B_k.

// Trilinear Lagrange weights of the 8 proxies (bit 0: x, bit 1: y, bit 2: z;
// a clear bit is the node at -h/sqrt(2), a set bit the one at +h/sqrt(2)) at
// position x of a box (c, h); the fast division's 2-ulp error is far below
// the interpolation's own.
__device__ __forceinline__ void ff_weights(float3 x, float4 c, float4 h, float w[8]) {
    const float tx = __fdividef(x.x - c.x, h.x * kFFNode), ty = __fdividef(x.y - c.y, h.y * kFFNode),
                tz = __fdividef(x.z - c.z, h.z * kFFNode);
    const float lx[2] = {0.5f * (1.0f - tx), 0.5f * (1.0f + tx)};
    const float ly[2] = {0.5f * (1.0f - ty), 0.5f * (1.0f + ty)};
    const float lz[2] = {0.5f * (1.0f - tz), 0.5f * (1.0f + tz)};
#pragma unroll
    for (int m = 0; m < 8; m++) w[m] = lx[m & 1] * ly[(m >> 1) & 1] * lz[(m >> 2) & 1];
}
__device__ __forceinline__ float3 ff_proxy(float4 c, float4 h, int m) {
    return make_float3(c.x + ((m & 1) ? kFFNode : -kFFNode) * h.x, c.y + ((m & 2) ? kFFNode : -kFFNode) * h.y,
                       c.z + ((m & 4) ? kFFNode : -kFFNode) * h.z);
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over the 32 lanes of a warp of 32 values per lane, scattered: lane l
// ends with the sum of value l (recursive halving: at offset o a lane keeps
// the half of its values selected by bit o of its index and receives its
// partner's partial sums of that half; 31 shuffles instead of 160).
__device__ __forceinline__ float warp_reduce_scatter32(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, n = 32; o > 0; o >>= 1, n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (i >= n / 2) break;
            const float send = up ? v[i] : v[i + n / 2];
            const float keep = up ? v[i + n / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

constexpr int kP2MWarps = 4;   // warps of a P2M block, one node each

// Writes the 48 charge sums of a warp (acc[6m + v], summed per lane) as the
// node's proxy charges: (QF.xyz, QR.x) at float4 16N + m, (QR.y, QR.z) at
// 16N + 8 + m.
__device__ __forceinline__ void ff_store_charges(const FFBuffers &F, int N, float (&acc)[48]) {
    const int lane = threadIdx.x & 31;
    float lo[32], hi[32];
#pragma unroll
    for (int i = 0; i < 32; i++) lo[i] = acc[i];
#pragma unroll
    for (int i = 0; i < 16; i++) hi[i] = acc[32 + i];
#pragma unroll
    for (int i = 16; i < 32; i++) hi[i] = 0.f;
    const float s_lo = warp_reduce_scatter32(lo);   // value lane
    const float s_hi = warp_reduce_scatter32(hi);   // value 32 + lane (lanes < 16)
    float *q = reinterpret_cast<float *>(F.q);
    auto put = [&](int idx, float val) {
        const int m = idx / 6, c = idx % 6;
        q[(size_t)4 * (16 * N + (c < 4 ? m : 8 + m)) + (c < 4 ? c : c - 4)] = val;
    };
    put(lane, s_lo);
    if (lane < 16) put(32 + lane, s_hi);
}

// Writes lane k's bead (or an empty slot: far away, zero F and R) into leaf
// N's pack: lanes 2p and 2p + 1 swap their values and write bead pair p as
// whole 16-byte words (the even lane the position words, the odd lane the
// force and random-force words, the even lane Rz with its neighbour pair's).
// Called by all 32 lanes of the warp.
__device__ __forceinline__ void ff_pack_warp(const FFBuffers &F, int N, float3 x, float4 Fv, float4 R) {
    const int lane = threadIdx.x & 31, p = lane >> 1;
    const bool odd = lane & 1;
    const float v[9] = {x.x, x.y, x.z, Fv.x, Fv.y, Fv.z, R.x, R.y, R.z};
    float o[9];
#pragma unroll
    for (int i = 0; i < 9; i++) o[i] = __shfl_xor_sync(0xffffffffu, v[i], 1);
    // (a, b) = (even lane's bead, odd lane's bead)
    float a[9], b[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        a[i] = odd ? o[i] : v[i];
        b[i] = odd ? v[i] : o[i];
    }
    float4 *pk = F.pack + (size_t)N * kFFPackF4;
    if (!odd) {
        pk[p] = make_float4(a[0], b[0], a[1], b[1]);                      // xa xb ya yb
        pk[kFFPairSlots + p] = make_float4(a[2], b[2], a[3], b[3]);       // za zb Fxa Fxb
    } else {
        pk[2 * kFFPairSlots + p] = make_float4(a[4], b[4], a[5], b[5]);   // Fya Fyb Fza Fzb
        pk[3 * kFFPairSlots + p] = make_float4(a[6], b[6], a[7], b[7]);   // Rxa Rxb Rya Ryb
    }
    // Rz of pairs p (lanes 4w, 4w+1) and p + 1 (lanes 4w+2, 4w+3) in one word
    const float rz2a = __shfl_down_sync(0xffffffffu, a[8], 2), rz2b = __shfl_down_sync(0xffffffffu, b[8], 2);
    if ((lane & 3) == 0) pk[4 * kFFPairSlots + (p >> 1)] = make_float4(a[8], b[8], rz2a, rz2b);
}

// P2M of the leaves, one warp per leaf (lane k: bead k): the bounding box,
// the proxy charges Q_m = sum_j w_m(x_j) (F_j, R_j), and the leaf's beads in
// the step kernel's tile layout (leaf nleaf: the padding leaf's pack).
__global__ void __launch_bounds__(32 * kP2MWarps) k_ff_p2m(KParams P, DevBuffers B, FFBuffers F, const int *gate) {
    chain_wait();
    if (gate && *gate != 0) return;
    const int N = blockIdx.x * kP2MWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (N > F.nleaf) return;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float3 away = make_float3(kFarAway, kFarAway, kFarAway);
    if (N == F.nleaf) {
        ff_pack_warp(F, N, away, zero, zero);
        return;
    }
    const int b0 = F.leaf_start[N], n = F.leaf_start[N + 1] - b0;
    float3 x = make_float3(0.f, 0.f, 0.f);
    float4 Fv = zero, R = zero;
    if (lane < n) {
        const int g = F.leaf_bead[b0 + lane];
        x = f3(B.frame_in[g]);
        Fv = B.force[g];
        R = B.tea_r[g];
    }
    const float3 lo = make_float3(warp_min(lane < n ? x.x : 3.4e38f), warp_min(lane < n ? x.y : 3.4e38f),
                                  warp_min(lane < n ? x.z : 3.4e38f));
    const float3 hi = make_float3(warp_max(lane < n ? x.x : -3.4e38f), warp_max(lane < n ? x.y : -3.4e38f),
                                  warp_max(lane < n ? x.z : -3.4e38f));
    const float4 c = make_float4(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z), 0.f);
    const float4 h = make_float4(fmaxf(0.5f * (hi.x - lo.x), 1e-3f), fmaxf(0.5f * (hi.y - lo.y), 1e-3f),
                                 fmaxf(0.5f * (hi.z - lo.z), 1e-3f), 0.f);
    ff_pack_warp(F, N, lane < n ? x : away, Fv, R);
    float w[8];
    ff_weights(x, c, h, w);
    const float val[6] = {Fv.x, Fv.y, Fv.z, R.x, R.y, R.z};
    float acc[48];
#pragma unroll
    for (int m = 0; m < 8; m++)
#pragma unroll
        for (int v = 0; v < 6; v++) acc[6 * m + v] = lane < n ? w[m] * val[v] : 0.f;
    ff_store_charges(F, N, acc);
    if (lane == 0) {
        F.box[2 * N] = c;
        F.box[2 * N + 1] = h;
    }
}

// P2M of the inner nodes, one warp per node, from the node's leaves: the
// bounding box is the union of theirs, and since trilinear interpolation on
// a leaf's proxies reproduces every trilinear function, the node's weights
// at the leaf proxies carry the leaf charges over exactly:
// Q^N_m = sum_leaves sum_k w^N_m(y_k) Q^leaf_k.
__global__ void __launch_bounds__(32 * kP2MWarps) k_ff_p2m_inner(KParams P, FFBuffers F, const int *gate) {
    if (gate && *gate != 0) return;
    const int k = blockIdx.x * kP2MWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= F.ninner) return;
    const int N = F.inner[k];
    const int l0 = F.node_leaves[2 * N], l1 = F.node_leaves[2 * N + 1];
    float3 lo = make_float3(3.4e38f, 3.4e38f, 3.4e38f), hi = make_float3(-3.4e38f, -3.4e38f, -3.4e38f);
    for (int l = l0 + lane; l < l1; l += 32) {
        const float4 c = F.box[2 * l], h = F.box[2 * l + 1];
        lo = make_float3(fminf(lo.x, c.x - h.x), fminf(lo.y, c.y - h.y), fminf(lo.z, c.z - h.z));
        hi = make_float3(fmaxf(hi.x, c.x + h.x), fmaxf(hi.y, c.y + h.y), fmaxf(hi.z, c.z + h.z));
    }
    lo = make_float3(warp_min(lo.x), warp_min(lo.y), warp_min(lo.z));
    hi = make_float3(warp_max(hi.x), warp_max(hi.y), warp_max(hi.z));
    const float4 c = make_float4(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z), 0.f);
    const float4 h = make_float4(fmaxf(0.5f * (hi.x - lo.x), 1e-3f), fmaxf(0.5f * (hi.y - lo.y), 1e-3f),
                                 fmaxf(0.5f * (hi.z - lo.z), 1e-3f), 0.f);
    float acc[48];
#pragma unroll
    for (int i = 0; i < 48; i++) acc[i] = 0.f;
    // lane t takes proxy t % 8 of every fourth leaf
    for (int e = l0 * 8 + lane; e < l1 * 8; e += 32) {
        const int l = e >> 3, m = e & 7;
        const float3 y = ff_proxy(F.box[2 * l], F.box[2 * l + 1], m);
        const float4 qa = F.q[16 * l + m], qb = F.q[16 * l + 8 + m];
        const float val[6] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y};
        float w[8];
        ff_weights(y, c, h, w);
#pragma unroll
        for (int mm = 0; mm < 8; mm++)
#pragma unroll
            for (int v = 0; v < 6; v++) acc[6 * mm + v] = fmaf(w[mm], val[v], acc[6 * mm + v]);
    }
    ff_store_charges(F, N, acc);
    if (lane == 0) {
        F.box[2 * N] = c;
        F.box[2 * N + 1] = h;
    }
}

// M2L: 4 x kM2LSlices lanes per target node; lane t serves the target
// proxies t % 4 and t % 4 + 4 (the same x and y, opposite z) as one packed
// pair over every kM2LSlices-th far node, and the slices meet by shuffles in
// a fixed order.
constexpr int kM2LWarps = 4;
// 8 slices (a warp per target); 4 and 2 (two and four targets per warp)
// measured the same and slower
constexpr int kM2LSlices = 8, kM2LLanes = 4 * kM2LSlices;
__global__ void __launch_bounds__(32 * kM2LWarps) k_ff_m2l(KParams P, FFBuffers F, const int *gate) {
    if (gate && *gate != 0) return;
    const int lane = threadIdx.x & 31;
    const int wk = (blockIdx.x * kM2LWarps + (threadIdx.x >> 5)) * (32 / kM2LLanes) + lane / kM2LLanes;
    const bool active = wk < F.ntgt;
    const int L = active ? F.tgt[wk] : 0, t = lane % kM2LLanes, np = t & 3, sl = t >> 2;
    const TeaConst K = tea_const(P.tea_a);
    const float4 cL = F.box[2 * L], hL = F.box[2 * L + 1];
    const float3 x0 = ff_proxy(cL, hL, np), x1 = ff_proxy(cL, hL, np + 4);
    const float2 nxx = f2(-x0.x), nxy = f2(-x0.y), nxz = make_float2(-x0.z, -x1.z);
    const float2 vkap = f2(K.kap), vn2a2 = f2(-K.two_a2), one = f2(1.0f);
    float2 acc[12];
#pragma unroll
    for (int c = 0; c < 12; c++) acc[c] = f2(0.f);
    for (int k = F.far_start[L] + sl; active && k < F.far_start[L + 1]; k += kM2LSlices) {
        const int J = F.far[k];
        const float4 cJ = F.box[2 * J], hJ = F.box[2 * J + 1];
#pragma unroll
        for (int m = 0; m < 8; m++) {
            const float3 y = ff_proxy(cJ, hJ, m);
            const float2 dx = __fadd2_rn(f2(y.x), nxx), dy = __fadd2_rn(f2(y.y), nxy), dz = __fadd2_rn(f2(y.z), nxz);
            const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            const float2 rinv = make_float2(rsqrt_hw(r2.x), rsqrt_hw(r2.y));
            const float2 q2 = __fmul2_rn(rinv, rinv), tq = __fmul2_rn(q2, rinv);
            const float2 cii = __ffma2_rn(vkap, tq, rinv);
            const float2 cr = __fmul2_rn(tq, __ffma2_rn(vn2a2, q2, one));
            const float4 qa = F.q[16 * J + m], qb = F.q[16 * J + 8 + m];
            const float2 qfx = f2(qa.x), qfy = f2(qa.y), qfz = f2(qa.z);
            const float2 sF = __fmul2_rn(cr, __ffma2_rn(dx, qfx, __ffma2_rn(dy, qfy, __fmul2_rn(dz, qfz))));
            acc[0] = __ffma2_rn(cii, qfx, __ffma2_rn(sF, dx, acc[0]));
            acc[1] = __ffma2_rn(cii, qfy, __ffma2_rn(sF, dy, acc[1]));
            acc[2] = __ffma2_rn(cii, qfz, __ffma2_rn(sF, dz, acc[2]));
            const float2 rx = f2(qa.w), ry = f2(qb.x), rz = f2(qb.y);
            const float2 s0 = __fmul2_rn(__fmul2_rn(cr, dx), rx), s1 = __fmul2_rn(__fmul2_rn(cr, dy), ry),
                         s2 = __fmul2_rn(__fmul2_rn(cr, dz), rz);
            acc[3] = __ffma2_rn(cii, rx, __ffma2_rn(s0, dx, acc[3]));
            acc[4] = __ffma2_rn(s0, dy, acc[4]);
            acc[5] = __ffma2_rn(s0, dz, acc[5]);
            acc[6] = __ffma2_rn(s1, dx, acc[6]);
            acc[7] = __ffma2_rn(cii, ry, __ffma2_rn(s1, dy, acc[7]));
            acc[8] = __ffma2_rn(s1, dz, acc[8]);
            acc[9] = __ffma2_rn(s2, dx, acc[9]);
            acc[10] = __ffma2_rn(s2, dy, acc[10]);
            acc[11] = __ffma2_rn(cii, rz, __ffma2_rn(s2, dz, acc[11]));
        }
    }
#pragma unroll
    for (int o = 4; o < kM2LLanes; o <<= 1)
#pragma unroll
        for (int c = 0; c < 12; c++) {
            acc[c].x += __shfl_xor_sync(0xffffffffu, acc[c].x, o);
            acc[c].y += __shfl_xor_sync(0xffffffffu, acc[c].y, o);
        }
    if (active && sl == 0) {
        float *phi = reinterpret_cast<float *>(F.phi) + (size_t)96 * L;
#pragma unroll
        for (int c = 0; c < 12; c++) {
            phi[12 * np + c] = acc[c].x;
            phi[12 * (np + 4) + c] = acc[c].y;
        }
    }
}

// Near pairs.  The near lists of all leaves, one after another, are cut into
// runs of about equal length, one warp each, twice as many as the GPU holds at once; a warp goes through the
// leaves its run touches, a bead a lane, with the near leaves' beads copied one
// leaf at a time, two ahead, into its own ring in shared memory: no barrier, no
// partly filled wave, and equal work for all four schedulers of an SM.  The pair loop
// is that of the all-pairs pass (StepOp), and like it the kernel is bound by the FP32 pipe.
// A leaf's list is summed in segments of kFFSeg entries, added in order, and runs begin at the
// heads of segments, so a bead's sum depends on its leaf alone, not on where the runs of
// its batch are cut.  A leaf that one run holds goes to FFBuffers::nearsum; of a leaf that several
// share each segment's sum goes to its slot and k_ff_far adds them.
// 64 x 5600 beads, 225 M pairs: 256 us with four warps a leaf on 128-bead tiles (2100 of
// 3950 instructions a warp were not pair arithmetic), 268 us with a whole leaf
// a warp (a third of the time was the last wave), 242 us so (238 with runs cut at any entry).
// Overlapping pairs (r <= 2a): with LISTCORR the far-field term of the pair loop is
// replaced while walking the bead's LJ list once, which holds every pair
// that close (checked by the launcher), by the run that begins the leaf;
// otherwise they are looked for in the leaves whose smallest r^2 shows one, as
// the all-pairs pass does.
constexpr int kFFStages = 3;
static_assert(kFFLeaf == kTeaBlock && kFFPackF4 == kTeaBlockF4, "leaves are blocks of the pair loop");
template <bool LISTCORR>
__global__ void __launch_bounds__(32 * kFFWarps, kFFCtas) k_ff_near(KParams P, DevBuffers B, FFBuffers F, const int *gate) {
    chain_wait();
    if (gate && *gate != 0) return;
    __shared__ float4 s_leaf[kFFWarps][kFFStages][kFFPackF4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, run = blockIdx.x * kFFWarps + warp;
    if (run >= F.near_runs) return;
    const int u0 = F.near_run[run], u1 = F.near_run[run + 1];   // entries
    int L = F.run_leaf[run];
    auto issue = [&](int u) {
        if (u < u1) {
            const float4 *src = F.pack + (size_t)F.near[u] * kFFPackF4;
            float4 *dst = s_leaf[warp][(u - u0) % kFFStages];
#pragma unroll
            for (int c = 0; c < kFFPackF4; c += 32)
                if (c + lane < kFFPackF4) cp_async16(dst + c + lane, src + c + lane);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int k = 0; k < kFFStages - 1; k++) issue(u0 + k);
    const TeaConst K = tea_const(P.tea_a);
    for (int u = u0; u < u1; L++) {
        const int e0 = F.near_start[L], e1 = F.near_start[L + 1], stop = min(u1, e1);
        const int s0 = F.leaf_start[L], n = F.leaf_start[L + 1] - s0, traj = F.leaf_traj[L];
        const bool valid = lane < n;
        const int g = valid ? F.leaf_bead[s0 + lane] : 0;
        const float4 x = valid ? B.frame_in[g] : make_float4(0.f, 0.f, 0.f, 0.f);
        StepOp<false> X;
        X.start(P, B, traj, x, g, valid);
        float3 corr = make_float3(0.f, 0.f, 0.f);
        if (LISTCORR && valid && u == e0) {
            const int base = B.off[traj], nb = P.nb;
            const int cnt = B.ljc[g];
            for (int q0 = 0; q0 < cnt; q0 += 4) {   // four entries in flight
                float4 xj[4];
                int pj[4];
#pragma unroll
                for (int v = 0; v < 4; v++) pj[v] = q0 + v < cnt ? base + B.lj[(q0 + v) * nb + g] : -1;
#pragma unroll
                for (int v = 0; v < 4; v++)
                    xj[v] = pj[v] >= 0 ? B.frame_in[pj[v]] : make_float4(kFarAway, 0.f, 0.f, 0.f);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const float dx = xj[v].x - x.x, dy = xj[v].y - x.y, dz = xj[v].z - x.z;
                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    if (!(r2 <= K.four_a2) || (B.flags[pj[v]] & kFlagExtra)) continue;
                    const float4 Fj = B.force[pj[v]], Rj = B.tea_r[pj[v]];
                    const float gx = fmaf(Rj.x, X.cbx.x, Fj.x), gy = fmaf(Rj.y, X.cby.x, Fj.y),
                                gz = fmaf(Rj.z, X.cbz.x, Fj.z);
                    const float3 fa = tea_far1(K, dx, dy, dz, gx, gy, gz);
                    const float3 nr = tea_pair1(K, dx, dy, dz, gx, gy, gz);
                    corr.x += nr.x - fa.x;
                    corr.y += nr.y - fa.y;
                    corr.z += nr.z - fa.z;
                }
            }
        }
        const int slot = F.near_slot[L];   // of the leaf's first segment, or -1
        float4 sum = make_float4(corr.x, corr.y, corr.z, 0.f), total = make_float4(0.f, 0.f, 0.f, 0.f);
        for (; u < stop; u++) {
            cp_async_wait<kFFStages - 2>();
            __syncwarp();
            const float4 *blk = s_leaf[warp][(u - u0) % kFFStages];
            const bool own = F.near[u] == L;
            issue(u + kFFStages - 1);
            float rm = 3.4e38f;
            if (own) {
#pragma unroll 1
                for (int t = 0; t < kTeaPairSlots; t++) X.template pair<true>(K, blk, t, lane >> 1, lane & 1, rm);
            } else {
#pragma unroll 8
                for (int t = 0; t < kTeaPairSlots; t++) X.template pair<false>(K, blk, t, 0, 0, rm);
            }
            if (!LISTCORR && rm <= K.four_a2) tea_near_block(X, K, blk, own ? lane : -1);
            if ((u - e0) % kFFSeg < kFFSeg - 1 && u + 1 < e1) continue;
            sum = add4(X.sum(), sum);   // with the overlapping pairs in the first segment's
            X.clear();
            if (slot < 0)
                total = add4(total, sum);
            else
                F.nearpart[(size_t)(slot + (u - e0) / kFFSeg) * kFFLeaf + lane] = sum;
            sum = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (slot < 0 && valid) F.nearsum[s0 + lane] = total;
    }
}
// The near sum of bead `lane` of leaf L (leaf bead s0 + lane) from its segments.
__device__ __forceinline__ float4 ff_near_sum(const FFBuffers &F, int L, int s0, int lane) {
    const int slot = F.near_slot[L];
    if (slot < 0) return F.nearsum[s0 + lane];
    const int n = (F.near_start[L + 1] - F.near_start[L] + kFFSeg - 1) / kFFSeg;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < n; k += 4) {   // four requested at once
        float4 q[4];
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (k + h < n) q[h] = F.nearpart[(size_t)(slot + k + h) * kFFLeaf + lane];
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (k + h < n) v = add4(v, q[h]);
    }
    return v;
}

// Far field and update: one warp per leaf.  The far fields of the leaf and
// of each ancestor with a far list are brought to the leaf's 8 proxies (L2L:
// one (ancestor, proxy) per lane, exact because interpolating on the leaf
// reproduces any trilinear field), summed in ancestor order, interpolated to
// each bead (L2P), added to its near sum, and the bead moves (FEFF: its
// effective force goes to feff instead).
template <bool FEFF>
__global__ void __launch_bounds__(32) k_ff_far(KParams P, DevBuffers B, FFBuffers F, float4 *feff, const int *gate) {
    if (gate && *gate != 0) return;
    const int L = blockIdx.x, lane = threadIdx.x;
    const int s0 = F.leaf_start[L], n = F.leaf_start[L + 1] - s0;
    // per ancestor: box (2) and potentials (24); sized for the tree's longest
    // ancestor list (max_anc)
    extern __shared__ float4 s_far[];
    __shared__ float4 s_pl[8 * 3];             // the far field at the leaf's proxies
    __shared__ float4 s_lbox[2];
    const int a0 = F.anc_start[L], na = min(F.anc_start[L + 1] - a0, F.max_anc);
    for (int k = lane; k < 26 * na; k += 32) {
        const int N = F.anc[a0 + k / 26], w = k % 26;
        s_far[k] = w < 2 ? F.box[2 * N + w] : F.phi[24 * N + w - 2];
    }
    if (lane < 2) s_lbox[lane] = F.box[2 * L + lane];
    __syncwarp();
    {   // lane (A, pn): ancestors A, A + 4, ... at the leaf's proxy pn, the four
        // groups of ancestors summed by shuffles
        const int pn = lane & 7;
        const float3 y = ff_proxy(s_lbox[0], s_lbox[1], pn);
        float4 v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int A = lane >> 3; A < na; A += 4) {
            const float4 *fr = s_far + 26 * A;
            float w[8];
            ff_weights(y, fr[0], fr[1], w);
#pragma unroll
            for (int m = 0; m < 8; m++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float4 q = fr[2 + 3 * m + c];
                    v[c] = make_float4(fmaf(w[m], q.x, v[c].x), fmaf(w[m], q.y, v[c].y), fmaf(w[m], q.z, v[c].z),
                                       fmaf(w[m], q.w, v[c].w));
                }
        }
#pragma unroll
        for (int o = 8; o < 32; o <<= 1)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                v[c].x += __shfl_xor_sync(0xffffffffu, v[c].x, o);
                v[c].y += __shfl_xor_sync(0xffffffffu, v[c].y, o);
                v[c].z += __shfl_xor_sync(0xffffffffu, v[c].z, o);
                v[c].w += __shfl_xor_sync(0xffffffffu, v[c].w, o);
            }
        if (lane < 8)
#pragma unroll
            for (int c = 0; c < 3; c++) s_pl[3 * lane + c] = v[c];
    }
    __syncwarp();
    if (lane >= n) return;
    const int g = F.leaf_bead[s0 + lane];
    const int traj = F.leaf_traj[L];
    const float beta = B.tea_beta[traj], b2 = beta * beta;
    const float3 xi = f3(B.frame_in[g]);
    const float4 ci = B.tea_ci[g];
    const float3 cbi = make_float3(beta / sqrtf(1.0f + b2 * ci.x), beta / sqrtf(1.0f + b2 * ci.y),
                                   beta / sqrtf(1.0f + b2 * ci.z));
    const float4 ns = ff_near_sum(F, L, s0, lane);
    float sx = ns.x, sy = ns.y, sz = ns.z;
    if (na > 0) {   // L2P from the leaf's proxies
        float w[8];
        ff_weights(xi, s_lbox[0], s_lbox[1], w);
#pragma unroll
        for (int m = 0; m < 8; m++) {
            // A.xyz, B_x.xyz, B_y.xyz, B_z.xyz
            const float4 p = s_pl[3 * m], q = s_pl[3 * m + 1], r = s_pl[3 * m + 2];
            // A + beta C_x B_x + beta C_y B_y + beta C_z B_z
            const float ux = p.x + cbi.x * p.w + cbi.y * q.z + cbi.z * r.y;
            const float uy = p.y + cbi.x * q.x + cbi.y * q.w + cbi.z * r.z;
            const float uz = p.z + cbi.x * q.y + cbi.y * r.x + cbi.z * r.w;
            sx = fmaf(w[m], ux, sx);
            sy = fmaf(w[m], uy, sy);
            sz = fmaf(w[m], uz, sz);
        }
    }
    tea_bead_update<FEFF>(P, B, g, sx, sy, sz, b2, tea_const(P.tea_a), feff);
}

// Beads in no leaf (extra beads): the update draws their angular noise and
// keeps their frame, as the all-pairs update does.
template <bool FEFF>
__global__ void k_ff_rest(KParams P, DevBuffers B, FFBuffers F, float4 *feff, const int *gate) {
    if (gate && *gate != 0) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= F.nrest) return;
    const int g = F.rest[k];
    const float beta = B.tea_beta[B.traj[g]];
    tea_bead_update<FEFF>(P, B, g, 0.f, 0.f, 0.f, beta * beta, tea_const(P.tea_a), feff);
}

void launch_ff_p2m_leaves(const KParams &P, const DevBuffers &B, const FFBuffers &F, const int *gate,
                          cudaStream_t s) {
    if (F.nleaf == 0) return;
    launch_chained(P, k_ff_p2m, (F.nleaf + kP2MWarps) / kP2MWarps, 32 * kP2MWarps, 0, s, P, B, F, gate);
}
void launch_ff_m2l(const KParams &P, const FFBuffers &F, const int *gate, cudaStream_t s) {
    if (F.nleaf == 0) return;
    if (F.ninner > 0)
        k_ff_p2m_inner<<<(F.ninner + kP2MWarps - 1) / kP2MWarps, 32 * kP2MWarps, 0, s>>>(P, F, gate);
    constexpr int per_block = kM2LWarps * (32 / kM2LLanes);
    if (F.ntgt > 0) k_ff_m2l<<<(F.ntgt + per_block - 1) / per_block, 32 * kM2LWarps, 0, s>>>(P, F, gate);
}
void launch_ff_proxies(const KParams &P, const DevBuffers &B, const FFBuffers &F, const int *gate, cudaStream_t s) {
    launch_ff_p2m_leaves(P, B, F, gate, s);
    launch_ff_m2l(P, F, gate, s);
}

// Overlapping pairs can be taken from the LJ list when it holds every pair
// within 2a (plus 2 nm for the motion since its rebuild).
static bool ff_list_corr(const KParams &P) { return P.lj_on && P.ljcut >= 2.0f * P.tea_a + 2.0f; }

void launch_ff_near(const KParams &P, const DevBuffers &B, const FFBuffers &F, const int *gate, cudaStream_t s) {
    if (F.nleaf == 0) return;
    const int ctas = (F.near_runs + kFFWarps - 1) / kFFWarps;
    if (ff_list_corr(P))
        launch_chained(P, k_ff_near<true>, ctas, 32 * kFFWarps, 0, s, P, B, F, gate);
    else
        launch_chained(P, k_ff_near<false>, ctas, 32 * kFFWarps, 0, s, P, B, F, gate);
}
void launch_ff_far(const KParams &P, const DevBuffers &B, const FFBuffers &F, bool feff_only, float4 *feff,
                   const int *gate, cudaStream_t s) {
    if (F.nleaf > 0) {
        const size_t smem = (size_t)F.max_anc * 26 * sizeof(float4);
        if (feff_only)
            k_ff_far<true><<<F.nleaf, 32, smem, s>>>(P, B, F, feff, gate);
        else
            k_ff_far<false><<<F.nleaf, 32, smem, s>>>(P, B, F, feff, gate);
    }
    if (F.nrest > 0) {
        if (feff_only)
            k_ff_rest<true><<<(F.nrest + 127) / 128, 128, 0, s>>>(P, B, F, feff, gate);
        else
            k_ff_rest<false><<<(F.nrest + 127) / 128, 128, 0, s>>>(P, B, F, feff, gate);
    }
}
void launch_ff_step(const KParams &P, const DevBuffers &B, const FFBuffers &F, bool feff_only, float4 *feff,
                    const int *gate, cudaStream_t s) {
    launch_ff_near(P, B, F, gate, s);
    launch_ff_far(P, B, F, feff_only, feff, gate, s);
}

}  // namespace mtg
