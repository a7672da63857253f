// kernels_cells.cu - neighbour-list rebuild through a per-trajectory spatial
// hash (cell list), producing the same lists as the brute-force kernel.
// k_cell_lists_smem, further down, does it in one launch where the trajectories fit in
// shared memory; what follows here is the general path.
//
// Cells are cubes of edge `reach` (the largest list cutoff, or the 6.6 nm
// prefilter of the assembly lists), so every partner lies in the 27 cells
// around a bead.  Each trajectory owns a hash table of next_pow2(max(32, N))
// buckets; colliding cells share a bucket and only add candidates.
//   1. k_cell_count : bucket of every bead, bucket populations
//   2. k_cell_scan  : one CTA per trajectory, exclusive scan of its table
//   3. k_cell_fill  : beads scattered into bucket order
//   4. k_cell_lists : per bead, candidates from the 27 cells' buckets (each
//      bucket visited once) read from a bucket-ordered copy of the
//      positions, the reference's list tests, then an insertion sort so each
//      list is in ascending j (orientation 0 before 1 for the lateral list),
//      exactly the order of the reference's j loops
//      (src/compute_cuda.cu:564-661, :927-936).
#include <cmath>

#include "mtg_internal.cuh"

namespace mtg {

namespace {

constexpr float kPairReach = 6.6f;  // see kPairPrefilter

__global__ void k_cell_count(KParams P, const float4 *pos, const int *traj, const int *tbase, const int *tmask,
                             float inv_cell, int *key, int *cnt) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const float4 p = pos[g];
    const int t = traj[g];
    const uint32_t h = cell_hash(cell_coord(p.x, inv_cell), cell_coord(p.y, inv_cell), cell_coord(p.z, inv_cell));
    const int k = tbase[t] + (int)(h & (uint32_t)tmask[t]);
    key[g] = k;
    atomicAdd(&cnt[k], 1);
}

// Exclusive scan of each trajectory's table; start and cursor get the result.
__global__ void __launch_bounds__(1024) k_cell_scan(const int *tbase, const int *cnt, int *start, int *cursor) {
    const int t = blockIdx.x;
    const int b0 = tbase[t], n = tbase[t + 1] - tbase[t];
    __shared__ int s_warp[32];
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
    int local = 0;
    for (int i = lo; i < hi; i++) local += cnt[b0 + i];
    // block exclusive scan of `local`
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int v = local;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) s_warp[wid] = v;
    __syncthreads();
    if (wid == 0) {
        int w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    int run = (v - local) + (wid > 0 ? s_warp[wid - 1] : 0);
    for (int i = lo; i < hi; i++) {
        start[b0 + i] = run;
        cursor[b0 + i] = run;
        run += cnt[b0 + i];
    }
}

// Bucket-ordered bead lists; positions are relative to the trajectory's
// first bead, so slots of trajectory t start at off[t].
__global__ void k_cell_fill(int nb, const int *traj, const int *off, const int *key, const int *flags, int *cursor,
                            int *cell_bead, const float4 *pos, float4 *cell_pos) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nb) return;
    const int slot = off[traj[g]] + atomicAdd(&cursor[key[g]], 1);
    cell_bead[slot] = g;
    float4 p = pos[g];
    // bucket-ordered copy of the positions, bead index (and the extra flag) in w
    p.w = __int_as_float(g | ((flags[g] & kFlagExtra) ? kCellExtraBit : 0));
    cell_pos[slot] = p;
}

// Ascending bead index within every bucket (the atomic fill leaves them in
// arrival order), so that sums over a bucket are reproducible.  Grid
// (trajectory, bucket chunk), one thread per bucket; buckets hold a few beads.
__global__ void k_cell_sort(const int *off, const int *tbase, const int *tmask, const int *start, const int *cnt,
                            int *cell_bead, float4 *cell_pos) {
    const int t = blockIdx.x, base = off[t], tb = tbase[t], nbk = tmask[t] + 1;
    const int b = blockIdx.y * blockDim.x + threadIdx.x;
    if (b >= nbk) return;
    const int n = cnt[tb + b];
    if (n < 2) return;
    int *cb = cell_bead + base + start[tb + b];
    float4 *cp = cell_pos + base + start[tb + b];
    for (int i = 1; i < n; i++) {
        const int v = cb[i];
        const float4 pv = cp[i];
        int j = i - 1;
        while (j >= 0 && cb[j] > v) {
            cb[j + 1] = cb[j];
            cp[j + 1] = cp[j];
            j--;
        }
        cb[j + 1] = v;
        cp[j + 1] = pv;
    }
}

__device__ __forceinline__ void isort(int *a, int n) {
    for (int i = 1; i < n; i++) {
        const int v = a[i];
        int j = i - 1;
        while (j >= 0 && a[j] > v) {
            a[j + 1] = a[j];
            j--;
        }
        a[j + 1] = v;
    }
}

// In-place insertion sort of a k-major list (rare path: > kLocalLJ entries).
__device__ void isort_strided(int *a, int n, int stride) {
    for (int i = 1; i < n; i++) {
        const int v = a[(size_t)i * stride];
        int j = i - 1;
        while (j >= 0 && a[(size_t)j * stride] > v) {
            a[(size_t)(j + 1) * stride] = a[(size_t)j * stride];
            j--;
        }
        a[(size_t)(j + 1) * stride] = v;
    }
}

constexpr int kLocalLJ = 16;   // LJ hits sorted in shared memory; more are sorted in place

// Insertion sort of one thread's column of a [rows][kTile] shared array.
__device__ __forceinline__ void isort_col(int (*a)[kTile], int n, int t) {
    for (int i = 1; i < n; i++) {
        const int v = a[i][t];
        int j = i - 1;
        while (j >= 0 && a[j][t] > v) {
            a[j + 1][t] = a[j][t];
            j--;
        }
        a[j + 1][t] = v;
    }
}

// Thread per bead: candidates are read from the bucket-ordered position copy
// (one contiguous 16 B load each); the rare assembly candidates (< 6.6 nm)
// also read the neighbour's site planes.
template <bool PAIRS>
__global__ void __launch_bounds__(kTile, 6) k_cell_lists(KParams P, DevBuffers B, const int2 *work, const int *tbase,
                                                         const int *tmask, const int *start, const int *cnt,
                                                         const float4 *cell_pos, float inv_cell) {
    const int2 w = work[blockIdx.x];
    const int traj = w.x, base = B.off[traj], end = B.off[traj + 1];
    const int g = w.y + threadIdx.x;
    if (g >= end) return;
    const int nb = P.nb;
    const float4 *fr = B.frame_in;
    const int flags = B.flags[g];
    const bool extra_i = (flags & kFlagExtra) != 0;
    const bool do_lj = P.lj_on && !extra_i;
    const bool do_pairs = PAIRS && P.is_assembly && !extra_i;
    if (!do_lj && !do_pairs) {
        if (P.lj_on) B.ljc[g] = 0;
        if (PAIRS && P.is_assembly) {
            B.lonc[g] = 0;
            B.latc[g] = 0;
        }
        return;
    }
    const float4 pi = fr[g];
    const int il = g - base;
    const int h0 = B.harm[g * P.maxH];
    const int hpart = h0 < 0 ? -h0 : h0;
    const int cx = cell_coord(pi.x, inv_cell), cy = cell_coord(pi.y, inv_cell), cz = cell_coord(pi.z, inv_cell);
    const int tb = tbase[traj];
    const uint32_t mask = (uint32_t)tmask[traj];

    // this thread's LJ hits: a column of shared memory (its own bank), so the
    // buffer and its sort never leave the SM
    __shared__ int s_lj[kLocalLJ][kTile];
    int lo_buf[kCellMaxLong], la_buf[kCellMaxLat];
    int nlj = 0, nlo = 0, nla = 0;
    bool overflow = false;
    // the ranges of the 27 cells' buckets, all requested at once and kept in
    // shared memory for the rolled cell loop, and a mask of the cells whose
    // bucket an earlier cell already has
    __shared__ int s_st[27][kTile], s_ct[27][kTile];
    uint32_t dup = 0;
    {
        int bk[27];
#pragma unroll
        for (int c = 0; c < 27; c++)
            bk[c] = tb + (int)(cell_hash(cx + c % 3 - 1, cy + (c / 3) % 3 - 1, cz + c / 9 - 1) & mask);
#pragma unroll
        for (int c = 0; c < 27; c++) {
            s_st[c][threadIdx.x] = start[bk[c]];
            s_ct[c][threadIdx.x] = cnt[bk[c]];
        }
#pragma unroll
        for (int c = 1; c < 27; c++) {
            bool seen = false;
#pragma unroll
            for (int v = 0; v < c; v++) seen |= (bk[v] == bk[c]);
            dup |= (seen ? 1u : 0u) << c;
        }
    }
    // drop the buckets an earlier cell already has, then walk the remaining
    // candidates in cell order four at a time across cell boundaries, so a
    // sparse neighbourhood still has four loads in flight
    for (int c = 0; c < 27; c++)
        if ((dup >> c) & 1u) s_ct[c][threadIdx.x] = 0;
    int c = 0, off = 0;
    while (c < 27 && s_ct[c][threadIdx.x] == 0) c++;
    while (c < 27) {
        int sl[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            sl[u] = -1;
            if (c < 27) {
                sl[u] = base + s_st[c][threadIdx.x] + off;
                if (++off == s_ct[c][threadIdx.x]) {
                    off = 0;
                    do {
                        c++;
                    } while (c < 27 && s_ct[c][threadIdx.x] == 0);
                }
            }
        }
        float4 qq[4];   // four candidates in flight
#pragma unroll
        for (int u = 0; u < 4; u++) qq[u] = sl[u] >= 0 ? cell_pos[sl[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (sl[u] < 0) break;
            const float4 q = qq[u];
            const int jg = __float_as_int(q.w) & kCellIndexMask;
            const int jl = jg - base;
            const float cd = centre_dist(pi, q);
            if (do_lj && jl != il && cd < P.ljcut) {
                if (nlj >= P.maxLJ) {
                    overflow = true;
                } else if (nlj < kLocalLJ) {
                    s_lj[nlj][threadIdx.x] = jl;
                } else {
                    if (nlj == kLocalLJ)  // spill the local part first
                        for (int k = 0; k < kLocalLJ; k++) B.lj[k * nb + g] = s_lj[k][threadIdx.x];
                    B.lj[nlj * nb + g] = jl;
                }
                nlj++;
            }
            if (do_pairs && cd < kPairReach && jl != hpart) {
                const float4 pj = fr[jg];   // the exact state (q carries the index in w)
                const float rmon = h0 < 0 ? -2.0f : 2.0f;
                const int fj = B.flags[jg];
                if (((flags ^ fj) & kFlagBeta) != 0) {
                    const float4 ui = fr[nb + g], uj = fr[nb + jg];
                    const float3 wi = make_float3(ui.x * rmon, ui.y * rmon, ui.z * rmon);
                    if (norm3_rn(site_delta(pi, pj, wi, make_float3(-uj.x * rmon, -uj.y * rmon, -uj.z * rmon))) <
                        2.5f) {
                        if (nlo < P.maxLong)
                            lo_buf[nlo] = jl;
                        else
                            overflow = true;
                        nlo++;
                    }
                }
                if (jl != il) {
                    const float4 li1 = fr[2 * nb + g], li2 = fr[3 * nb + g];
                    const float4 l1 = fr[2 * nb + jg], l2 = fr[3 * nb + jg];
                    if (norm3_rn(site_delta(pi, pj, f3(li1), f3(l2))) < 2.5f) {
                        if (nla < P.maxLat)
                            la_buf[nla] = 2 * jl;       // orientation 0 -> -j
                        else
                            overflow = true;
                        nla++;
                    }
                    if (norm3_rn(site_delta(pi, pj, f3(li2), f3(l1))) < 2.5f) {
                        if (nla < P.maxLat)
                            la_buf[nla] = 2 * jl + 1;   // orientation 1 -> +j
                        else
                            overflow = true;
                        nla++;
                    }
                }
            }
        }
    }
    if (P.lj_on) {
        const int n = min(nlj, P.maxLJ);
        if (n <= kLocalLJ) {
            isort_col(s_lj, n, threadIdx.x);
            for (int k = 0; k < n; k++) B.lj[k * nb + g] = s_lj[k][threadIdx.x];
        } else {
            isort_strided(B.lj + g, n, nb);
        }
        B.ljc[g] = n;
    }
    if (PAIRS && P.is_assembly) {
        const int n1 = min(nlo, P.maxLong), n2 = min(nla, P.maxLat);
        isort(lo_buf, n1);
        isort(la_buf, n2);
        for (int k = 0; k < n1; k++) B.lon[k * nb + g] = h0 < 0 ? lo_buf[k] : -lo_buf[k];
        for (int k = 0; k < n2; k++) {
            const int j = la_buf[k] >> 1;
            const int code = j != 0 ? j : kZeroCode;
            B.lat[k * nb + g] = (la_buf[k] & 1) ? code : -code;
        }
        B.lonc[g] = n1;
        B.latc[g] = n2;
    }
    if (overflow) atomicOr(B.err, kErrOverflow);
}

// Longitudinal and lateral lists (pairs_kernel, src/compute_cuda.cu:527-674)
// from the bead's LJ list: every assembly candidate (centre distance below
// kPairReach) is in the LJ list when the LJ cutoff is longer, and the LJ list
// is in ascending j, so the lists come out in the reference's order without a
// sort.  Runs after k_cell_lists<false>.
__global__ void __launch_bounds__(kTile) k_pairs_from_lj(KParams P, DevBuffers B) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P.nb) return;
    const int nb = P.nb;
    const int flags = B.flags[g];
    if (flags & kFlagExtra) {
        B.lonc[g] = 0;
        B.latc[g] = 0;
        return;
    }
    const float4 *fr = B.frame_in;
    const int base = B.off[B.traj[g]], il = g - base;
    const float4 pi = fr[g], ui = fr[nb + g], li1 = fr[2 * nb + g], li2 = fr[3 * nb + g];
    const int h0 = B.harm[g * P.maxH];
    const int hpart = h0 < 0 ? -h0 : h0;
    const float rmon = h0 < 0 ? -2.0f : 2.0f;
    const float3 wi = make_float3(ui.x * rmon, ui.y * rmon, ui.z * rmon);
    const int n = min(B.ljc[g], P.maxLJ);
    int nlo = 0, nla = 0;
    bool overflow = false;
    for (int k0 = 0; k0 < n; k0 += 4) {
        int jj[4];
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) jj[u] = k0 + u < n ? B.lj[(k0 + u) * nb + g] : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) q[u] = jj[u] >= 0 ? fr[base + jj[u]] : pi;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int jl = jj[u];
            if (jl < 0 || jl == hpart || !(centre_dist(pi, q[u]) < kPairReach)) continue;
            const int jg = base + jl;
            const float4 pj = q[u];
            const int fj = B.flags[jg];
            if (((flags ^ fj) & kFlagBeta) != 0) {
                const float4 uj = fr[nb + jg];
                if (norm3_rn(site_delta(pi, pj, wi, make_float3(-uj.x * rmon, -uj.y * rmon, -uj.z * rmon))) < 2.5f) {
                    if (nlo < P.maxLong)
                        B.lon[nlo * nb + g] = h0 < 0 ? jl : -jl;
                    else
                        overflow = true;
                    nlo++;
                }
            }
            if (jl != il) {
                const float4 l1 = fr[2 * nb + jg], l2 = fr[3 * nb + jg];
                const int code = jl != 0 ? jl : kZeroCode;
                if (norm3_rn(site_delta(pi, pj, f3(li1), f3(l2))) < 2.5f) {
                    if (nla < P.maxLat)
                        B.lat[nla * nb + g] = -code;   // orientation 0 -> -j
                    else
                        overflow = true;
                    nla++;
                }
                if (norm3_rn(site_delta(pi, pj, f3(li2), f3(l1))) < 2.5f) {
                    if (nla < P.maxLat)
                        B.lat[nla * nb + g] = code;    // orientation 1 -> +j
                    else
                        overflow = true;
                    nla++;
                }
            }
        }
    }
    B.lonc[g] = min(nlo, P.maxLong);
    B.latc[g] = min(nla, P.maxLat);
    if (overflow) atomicOr(B.err, kErrOverflow);
}

// ---------------------------------------------- the whole rebuild in one CTA
// Trajectories of up to kSmemBeads beads, LJ on and either no assembly lists or
// every assembly candidate inside the LJ cutoff: one launch, one CTA per
// chunk of a trajectory's beads.  Each CTA bins its whole trajectory into
// shared memory, so a candidate costs a shared-memory load instead of a
// dependent L2 one, and the beads of the chunk then walk their cells; of chunks
// smaller than the CTA 2 or 4 threads share a bead's rows and keys, and the first sorts
// and writes (small batches last as long as one bead's chain: 18 -> 11 us for 1520 beads).
//   * The bucket of cell (cx, cy, cz) is (row hash of (cy, cz) + cx) mod M, so
//     the three cells of a row are neighbouring buckets: 9 contiguous ranges a
//     bead instead of 27 buckets, and no search for repeated buckets.  Rows that
//     share buckets only add candidates; a hit counts in the row that is its
//     own, so it counts once.  M >= 2 n keeps such extra candidates few (about one
//     a row).
//   * The bucket table holds 16-bit counts, then starts, then (after the fill)
//     ends.
//   * Distances are compared squared, against the largest square whose root is
//     below the cutoff (sq_below), which is the same decision.
//   * A hit is a 16-bit key: index * 8 + which site tests can succeed (the
//     partner's centre within 4.51 nm of the bead's own site: sites are at most
//     2 nm from a centre and bonds at most 2.5 nm long).  Keys are sorted in
//     registers (Batcher's odd-even merge network, up to 24), so the lists come out in
//     ascending j; only the site planes that a test needs are then gathered.
// Bound by instruction issue and, in the walk, by shared-memory bandwidth.
// 256 x 1520 beads: 203 us for the general path's six launches (the 27-bucket
// walk ran 7600 instructions a warp, half of them on repeated buckets), 61 us here;
// 1024 uneven trajectories of up to 3560 beads 775 -> 275 us, 101 lattices of 780 beads
// 66 -> 21 us, one trajectory of 156 beads 45 (tiles) -> 10 us.
constexpr int kSmemKeys = 32;      // slots for a bead's hits; beads with more than 28 are walked again, below
constexpr int kSmemBeads = 8192;   // 13 bits of a key
constexpr unsigned kNoKey = 0x10000u;

size_t smem_list_bytes(int nmax) {
    return sizeof(float4) * ((size_t)nmax + 3) +
           sizeof(uint16_t) * ((size_t)row_buckets(nmax) + kSmemKeys * kListThreads);
}

// Batcher's odd-even merge sort of N keys in registers, ascending.
template <int N>
__device__ __forceinline__ void sort_network(unsigned (&k)[N]) {
#pragma unroll
    for (int p = 1; p < N; p *= 2)
#pragma unroll
        for (int q = p; q >= 1; q /= 2)
#pragma unroll
            for (int j = q % p; j + q < N; j += 2 * q)
#pragma unroll
                for (int i = 0; i < q; i++)
                    if (i + j + q < N && (i + j) / (2 * p) == (i + j + q) / (2 * p)) {
                        const unsigned a = k[i + j], b = k[i + j + q];
                        k[i + j] = min(a, b);
                        k[i + j + q] = max(a, b);
                    }
}
template <int N>
__device__ __forceinline__ void sort_keys(uint16_t (*s_key)[kListThreads], int n) {
    unsigned k[N];
#pragma unroll
    for (int i = 0; i < N; i++) k[i] = i < n ? s_key[i][threadIdx.x] : 0xffffu;
    sort_network<N>(k);
#pragma unroll
    for (int i = 0; i < N; i++)
        if (i < n) s_key[i][threadIdx.x] = (uint16_t)k[i];
}

// A trajectory's beads in bucket order, in shared memory.
struct SmemCells {
    const float4 *pos;    // w = index in the trajectory
    const uint16_t *end;  // end of each bucket's range (a range starts where the one before ends)
    int n, m;
    float inv;
};
// The slots of the buckets of cells cx - 1 .. cx + 1 of a row: [s, e) and, of a range
// that wraps round the table, [0, e2).
__device__ __forceinline__ void row_range(const SmemCells &C, int cx, int cy, int cz, int &s, int &e, int &e2) {
    const int b0 = (int)((row_hash(cy, cz) + (uint32_t)(cx - 1)) & (uint32_t)(C.m - 1)), b2 = b0 + 2;
    s = b0 > 0 ? C.end[b0 - 1] : 0;
    e = C.end[min(b2, C.m - 1)];
    e2 = b2 >= C.m ? C.end[b2 - C.m] : 0;
}
// Calls hit(position and index) for every bead of the trajectory in the cells around p that
// is closer than the root of t2, in no particular order; once for every row whose
// buckets hold it, so a bead whose own row shares them can come twice.
template <class F>
__device__ __forceinline__ void smem_candidates(const SmemCells &C, float4 p, float t2, F &&hit) {
    const int cx = cell_coord(p.x, C.inv), cy = cell_coord(p.y, C.inv), cz = cell_coord(p.z, C.inv);
#pragma unroll 1
    for (int r = 0; r < 9; r++) {
        int s, e, e2;
        row_range(C, cx, cy + r % 3 - 1, cz + r / 3 - 1, s, e, e2);
#pragma unroll 1
        for (; s < e || e2 > 0; s += 4) {
            if (s >= e) {
                s = 0;
                e = e2;
                e2 = 0;
            }
            float4 q[4];   // four candidates in flight
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = C.pos[min(s + u, e - 1)];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (s + u < e && dist2_rn(p, q[u]) < t2) hit(q[u]);
        }
    }
}
// The same slots, and perhaps a few a rounding further off, written down one key row after
// another; returns their number, or more than kSmemKeys - 4 if that many were met
// (the walk ends there).  The ranges of the 32 beads of a warp differ in length, so the
// loop over candidates runs for the longest (22 iterations of four a warp where a
// bead has 30 candidates) and what an iteration costs is what counts: no branch
// for a hit, the distance contracted, the ends of the next row requested ahead, and
// no shared-memory wavefronts for lanes past their range (half of the time before).
__device__ __forceinline__ int smem_slots(const SmemCells &C, float4 p, float t2, int row, int last, uint16_t *key) {
    const int cx = cell_coord(p.x, C.inv), cy = cell_coord(p.y, C.inv), cz = cell_coord(p.z, C.inv);
    const float loose = t2 * 1.00001f;   // over the difference between the two roundings
    const unsigned k0 = (unsigned)__cvta_generic_to_shared(key), stride = sizeof(uint16_t) * kListThreads;
    const unsigned full = k0 + (kSmemKeys - 4) * stride;
    unsigned to = k0;   // where the next hit goes
    const unsigned pos = (unsigned)__cvta_generic_to_shared(C.pos);
    auto load = [&](int slot, int end) {   // a lane past its range takes no bandwidth
        float4 q;
        asm volatile("{ .reg .pred a;\n\t"
                     "setp.lt.s32 a, %4, %5;\n\t"
                     "@a ld.shared.v4.f32 {%0, %1, %2, %3}, [%6]; }"
                     : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                     : "r"(slot), "r"(end), "r"(pos + 16u * (unsigned)slot)
                     : "memory");
        return q;
    };
    auto test = [&](float4 q, int slot, int end) {
        const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        asm volatile("{ .reg .pred a, b;\n\t"
                     "setp.lt.s32 a, %1, %2;\n\t"
                     "setp.lt.and.f32 b, %3, %4, a;\n\t"
                     "@b st.shared.u16 [%0], %5;\n\t"
                     "@b add.u32 %0, %0, %6; }"
                     : "+r"(to)
                     : "r"(slot), "r"(end), "f"(r2), "f"(loose), "h"((uint16_t)slot), "n"(sizeof(uint16_t) * kListThreads)
                     : "memory");
    };
    int s, e, e2;
    row_range(C, cx, cy + row % 3 - 1, cz + row / 3 - 1, s, e, e2);
#pragma unroll 1
    for (int r = row + 1; r <= last; r++) {
        int k = s, end = e, again = e2;
        if (r < last) row_range(C, cx, cy + r % 3 - 1, cz + r / 3 - 1, s, e, e2);   // the next one's, ahead
        while (true) {
#pragma unroll 1
            for (; k < end && to <= full; k += 4) {
                float4 q[4];
#pragma unroll
                for (int u = 0; u < 4; u++) q[u] = load(k + u, end);
#pragma unroll
                for (int u = 0; u < 4; u++) test(q[u], k + u, end);
            }
            if (again == 0) break;
            k = 0;
            end = again;
            again = 0;
        }
    }
    return (int)((to - k0) / stride);
}

// The lists of one bead as its keys come in ascending order.
struct ListWriter {
    int nlj, nlo, nla;
    bool overflow;
};
// The site tests of pairs_kernel (src/compute_cuda.cu:527-674) for one key:
// the planes they need are requested together, then decided as list_bits does.
struct PairPlanes {
    float4 p, u, l1, l2;
    int flags;
};
__device__ __forceinline__ PairPlanes pair_load(const DevBuffers &B, int nb, int jg, unsigned bits) {
    const float4 *fr = B.frame_in;
    PairPlanes J;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    J.p = bits ? fr[jg] : z;
    J.u = (bits & 1u) ? fr[nb + jg] : z;
    J.flags = (bits & 1u) ? B.flags[jg] : 0;
    J.l2 = (bits & 2u) ? fr[3 * nb + jg] : z;
    J.l1 = (bits & 4u) ? fr[2 * nb + jg] : z;
    return J;
}
__device__ __forceinline__ void pair_decide(const KParams &P, const DevBuffers &B, int g, const ListSite &I, int jl,
                                            unsigned bits, const PairPlanes &J, float t_site, ListWriter &W) {
    unsigned got = 0;
    if ((bits & 1u) && ((I.flags ^ J.flags) & kFlagBeta)) {
        const float3 wj = make_float3(-J.u.x * I.rmon, -J.u.y * I.rmon, -J.u.z * I.rmon);
        if (norm2_rn(site_delta(I.p, J.p, I.wi, wj)) < t_site) got |= 2u;
    }
    if ((bits & 2u) && norm2_rn(site_delta(I.p, J.p, f3(I.l1), f3(J.l2))) < t_site) got |= 4u;
    if ((bits & 4u) && norm2_rn(site_delta(I.p, J.p, f3(I.l2), f3(J.l1))) < t_site) got |= 8u;
    if (got == 0) return;
    list_append(P, B, g, I, got, jl, W.nlj, W.nlo, W.nla, W.overflow);
}

// A hit as a key.  A bond needs the partner's centre within 2.5 + 2 nm of one of the bead's own
// sites (0.01 nm over the rounding of distances, and of a site's coordinates three units in the
// last place: beads may be far from the origin).
struct KeyTest {
    float4 p;             // the bead
    float3 a0, a1, a2;    // its sites
    float site, lj, pair; // squared limits
    int il, hpart;
    static __device__ __forceinline__ float site2(float3 a, float4 q) {   // a coarse test: contracted
        const float dx = a.x - q.x, dy = a.y - q.y, dz = a.z - q.z;
        return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    }
    __device__ __forceinline__ unsigned key(float4 q) const {
        const float r2 = dist2_rn(p, q);
        const int jl = __float_as_int(q.w);
        unsigned bits = (site2(a0, q) < site ? 1u : 0u) | (site2(a1, q) < site ? 2u : 0u) | (site2(a2, q) < site ? 4u : 0u);
        if (!(r2 < pair) || jl == hpart) bits = 0;
        return r2 < lj && jl != il ? ((unsigned)jl << 3) | bits : kNoKey;
    }
};
__device__ __forceinline__ KeyTest key_test(const KParams &P, const ListSite &I, const ListCuts &cut) {
    const float4 p = I.p;
    const float reach = fmaf(4.0e-7f, fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z)), 4.51f);
    return {p, make_float3(p.x + I.wi.x, p.y + I.wi.y, p.z + I.wi.z), make_float3(p.x + I.l1.x, p.y + I.l1.y, p.z + I.l1.z),
            make_float3(p.x + I.l2.x, p.y + I.l2.y, p.z + I.l2.z), P.is_assembly ? reach * reach : 0.f, cut.lj, cut.pair,
            I.il, I.hpart};
}
// The next n keys of a bead's column, ascending, into its lists; before: the last key taken.
__device__ __forceinline__ void take_keys(const KParams &P, const DevBuffers &B, const ListSite &I, int g, int base,
                                          float t_site, int n, uint16_t *col, unsigned &before, ListWriter &W) {
    // the LJ list; the keys with a site test close up in place
    int np = 0;
    for (int k = 0; k < n; k++) {
        const unsigned key = col[k * kListThreads];
        const bool keep = key != before;   // not found from two rows
        before = key;
        if (keep && W.nlj < P.maxLJ) B.lj[W.nlj * P.nb + g] = (int)(key >> 3);
        W.nlj += keep;
        col[np * kListThreads] = (uint16_t)key;   // np <= k
        np += keep && (key & 7u) != 0;
    }
    W.overflow = W.overflow || W.nlj > P.maxLJ;
    for (int k = 0; k < np; k += 2) {   // two partners in flight
        const unsigned k0 = col[k * kListThreads], k1 = k + 1 < np ? col[(k + 1) * kListThreads] : 0u;
        const PairPlanes J0 = pair_load(B, P.nb, base + (int)(k0 >> 3), k0 & 7u);
        const PairPlanes J1 = pair_load(B, P.nb, base + (int)(k1 >> 3), k1 & 7u);
        pair_decide(P, B, g, I, (int)(k0 >> 3), k0 & 7u, J0, t_site, W);
        pair_decide(P, B, g, I, (int)(k1 >> 3), k1 & 7u, J1, t_site, W);
    }
}
__device__ __forceinline__ void store_counts(const KParams &P, const DevBuffers &B, int g, const ListWriter &W) {
    B.ljc[g] = min(W.nlj, P.maxLJ);
    if (P.is_assembly) {
        B.lonc[g] = min(W.nlo, P.maxLong);
        B.latc[g] = min(W.nla, P.maxLat);
    }
    if (W.overflow) atomicOr(B.err, kErrOverflow);
}
// The lists of a bead with more hits than its slots hold (long cutoffs, dense systems): the
// smallest keys above the last one taken, kept in order as a walk meets them (a key can come
// twice), slots after slots.  A call that starts from the bead's index, so that the
// ordinary path keeps its registers.  256 x 1520 beads with a cutoff of 10, 12, 14 nm: 254, 508,
// 832 us; 1374, 4175, 8243 with a walk for every entry; 503, 880, 1576 in the general path (which is
// ahead in one corner measured: 40 x 8100 beads at 12 nm, up to 68 hits, 1380 against 1260).
static __device__ __noinline__ void many_hits(const KParams &P, const DevBuffers &B, SmemCells C, ListCuts cut, int g,
                                              int il, uint16_t *col) {
    const int nb = P.nb;
    const float4 *fr = B.frame_in;
    const ListSite I =
        list_site(P, fr[g], fr[nb + g], fr[2 * nb + g], fr[3 * nb + g], B.flags[g], il, B.harm[g * P.maxH]);
    const KeyTest K = key_test(P, I, cut);
    ListWriter W = {0, 0, 0, false};
    unsigned before = kNoKey;
    int n, last = -1;
    do {
        n = 0;
        smem_candidates(C, K.p, K.lj, [&](float4 q) {
            const unsigned key = K.key(q);
            if (key == kNoKey || (int)key <= last || (n == kSmemKeys && key >= col[(kSmemKeys - 1) * kListThreads])) return;
            int k = n < kSmemKeys ? n++ : kSmemKeys - 1;
            for (; k > 0 && col[(k - 1) * kListThreads] > key; k--) col[k * kListThreads] = col[(k - 1) * kListThreads];
            col[k * kListThreads] = (uint16_t)key;
        });
        if (n > 0) last = col[(n - 1) * kListThreads];
        take_keys(P, B, I, g, g - il, cut.site, n, col, before, W);
    } while (n == kSmemKeys);
    store_counts(P, B, g, W);
}

template <int PARTS>
__global__ void __launch_bounds__(kListThreads, 2) k_cell_lists_smem(const __grid_constant__ KParams P,
                                                                  const __grid_constant__ DevBuffers B, const int4 *work, int nmax,
                                                                  float inv, ListCuts cut) {
    extern __shared__ float4 s_dyn[];
    const int4 w = work[blockIdx.x];   // trajectory, first bead, number of beads
    const int base = B.off[w.x], n = B.off[w.x + 1] - base, nb = P.nb;
    const int m = row_buckets(n), t = threadIdx.x;
    const float4 *fr = B.frame_in;
    float4 *s_pos = s_dyn;
    unsigned *s_tab = reinterpret_cast<unsigned *>(s_dyn + nmax + 3);         // two 16-bit buckets a word
    uint16_t *s_end = reinterpret_cast<uint16_t *>(s_tab);
    uint16_t (*s_key)[kListThreads] = reinterpret_cast<uint16_t (*)[kListThreads]>(s_end + row_buckets(nmax));
    __shared__ unsigned s_warp[kListThreads / 32];
    __shared__ uint8_t s_count[kListThreads];

    // the beads in bucket order
    for (int k = t; k < m / 2; k += kListThreads) s_tab[k] = 0;
    chain_wait();   // no kernel writes the plan that was read so far
    __syncthreads();
    auto bucket = [&](float4 p) {
        return (int)((row_hash(cell_coord(p.y, inv), cell_coord(p.z, inv)) + (uint32_t)cell_coord(p.x, inv)) &
                     (uint32_t)(m - 1));
    };
    // the first beads of a thread stay in registers until the fill (read again there: 62.4
    // against 61.1 us for 256 x 1520 beads)
    constexpr int kKeep = 4;
    float4 kept[kKeep];
#pragma unroll
    for (int k = 0; k < kKeep; k++)
        if (t + k * kListThreads < n) kept[k] = fr[base + t + k * kListThreads];
    auto count = [&](float4 p) {
        const int b = bucket(p);
        atomicAdd(&s_tab[b >> 1], 1u << (16 * (b & 1)));
    };
#pragma unroll
    for (int k = 0; k < kKeep; k++)
        if (t + k * kListThreads < n) count(kept[k]);
    for (int j = t + kKeep * kListThreads; j < n; j += kListThreads) count(fr[base + j]);
    __syncthreads();
    {   // exclusive scan of the counts, whole words a thread
        const int per = (m / 2 + kListThreads - 1) / kListThreads, lo = min(m / 2, t * per), hi = min(m / 2, lo + per);
        unsigned sum = 0;
        for (int k = lo; k < hi; k++) sum += (s_tab[k] & 0xffffu) + (s_tab[k] >> 16);
        const int lane = t & 31, wid = t >> 5;
        unsigned v = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) s_warp[wid] = v;
        __syncthreads();
        unsigned run = v - sum + __reduce_add_sync(0xffffffffu, lane < wid ? s_warp[lane] : 0u);
        for (int k = lo; k < hi; k++) {
            const unsigned c = s_tab[k], c0 = c & 0xffffu;
            s_tab[k] = run | ((run + c0) << 16);
            run += c0 + (c >> 16);
        }
    }
    __syncthreads();
    auto place = [&](int j, float4 p) {
        const int b = bucket(p), sh = 16 * (b & 1);
        const unsigned slot = (atomicAdd(&s_tab[b >> 1], 1u << sh) >> sh) & 0xffffu;
        p.w = __int_as_float(j);
        s_pos[slot] = p;
    };
#pragma unroll
    for (int k = 0; k < kKeep; k++)
        if (t + k * kListThreads < n) place(t + k * kListThreads, kept[k]);
    for (int j = t + kKeep * kListThreads; j < n; j += kListThreads) place(j, fr[base + j]);
    __syncthreads();

    // the bead of this thread, and which of the bead's threads it is
    constexpr int cap = kListThreads / PARTS;
    const int part = t / cap, il = w.y - base + t % cap, g = base + il;
    const bool valid = t % cap < w.z;
    if (PARTS == 1 && !valid) return;   // no barrier after this point
    const int flags = valid ? B.flags[g] : kFlagExtra;
    const bool live = !(flags & kFlagExtra);
    const SmemCells C = {s_pos, s_end, n, m, inv};
    ListSite I;
    KeyTest K;
    auto make_key = [&](int slot) { return K.key(s_pos[slot]); };
    int nk = 0;
    bool many = false;
    if (live) {
        const float4 p = fr[g];
        const int met = smem_slots(C, p, cut.lj, part * 9 / PARTS, (part + 1) * 9 / PARTS, &s_key[0][t]);
        // the bead's other planes only now: the walk has no registers to spare
        I = list_site(P, p, fr[nb + g], fr[2 * nb + g], fr[3 * nb + g], flags, il, B.harm[g * P.maxH]);
        K = key_test(P, I, cut);
        many = met > kSmemKeys - 4;
        if (!many)
            for (int k = 0; k < met; k++) {
                const unsigned key = make_key(s_key[k][t]);
                s_key[nk][t] = (uint16_t)key;   // nk <= k
                nk += key != kNoKey;
            }
    }
    if (PARTS > 1) {   // the keys of the bead's other threads join those of its first
        s_count[t] = (uint8_t)(many ? 255 : nk);
        __syncthreads();
        if (part > 0) return;
        for (int o = t + cap; o < kListThreads && live; o += cap) {
            const int c = s_count[o];
            many = many || nk + c > kSmemKeys;
            for (int k = 0; k < c && !many; k++) s_key[nk++][t] = s_key[k][o];
        }
    }
    if (!valid) return;
    ListWriter W = {0, 0, 0, false};
    if (live) {
        if (many) {
            many_hits(P, B, C, cut, g, il, &s_key[0][t]);
            return;
        }
        // one way for the whole warp: a warp with both would run both
        const unsigned warp = __activemask();
        if (!__any_sync(warp, nk > 8)) {
            sort_keys<8>(s_key, nk);
        } else if (!__any_sync(warp, nk > 16)) {
            sort_keys<16>(s_key, nk);
        } else if (!__any_sync(warp, nk > 24)) {
            sort_keys<24>(s_key, nk);
        } else {
            for (int i = 1; i < nk; i++) {
                const uint16_t v = s_key[i][t];
                int j = i - 1;
                while (j >= 0 && s_key[j][t] > v) {
                    s_key[j + 1][t] = s_key[j][t];
                    j--;
                }
                s_key[j + 1][t] = v;
            }
        }
        unsigned before = kNoKey;
        take_keys(P, B, I, g, base, cut.site, nk, &s_key[0][t], before, W);
    }
    store_counts(P, B, g, W);
}

// ------------------------------------------------ ordered binning in one CTA
// bin_beads with ordered buckets, one CTA per trajectory of up to kOrderBeads
// beads: counts, scan and fill in shared memory, then every bead's rank among the
// beads of its bucket (ascending index, so that sums over a bucket are
// reproducible) and its place in the ordered copy.  Also the trajectory's centroid
// and non-extra count.  Before: five launches, the sort with one thread a bucket
// in global memory; 64 x 5600 beads 138 us, 40 us so.
constexpr int kOrderThreads = kStatsThreads;
constexpr int kOrderBeads = 16384;
__host__ __device__ inline int order_buckets(int n) {   // the table sizes of CellBuffers
    int m = 32;
    while (m < n) m <<= 1;
    return m;
}
inline size_t order_bytes(int nmax) { return sizeof(uint16_t) * ((size_t)order_buckets(nmax) + nmax); }

__global__ void __launch_bounds__(kOrderThreads) k_cell_order(KParams P, DevBuffers B, CellBuffers C, float inv,
                                                              float4 *stats) {
    extern __shared__ unsigned s_tab[];                     // two 16-bit buckets a word, then the indices
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, traj = blockIdx.x;
    const int base = B.off[traj], n = B.off[traj + 1] - base, tb = C.tbase[traj], m = C.tmask[traj] + 1;
    uint16_t *s_end = reinterpret_cast<uint16_t *>(s_tab), *s_idx = s_end + m;
    __shared__ unsigned s_warp[kOrderThreads / 32];
    for (int k = t; k < m / 2; k += kOrderThreads) s_tab[k] = 0;
    __syncthreads();
    auto bucket = [&](float4 p) {
        return (int)(cell_hash(cell_coord(p.x, inv), cell_coord(p.y, inv), cell_coord(p.z, inv)) & (uint32_t)(m - 1));
    };
    TrajStats S;
    for (int j = t; j < n; j += kOrderThreads) {
        const float4 p = B.frame_in[base + j];
        const int b = bucket(p);
        atomicAdd(&s_tab[b >> 1], 1u << (16 * (b & 1)));
        if (!(B.flags[base + j] & kFlagExtra)) S.add(p);
    }
    S.store(stats + traj);
    __syncthreads();
    {   // exclusive scan of the counts, whole words a thread
        const int per = (m / 2 + kOrderThreads - 1) / kOrderThreads, lo = min(m / 2, t * per), hi = min(m / 2, lo + per);
        unsigned sum = 0;
        for (int k = lo; k < hi; k++) sum += (s_tab[k] & 0xffffu) + (s_tab[k] >> 16);
        unsigned v = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) s_warp[wid] = v;
        __syncthreads();
        unsigned run = v - sum;
        for (int k = 0; k < wid; k++) run += s_warp[k];
        for (int k = lo; k < hi; k++) {
            const unsigned both = s_tab[k], c0 = both & 0xffffu, c1 = both >> 16;
            s_tab[k] = run | ((run + c0) << 16);
            C.start[tb + 2 * k] = (int)run;
            C.start[tb + 2 * k + 1] = (int)(run + c0);
            C.cnt[tb + 2 * k] = (int)c0;
            C.cnt[tb + 2 * k + 1] = (int)c1;
            run += c0 + c1;
        }
    }
    __syncthreads();
    for (int j = t; j < n; j += kOrderThreads) {
        const int b = bucket(B.frame_in[base + j]), sh = 16 * (b & 1);
        s_idx[(atomicAdd(&s_tab[b >> 1], 1u << sh) >> sh) & 0xffffu] = (uint16_t)j;
    }
    __syncthreads();
    for (int j = t; j < n; j += kOrderThreads) {
        const int g = base + j;
        float4 p = B.frame_in[g];
        const int b = bucket(p), e = s_end[b];
        int slot = b > 0 ? s_end[b - 1] : 0;
        int rank = 0;
        for (int k = slot; k < e; k++) rank += s_idx[k] < j;
        slot += rank;
        C.cell_bead[base + slot] = g;
        p.w = __int_as_float(g | ((B.flags[g] & kFlagExtra) ? kCellExtraBit : 0));
        C.cell_pos[base + slot] = p;
    }
}

inline int nblk(int n, int t) { return (n + t - 1) / t; }

}  // namespace

float bin_beads(const KParams &P, const DevBuffers &B, const CellBuffers &C, float reach, bool ordered,
                cudaStream_t s) {
    // cells slightly larger than the reach, so that rounding of x / edge can
    // never put two beads closer than the reach two cells apart
    const float inv = 1.0f / (reach * 1.001f + 1e-3f);
    cudaMemsetAsync(C.cnt, 0, sizeof(int) * C.nbuckets, s);
    k_cell_count<<<nblk(P.nb, 256), 256, 0, s>>>(P, B.frame_in, B.traj, C.tbase, C.tmask, inv, C.key, C.cnt);
    k_cell_scan<<<P.nt, 1024, 0, s>>>(C.tbase, C.cnt, C.start, C.cursor);
    k_cell_fill<<<nblk(P.nb, 256), 256, 0, s>>>(P.nb, B.traj, B.off, C.key, B.flags, C.cursor, C.cell_bead,
                                                 B.frame_in, C.cell_pos);
    if (ordered)
        k_cell_sort<<<dim3(P.nt, (C.max_buckets + 127) / 128), 128, 0, s>>>(B.off, C.tbase, C.tmask, C.start, C.cnt,
                                                                            C.cell_bead, C.cell_pos);
    return inv;
}

bool order_beads_applies(int nmax) { return nmax <= kOrderBeads; }
int order_beads_prepare() {   // the limit of the largest trajectory: engines share the kernel
    return cudaFuncSetAttribute(k_cell_order, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)order_bytes(kOrderBeads)) == cudaSuccess
               ? 0
               : -1;
}
float order_beads(const KParams &P, const DevBuffers &B, const CellBuffers &C, float reach, int nmax, float4 *stats,
                  cudaStream_t s) {
    const float inv = 1.0f / (reach * 1.001f + 1e-3f);   // the cells of bin_beads
    k_cell_order<<<P.nt, kOrderThreads, order_bytes(nmax), s>>>(P, B, C, inv, stats);
    return inv;
}

bool smem_lists_apply(const KParams &P, int nmax) {
    return P.lj_on && P.ljcut > 0.0f && (!P.is_assembly || P.ljcut >= kPairReach) && nmax <= kSmemBeads;
}
int smem_lists_resident(int nmax) { return smem_list_bytes(nmax) <= 112 * 1024 ? 2 : 1; }
int smem_lists_prepare() {   // the limit of the largest trajectory, whatever this engine's, as engines share the kernel
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int bytes = (int)smem_list_bytes(kSmemBeads);
    return cudaFuncSetAttribute(k_cell_lists_smem<1>, attr, bytes) == cudaSuccess &&
                   cudaFuncSetAttribute(k_cell_lists_smem<2>, attr, bytes) == cudaSuccess &&
                   cudaFuncSetAttribute(k_cell_lists_smem<4>, attr, bytes) == cudaSuccess
               ? 0
               : -1;
}
// The smallest float whose rounded square root is not below c, so that
// r2 < sq_below(c) decides as sqrt(r2) < c does.
static float sq_below(float c) {
    if (!(c > 0.0f)) return 0.0f;
    float t = c * c;
    while (std::sqrt(t) >= c && t > 0.0f) t = std::nextafter(t, 0.0f);
    while (std::sqrt(t) < c) t = std::nextafter(t, INFINITY);
    return t;
}
ListCuts list_cuts(const KParams &P) { return {sq_below(P.ljcut), sq_below(kPairReach), sq_below(2.5f)}; }

void launch_rebuild_smem(const KParams &P, const DevBuffers &B, const int4 *work, int nwork, int parts, int nmax,
                         cudaStream_t s) {
    const float inv = 1.0f / (P.ljcut * 1.001f + 1e-3f);   // the cells of bin_beads
    const auto kernel = parts == 4 ? k_cell_lists_smem<4> : parts == 2 ? k_cell_lists_smem<2> : k_cell_lists_smem<1>;
    launch_chained(P, kernel, nwork, kListThreads, smem_list_bytes(nmax), s, P, B, work, nmax, inv, list_cuts(P));
}

void launch_rebuild_cells(const KParams &P, const DevBuffers &B, const CellBuffers &C, const int2 *work, int nwork,
                          cudaStream_t s) {
    const float reach = fmaxf(P.lj_on ? P.ljcut : 0.f, P.is_assembly ? kPairReach : 0.f);
    const float inv = bin_beads(P, B, C, reach, false, s);   // the lists are sorted afterwards
    if (P.is_assembly && P.lj_on && P.ljcut >= kPairReach) {
        // LJ lists from the cells, then the assembly lists from the LJ lists
        k_cell_lists<false><<<nwork, kTile, 0, s>>>(P, B, work, C.tbase, C.tmask, C.start, C.cnt, C.cell_pos, inv);
        k_pairs_from_lj<<<nblk(P.nb, kTile), kTile, 0, s>>>(P, B);
    } else {
        k_cell_lists<true><<<nwork, kTile, 0, s>>>(P, B, work, C.tbase, C.tmask, C.start, C.cnt, C.cell_pos, inv);
    }
}

}  // namespace mtg
