// Cluster neighbour lists of the resident engine.
//
// The reference rebuilds O(N^2) Verlet lists with a 4 A skin on the host and
// re-uploads 33 B per pair (src/neighbors.rs:102-281,
// src/gpu_interface.rs:243-410).  Here the rebuild runs on the device:
//   1. molecules / atoms are binned into columns of an xy grid and ranked by
//      z inside each column (deterministic: ties broken by index);
//   2. waters are physically permuted into that order, columns padded to a
//      multiple of 8, so every aligned 8-slot group is a compact cluster;
//   3. cluster bounding boxes are tested against each other (all pairs,
//      min-image on centres) and each i-cluster's hits are compacted with
//      warp ballots into a fixed-capacity list, ascending in j;
//   4. for water-water, 32-water groups get a tile of j-clusters and every
//      water a compact list of tile-local molecule indices (O-O distance
//      below cutoff + twice the O-H reach + buffer).
// Every kernel of the rebuild returns immediately unless the displacement
// check raised Scalars::need_rebuild; inside a captured step graph the
// rebuild kernels also sit under a conditional (switch) node that the check
// sets, so steps without a rebuild launch none of them.  The rebuild criterion is the reference's: max displacement since
// the last rebuild >= buffer / 2 (src/neighbors.rs:159-169), tracking water
// O only (src/neighbors.rs:71-82); water list radii add twice the O-H reach.
#include <algorithm>

#include "engine.cuh"

namespace {

__device__ __forceinline__ bool rebuild_on(const SysView& v, bool force) {
    return force || v.sc->need_rebuild;
}

__device__ __forceinline__ float frac_box(float x, float lo, float inv_ext) {
    float f = (x - lo) * inv_ext;
    f -= floorf(f);
    return f >= 1.0f ? 0.0f : f;
}

// Column rank along a boustrophedon path over the xy grid, and the sort key
// inside the column: z ascending in even-ranked columns, descending in odd
// ones, so consecutive slots are neighbours in space across column ends too.
__device__ __forceinline__ uint32_t column_of(float3 p, const BoxDev& b, uint32_t ncx, uint32_t ncy,
                                              float* key) {
    const float fx = frac_box(p.x, b.lo[0], b.inv_ext[0]);
    const float fy = frac_box(p.y, b.lo[1], b.inv_ext[1]);
    const float fz = frac_box(p.z, b.lo[2], b.inv_ext[2]);
    const uint32_t cx = min((uint32_t)(fx * ncx), ncx - 1);
    const uint32_t cy = min((uint32_t)(fy * ncy), ncy - 1);
    const uint32_t rank = cy * ncx + ((cy & 1u) ? (ncx - 1 - cx) : cx);
    *key = (rank & 1u) ? 1.0f - fz : fz;
    return rank;
}

// ---------------------------------------------------------------------------
// displacement check of an evaluation without a step; a step's first half
// checks as it moves (integrate.cu)
// ---------------------------------------------------------------------------
DYN_KERNEL(, k_disp_check, (), ()) {
    const BoxDev b = *v.box;
    float m = 0.f, mp = 0.f;
    const uint32_t tid = bk.idx * blockDim.x + threadIdx.x;
    const uint32_t stride = bk.cnt * blockDim.x;
    for (uint32_t s = tid; s < v.nw_cap; s += stride) {
        if (v.wid[s] == INVALID_ID) continue;
        const float3 o = xyz(v.wpos[4 * s]);
        const float3 d = min_image_rint(o - xyz(v.wref[s]), b);
        const float d2 = dot3(d, d);
        m = fmaxf(m, isfinite(d2) ? d2 : 1e30f);
        // since the last prune of the water-water lists
        const float3 dp = min_image_rint(o - xyz(v.wprune[s]), b);
        const float dp2 = dot3(dp, dp);
        mp = fmaxf(mp, isfinite(dp2) ? dp2 : 1e30f);
    }
    for (uint32_t a = tid; a < v.na; a += stride) {
        const float3 d = xyz(v.apos[a]) - xyz(v.aref[a]);
        const float d2 = dot3(d, d);
        m = fmaxf(m, isfinite(d2) ? d2 : 1e30f);
    }
    displacement_vote(v, m, mp, bk.cnt);
}

// ---------------------------------------------------------------------------
// column binning.  Six short kernels, each bound by the latency of a few
// dependent loads, so the chain is kept short and every thread does little:
// one atomic per column and warp, a block-wide scan, ranks counted from keys
// in shared memory, and the bounding boxes taken from registers as the
// permuted waters are copied back.  24,000 waters and 5,000 atoms: 32 us,
// against 144 us for ten kernels with an atomic per element, a serial scan
// (25), ranks counted in global memory (55) and a thread per box (23).
// ---------------------------------------------------------------------------
DYN_KERNEL(, k_col_clear, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const uint32_t tid = bk.idx * blockDim.x + threadIdx.x, stride = bk.cnt * blockDim.x;
    if (tid == 0) {
        v.sc->list_pairs = 0ull;
        v.sc->union_max = 0u;
    }
    const uint32_t nc = v.ncol > v.ancol ? v.ncol : v.ancol;
    for (uint32_t c = tid; c < nc; c += stride) {
        if (c < v.ncol) v.col_count[c] = 0;
        if (c < v.ancol) v.acol_count[c] = 0;
    }
    // the padding of the sorted order: slots no water or atom is moved to
    for (uint32_t s = v.nw + tid; s < v.nw_cap; s += stride) {
        v.wtmp_id[s] = INVALID_ID;
        for (int k = 0; k < 10; ++k) v.wtmp[10 * s + k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (uint32_t s = tid; s < v.na_cap; s += stride) {
        v.sidx[s] = INVALID_ID;
        v.slj[s] = make_float2(0.f, 0.f);
        v.spos[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// The place of each lane's element in its column's bucket (any order): one
// atomic per column and warp, as neighbours in slot order mostly share one.
__device__ __forceinline__ uint32_t column_place(uint32_t* count, uint32_t c, bool has, int lane) {
    const uint32_t peers = __match_any_sync(0xffffffffu, has ? c : INVALID_ID);
    const int leader = __ffs(peers) - 1;
    uint32_t first = 0;
    if (has && lane == leader) first = atomicAdd(&count[c], (uint32_t)__popc(peers));
    first = __shfl_sync(0xffffffffu, first, leader);
    return first + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

DYN_KERNEL(, k_col_assign, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const BoxDev b = *v.box;
    const int lane = threadIdx.x & 31;
    const uint32_t w0 = bk.idx * blockDim.x + (threadIdx.x & ~31u);
    const uint32_t stride = bk.cnt * blockDim.x;
    for (uint32_t s0 = w0; s0 < v.nw_cap; s0 += stride) {
        const uint32_t s = s0 + lane;
        const bool has = s < v.nw_cap && v.wid[s] != INVALID_ID;
        float zf = 0.f;
        uint32_t c = 0;
        if (has) c = column_of(xyz(v.wpos[4 * s]), b, v.ncx, v.ncy, &zf);
        const uint32_t pos = column_place(v.col_count, c, has, lane);
        if (has) {
            v.wcol[s] = c;
            v.wkey[s] = zf;
            v.wplace[s] = pos;
        }
    }
    for (uint32_t a0 = w0; a0 < v.na; a0 += stride) {
        const uint32_t a = a0 + lane;
        const bool has = a < v.na && v.asparse[a] == INVALID_ID;
        float zf = 0.f;
        uint32_t c = 0;
        if (has) c = column_of(xyz(v.apos[a]), b, v.ancx, v.ancy, &zf);
        const uint32_t pos = column_place(v.acol_count, c, has, lane);
        if (has) {
            v.acol[a] = c;
            v.akey[a] = zf;
            v.aplace[a] = pos;
        }
    }
}

// Exclusive sums of the column counts in path order, by one block; slots are
// contiguous along the path, padding sits at the end.  (A serial loop over
// the 529 atom columns of a 98 A box took 25 us, the block scan 3.)
constexpr int SCT = 1024;
__device__ __forceinline__ uint32_t block_scan_off(const uint32_t* cnt, uint32_t* off, uint32_t n, uint32_t* wsum) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t base = 0;
    for (uint32_t c0 = 0; c0 < n; c0 += SCT) {
        const uint32_t c = c0 + threadIdx.x;
        const uint32_t k = c < n ? cnt[c] : 0u;
        uint32_t x = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t t = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            wsum[lane] = t;
        }
        __syncthreads();
        if (c < n) off[c] = base + (w ? wsum[w - 1] : 0u) + x - k;
        base += wsum[SCT / 32 - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) off[n] = base;
    return base;
}

DYN_KERNEL(__launch_bounds__(SCT), k_col_scan, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    __shared__ uint32_t wsum[SCT / 32];
    const uint32_t qw = block_scan_off(v.col_count, v.col_off, v.ncol, wsum);
    const uint32_t qa = block_scan_off(v.acol_count, v.acol_off, v.ancol, wsum);
    if (threadIdx.x == 0) {
        v.sc->n_wclus = (qw + WCL - 1) / WCL;
        // clustered atoms fill whole clusters from slot 0; each atom without
        // bonds then gets a cluster of its own
        const uint32_t base = (qa + ACL - 1) / ACL * ACL;
        v.sc->a_sparse_base = base;
        v.sc->n_aclus = base / ACL + v.n_sparse;
    }
}

// Sort key of a column member: z (a non-negative float, so its bits order
// as it does), then the original index.
__device__ __forceinline__ unsigned long long column_key(float z, uint32_t id) {
    return (unsigned long long)__float_as_uint(z) << 32 | id;
}

DYN_KERNEL(, k_col_bucket, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const uint32_t tid = bk.idx * blockDim.x + threadIdx.x;
    const uint32_t stride = bk.cnt * blockDim.x;
    for (uint32_t s = tid; s < v.nw_cap; s += stride) {
        const uint32_t id = v.wid[s];
        if (id == INVALID_ID) continue;
        const uint32_t e = v.col_off[v.wcol[s]] + v.wplace[s];
        v.bucket[e] = s;
        v.bkey[e] = column_key(v.wkey[s], id);
    }
    for (uint32_t a = tid; a < v.na; a += stride) {
        if (v.asparse[a] != INVALID_ID) continue;
        const uint32_t e = v.acol_off[v.acol[a]] + v.aplace[a];
        v.abucket[e] = a;
        v.abkey[e] = column_key(v.akey[a], a);
    }
}

// Atom a's entry of the cluster order.
__device__ __forceinline__ void place_atom(const SysView& v, uint32_t a, uint32_t s) {
    const float4 p = v.apos[a];
    v.aslot[a] = s;
    v.sidx[s] = a;
    v.slj[s] = v.alj[a];
    v.spos[s] = p;
    v.aref[a] = p;
}

// Rank inside the column by (z, original index), a deterministic order, and
// the move there: a CTA per water column counts smaller keys from shared
// memory (294 of them at 24,000 waters), a warp per atom column (some ten
// atoms) straight from the bucket.  24,000 waters: 14 us with the move (55
// and 5.5 before, two dependent global loads per compare).
constexpr int RKT = 512;
constexpr uint32_t RK_CHUNK = 1024;

DYN_KERNEL(__launch_bounds__(RKT), k_col_rank, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    __shared__ unsigned long long key[RK_CHUNK];
    const int tid = threadIdx.x, lane = tid & 31;
    for (uint32_t c = bk.idx; c < v.ncol; c += bk.cnt) {
        const uint32_t b0 = v.col_off[c], n = v.col_off[c + 1] - b0;
        for (uint32_t i0 = 0; i0 < n; i0 += RKT) {
            const uint32_t i = i0 + tid;
            const unsigned long long mine = i < n ? v.bkey[b0 + i] : 0ull;
            uint32_t r = 0;
            for (uint32_t k0 = 0; k0 < n; k0 += RK_CHUNK) {
                const uint32_t m = min(RK_CHUNK, n - k0);
                if (i0 == 0 || n > RK_CHUNK) {
                    __syncthreads();  // the keys of the chunk before are done with
                    for (uint32_t t = tid; t < m; t += RKT) key[t] = v.bkey[b0 + k0 + t];
                    __syncthreads();
                }
#pragma unroll 8
                for (uint32_t k = 0; k < m; ++k) r += key[k] < mine ? 1u : 0u;
            }
            if (i < n) {
                const uint32_t s = v.bucket[b0 + i], d = b0 + r;
                float4 q[10];
#pragma unroll
                for (int k = 0; k < 4; ++k) q[k] = v.wpos[4 * s + k];
#pragma unroll
                for (int k = 0; k < 3; ++k) { q[4 + k] = v.wvel[3 * s + k]; q[7 + k] = v.wacc[3 * s + k]; }
#pragma unroll
                for (int k = 0; k < 10; ++k) v.wtmp[10 * d + k] = q[k];
                v.wtmp_id[d] = v.wid[s];
            }
        }
        __syncthreads();  // every thread is done with the column's keys
    }
    const uint32_t gw = (bk.idx * blockDim.x + tid) >> 5, nwarps = (bk.cnt * blockDim.x) >> 5;
    for (uint32_t c = gw; c < v.ancol; c += nwarps) {
        const uint32_t b0 = v.acol_off[c], n = v.acol_off[c + 1] - b0;
        for (uint32_t i = lane; i < n; i += 32) {
            const unsigned long long mine = v.abkey[b0 + i];
            uint32_t r = 0;
            for (uint32_t k = 0; k < n; ++k) r += v.abkey[b0 + k] < mine ? 1u : 0u;
            place_atom(v, v.abucket[b0 + i], b0 + r);
        }
    }
    for (uint32_t a = bk.idx * blockDim.x + tid; a < v.na; a += bk.cnt * blockDim.x)
        if (v.asparse[a] != INVALID_ID) place_atom(v, a, v.sc->a_sparse_base + ACL * v.asparse[a]);
}

// Bounding box over the W lanes of a cluster (W = 8) or group (32): members
// min-imaged to the first valid one, so a cluster straddling a periodic face
// still gets a compact box; lanes without a member leave it unchanged.
template <int W>
__device__ __forceinline__ void lanes_bbox(float3 p, bool ok, const BoxDev& b, int lane, float4* cen, float4* half) {
    const uint32_t all = __ballot_sync(0xffffffffu, ok);
    const int l0 = lane & ~(W - 1);
    const uint32_t m = W == 32 ? all : (all >> l0) & ((1u << (W & 31)) - 1u);
    const int src = m ? l0 + __ffs(m) - 1 : lane;
    const float3 ref = f3(__shfl_sync(0xffffffffu, p.x, src), __shfl_sync(0xffffffffu, p.y, src),
                          __shfl_sync(0xffffffffu, p.z, src));
    const float3 q = ref + min_image_rint(p - ref, b);
    float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
    if (ok) { lo[0] = hi[0] = q.x; lo[1] = hi[1] = q.y; lo[2] = hi[2] = q.z; }
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    }
    if (!m)
        for (int k = 0; k < 3; ++k) lo[k] = hi[k] = 0.f;
    *cen = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), 0.f);
    *half = make_float4(0.5f * (hi[0] - lo[0]), 0.5f * (hi[1] - lo[1]), 0.5f * (hi[2] - lo[2]), 0.f);
}

// The sorted waters back into place, with the bounding boxes (over O) of
// their clusters and groups, and those of the atom clusters.
DYN_KERNEL(, k_perm_copyback, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const BoxDev b = *v.box;
    const int lane = threadIdx.x & 31;
    const uint32_t w0 = bk.idx * blockDim.x + (threadIdx.x & ~31u);
    const uint32_t stride = bk.cnt * blockDim.x;
    // nw_cap is a multiple of 64: whole warps
    for (uint32_t s0 = w0; s0 < v.nw_cap; s0 += stride) {
        const uint32_t s = s0 + lane;
        float4 q[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) q[k] = v.wtmp[10 * s + k];
        const uint32_t id = v.wtmp_id[s];
#pragma unroll
        for (int k = 0; k < 4; ++k) v.wpos[4 * s + k] = q[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) { v.wvel[3 * s + k] = q[4 + k]; v.wacc[3 * s + k] = q[7 + k]; }
        v.wid[s] = id;
        v.wref[s] = q[0];
        float4 c, h;
        lanes_bbox<WCL>(xyz(q[0]), id != INVALID_ID, b, lane, &c, &h);
        if ((lane & (WCL - 1)) == 0) { v.wbb_c[s / WCL] = c; v.wbb_h[s / WCL] = h; }
        lanes_bbox<GRPW>(xyz(q[0]), id != INVALID_ID, b, lane, &c, &h);
        if (lane == 0) { v.gbb_c[s / GRPW] = c; v.gbb_h[s / GRPW] = h; }
    }
    for (uint32_t s0 = w0; s0 < v.na_cap; s0 += stride) {
        const uint32_t s = s0 + lane;
        const bool in = s < v.na_cap;
        const bool ok = in && v.sidx[s] != INVALID_ID;
        const float3 p = ok ? xyz(v.spos[s]) : f3(0.f, 0.f, 0.f);
        float4 c, h;
        lanes_bbox<ACL>(p, ok, b, lane, &c, &h);
        if (in && (lane & (ACL - 1)) == 0) { v.abb_c[s / ACL] = c; v.abb_h[s / ACL] = h; }
    }
}

__device__ __forceinline__ float bb_dist2(float4 ci, float4 hi, float4 cj, float4 hj, const BoxDev& b) {
    float3 d = f3(ci.x - cj.x, ci.y - cj.y, ci.z - cj.z);
    d = min_image_rint(d, b);
    const float gx = fmaxf(0.f, fabsf(d.x) - hi.x - hj.x);
    const float gy = fmaxf(0.f, fabsf(d.y) - hi.y - hj.y);
    const float gz = fmaxf(0.f, fabsf(d.z) - hi.z - hj.z);
    return gx * gx + gy * gy + gz * gz;
}

// The exclusions of atom cluster ci taken out of its cluster pairs' masks:
// each partner's cluster is looked up in the cluster's (ascending) list, so
// the cost is that of the exclusions (some 12 per atom) and not of the list.
// Called by a whole warp after the masks are written.
__device__ __forceinline__ void clear_excluded(const SysView& v, uint32_t ci, uint32_t n, int lane) {
    uint32_t a = INVALID_ID, off = 0, len = 0;
    if (lane < ACL) {
        a = v.sidx[ci * ACL + lane];
        if (a != INVALID_ID) { off = v.ex_off[a]; len = v.ex_off[a + 1] - off; }
    }
    uint32_t end = len;  // inclusive sums over the cluster's atoms
#pragma unroll
    for (int o = 1; o < ACL; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, end, ACL - 1);
    const uint32_t* list = v.ss_j + (size_t)ci * v.cap_ss;
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const uint32_t t = t0 + lane;
        int ii = 0;
        uint32_t e = 0;
#pragma unroll
        for (int k = 0; k < ACL; ++k) {
            const uint32_t ek = __shfl_sync(0xffffffffu, end, k), lk = __shfl_sync(0xffffffffu, len, k);
            const uint32_t ok = __shfl_sync(0xffffffffu, off, k);
            if (t < ek && t >= ek - lk) { ii = k; e = ok + (t - (ek - lk)); }
        }
        if (t >= total) continue;
        const uint32_t s = v.aslot[v.ex_idx[e]], cj = s / ACL;
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
            const uint32_t m = (lo + hi) >> 1;
            if (list[m] < cj) lo = m + 1; else hi = m;
        }
        if (lo < n && list[lo] == cj)
            atomicAnd(&v.ss_mask[(size_t)ci * v.cap_ss + lo], ~(1ull << (ii * ACL + (int)(s % ACL))));
    }
}

// Atom-atom cluster pairs: one warp per i-cluster, against the clusters with
// cj >= ci (each cluster pair once), with the interaction mask of the cluster
// pair (jj > ii on the diagonal, exclusions and pairs of two static atoms
// removed).  LU blocks of 32 candidates are tested per turn, so that their
// boxes' loads are in flight together.  A lane makes its hit's mask as the
// product of the two clusters' valid-atom bits (one byte per i-atom); the
// exclusions are cleared afterwards.  5,000 atoms: 14 us, against 180 us when
// the 64 pairs of every hit were decided by binary searches in the exclusion
// lists.
constexpr int LU = 4;
DYN_KERNEL(, k_list_ss, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const BoxDev b = *v.box;
    const int lane = threadIdx.x & 31;
    const uint32_t ci = (bk.idx * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nc = v.sc->n_aclus;
    if (ci >= nc) return;
    const float r2 = v.r_ss * v.r_ss;
    const uint32_t cap = v.cap_ss;
    const float4 c0 = v.abb_c[ci], h0 = v.abb_h[ci];
    // a byte per i-atom: 1 where the slot holds an atom, and where that atom is static
    unsigned long long vi = 0ull, si = 0ull;
    {
        const uint32_t a = lane < ACL ? v.sidx[ci * ACL + lane] : INVALID_ID;
        const bool st = a != INVALID_ID && v.astatic && v.astatic[a];
        const uint32_t mv = __ballot_sync(0xffffffffu, a != INVALID_ID), ms = __ballot_sync(0xffffffffu, st);
#pragma unroll
        for (int k = 0; k < ACL; ++k) {
            vi |= (unsigned long long)((mv >> k) & 1u) << (8 * k);
            si |= (unsigned long long)((ms >> k) & 1u) << (8 * k);
        }
    }
    uint32_t cnt = 0;
    for (uint32_t jb = ci & ~31u; jb < nc; jb += 32 * LU) {
        bool hit[LU];
#pragma unroll
        for (int u = 0; u < LU; ++u) {
            const uint32_t cj = jb + 32 * u + lane;
            hit[u] = cj < nc && cj >= ci && bb_dist2(c0, h0, v.abb_c[cj], v.abb_h[cj], b) < r2;
        }
#pragma unroll
        for (int u = 0; u < LU; ++u) {
            const uint32_t cj = jb + 32 * u + lane;
            const uint32_t m = __ballot_sync(0xffffffffu, hit[u]);
            const uint32_t k = cnt + __popc(m & ((1u << lane) - 1u));
            cnt += __popc(m);
            if (!hit[u] || k >= cap) continue;
            v.ss_j[(size_t)ci * cap + k] = cj;
            const uint4* sj = reinterpret_cast<const uint4*>(v.sidx + (size_t)cj * ACL);
            const uint4 s0 = sj[0], s1 = sj[1];
            const uint32_t aj[ACL] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
            uint32_t vj = 0;
#pragma unroll
            for (int jj = 0; jj < ACL; ++jj) vj |= aj[jj] != INVALID_ID ? 1u << jj : 0u;
            unsigned long long mk = vi * vj;  // byte ii: the j-atoms, where i-atom ii exists
            if (si) {
                uint32_t sj8 = 0;
#pragma unroll
                for (int jj = 0; jj < ACL; ++jj)
                    if (aj[jj] != INVALID_ID && v.astatic[aj[jj]]) sj8 |= 1u << jj;
                mk &= ~(si * sj8);
            }
            if (cj == ci) mk &= 0x0080C0E0F0F8FCFEull;  // byte ii: the bits jj > ii
            v.ss_mask[(size_t)ci * cap + k] = mk;
        }
    }
    const uint32_t n = min(cnt, cap);
    if (v.ex_off) {
        __syncwarp();  // the list and the masks are written
        clear_excluded(v, ci, n, lane);
    }
    if (lane == 0) {
        v.ss_n[ci] = n;
        if (cnt > cap) atomicMax(&v.sc->overflow, cnt);
        atomicAdd(&v.sc->list_pairs, (unsigned long long)n);
    }
}

// The waters of every atom cluster: those whose O lies within the list radius
// of any of the cluster's atoms, ascending by slot; a CTA per cluster.  Of
// every WLC water clusters, those whose box meets the atom cluster's (four
// boxes in flight per thread) are tested water by water, two waters per
// thread.  Bound by latency; 750 clusters against 3,000 water clusters:
// 32 us (53 with one box and one water per thread and turn).
constexpr int WLT = 256, WLU = 4, WLW = 2;
constexpr int WLC = WLT * WLU;
DYN_KERNEL(__launch_bounds__(WLT), k_list_ws, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const BoxDev b = *v.box;
    const float r2 = v.r_ws * v.r_ws;
    const int tid = threadIdx.x, lane = tid & 31, wid_ = tid >> 5;
    constexpr int NWP = WLT / 32;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t nwc = v.sc->n_wclus, nac = v.sc->n_aclus;
    __shared__ float4 ap[ACL];
    __shared__ uint32_t cl[WLC];       // water clusters met by the box
    __shared__ uint32_t wt[WLU][NWP];
    // where this warp's hits of pass u start after base; base moves past all
    auto place = [&](uint32_t& base, int u) {
        uint32_t at = base;
#pragma unroll
        for (int w = 0; w < NWP; ++w) {
            if (w < wid_) at += wt[u][w];
            base += wt[u][w];
        }
        return at;
    };
    for (uint32_t ci = bk.idx; ci < nac; ci += bk.cnt) {
        if (tid < ACL) {
            const float4 p = v.spos[ci * ACL + tid];
            ap[tid] = make_float4(p.x, p.y, p.z, v.sidx[ci * ACL + tid] != INVALID_ID ? 1.f : 0.f);
        }
        const float4 c0 = v.abb_c[ci], h0 = v.abb_h[ci];
        uint32_t* out = v.ws_j + (size_t)ci * v.cap_ws;
        uint32_t cnt = 0;
        for (uint32_t jb = 0; jb < nwc; jb += WLC) {
            uint32_t m[WLU];
#pragma unroll
            for (int u = 0; u < WLU; ++u) {
                const uint32_t cj = jb + u * WLT + tid;
                m[u] = __ballot_sync(0xffffffffu, cj < nwc && bb_dist2(c0, h0, v.wbb_c[cj], v.wbb_h[cj], b) < r2);
                if (lane == 0) wt[u][wid_] = __popc(m[u]);
            }
            __syncthreads();
            uint32_t nc = 0;
#pragma unroll
            for (int u = 0; u < WLU; ++u) {
                const uint32_t at = place(nc, u);
                if ((m[u] >> lane) & 1u) cl[at + __popc(m[u] & lt)] = jb + u * WLT + tid;
            }
            __syncthreads();
            for (uint32_t k0 = 0; k0 < nc * WCL; k0 += WLT * WLW) {
                uint32_t slot[WLW], mn[WLW];
                bool near[WLW];
#pragma unroll
                for (int u = 0; u < WLW; ++u) {
                    const uint32_t k = k0 + u * WLT + tid;
                    const bool in = k < nc * WCL;
                    slot[u] = in ? cl[k / WCL] * WCL + (k % WCL) : 0u;
                    near[u] = in && v.wid[slot[u]] != INVALID_ID;
                }
#pragma unroll
                for (int u = 0; u < WLW; ++u) {
                    const float3 o = xyz(v.wpos[4 * slot[u]]);
                    bool any = false;
#pragma unroll
                    for (int i = 0; i < ACL; ++i) {
                        const float4 q = ap[i];
                        const float3 d = min_image_fast(o - xyz(q), b);
                        any = any || (q.w != 0.f && dot3(d, d) < r2);
                    }
                    near[u] = near[u] && any;
                    mn[u] = __ballot_sync(0xffffffffu, near[u]);
                    if (lane == 0) wt[u][wid_] = __popc(mn[u]);
                }
                __syncthreads();
#pragma unroll
                for (int u = 0; u < WLW; ++u) {
                    const uint32_t pos = place(cnt, u) + __popc(mn[u] & lt);
                    if (near[u] && pos < v.cap_ws) out[pos] = slot[u];
                }
                __syncthreads();  // the counts are refilled
            }
        }
        if (tid == 0) {
            v.ws_n[ci] = min(cnt, v.cap_ws);
            if (cnt > v.cap_ws) atomicMax(&v.sc->overflow, cnt);
            atomicAdd(&v.sc->list_pairs, (unsigned long long)min(cnt, v.cap_ws));
        }
        __syncthreads();  // the atoms are refilled
    }
}

// Work items of the atom pair kernels: for every atom cluster (in order) one
// item per 32 waters or ch_mix clusters of its list, {cluster, first
// entry}.  Block 0 the water-atom items, block 1 the atom-atom ones; an
// exclusive scan of the per-cluster item counts, tile by tile.
constexpr int IT_T = 1024;
DYN_KERNEL(__launch_bounds__(IT_T), k_items, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const bool ws = bk.idx == 0;
    if (ws && !v.nw) return;
    const uint32_t ni = v.sc->n_aclus;
    const uint32_t* cnt = ws ? v.ws_n : v.ss_n;
    uint2* items = ws ? v.ws_item : v.ss_item;
    const uint32_t icap = ws ? v.ws_item_cap : v.ss_item_cap;
    const uint32_t per = ws ? 32u : v.ch_mix;
    __shared__ uint32_t wsum[IT_T / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t base = 0;
    for (uint32_t c0 = 0; c0 < ni; c0 += IT_T) {
        const uint32_t c = c0 + threadIdx.x;
        const uint32_t k = c < ni ? (cnt[c] + per - 1) / per : 0u;
        uint32_t x = k;  // inclusive scan inside the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t t = lane < IT_T / 32 ? wsum[lane] : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            if (lane < IT_T / 32) wsum[lane] = t;  // inclusive warp totals
        }
        __syncthreads();
        const uint32_t off = base + (w ? wsum[w - 1] : 0u) + x - k;
        for (uint32_t t = 0; t < k; ++t)
            if (off + t < icap) items[off + t] = make_uint2(c, t * per);
        base += wsum[IT_T / 32 - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (ws) v.sc->n_ws_items = min(base, icap);
        else v.sc->n_ss_items = min(base, icap);
    }
}

// The candidate clusters of a water group, the union of the waters its
// members need, and per i-water lists of indices into that union, in one
// pass; one CTA (256 threads) per group.
// Candidates: clusters within the list radius of the group's box, ascending;
// the molecule lists are half lists (a pair belongs to its lower slot), so
// only clusters from the group's own first on can hold a partner.  Each
// candidate water is then tested against all 32 members, giving two 32-bit
// masks: members within r_ww (the outer lists wnb) and within r_in (the
// pruned lists winb).  A candidate with any member is in the union; the
// needed ones are numbered with a block-wide scan.  A warp
// compacts the lists of four members from the masks with one ballot per 32
// candidates, so every list ascends.  Everything is deterministic.
// Bound by the distance tests, 32 per candidate: 24,000 waters in 98 A, 73 us,
// against 32 + 115 + 34 us for a tile pass, a union pass that tested twice
// and read its candidates back from global memory, and a prune.
constexpr int UT = 256;
constexpr int TU = 4;  // clusters tested per thread and turn

DYN_KERNEL(__launch_bounds__(UT), k_group_union, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    const BoxDev b = *v.box;
    const float r2 = v.r_ww * v.r_ww, rin2 = v.r_in * v.r_in;
    const uint32_t nwc = v.sc->n_wclus;
    const uint32_t ng = (nwc + GRPW / WCL - 1) / (GRPW / WCL);
    const int tid = threadIdx.x, lane = tid & 31, wid_ = tid >> 5;
    constexpr int NWP = UT / 32, MPW = GRPW / NWP;  // warps, members per warp
    __shared__ float4 io[GRPW];
    __shared__ uint32_t wt[TU][NWP], wn[NWP];
    __shared__ uint32_t sh_out[UT], sh_in[UT];
    __shared__ uint16_t sh_loc[UT];
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t g = bk.idx; g < ng; g += bk.cnt) {
        const uint32_t s_first = g * GRPW;
        if (tid < GRPW) {
            const uint32_t s = s_first + tid;
            const float4 p = v.wpos[4 * s];  // nw_cap holds whole groups
            io[tid] = make_float4(p.x, p.y, p.z, v.wid[s] != INVALID_ID ? 1.f : 0.f);
            v.wprune[s] = p;
        }
        uint32_t* tl = v.tile_j + (size_t)g * v.cap_tile;
        const float4 c0 = v.gbb_c[g], h0 = v.gbb_h[g];
        uint32_t nt = 0;
        for (uint32_t jb = g * (GRPW / WCL); jb < nwc; jb += TU * UT) {
            uint32_t m[TU];
#pragma unroll
            for (int u = 0; u < TU; ++u) {
                const uint32_t cj = jb + u * UT + tid;
                m[u] = __ballot_sync(0xffffffffu, cj < nwc && bb_dist2(c0, h0, v.wbb_c[cj], v.wbb_h[cj], b) < r2);
                if (lane == 0) wt[u][wid_] = __popc(m[u]);
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < TU; ++u) {
                uint32_t before = nt, all = 0;
#pragma unroll
                for (int w = 0; w < NWP; ++w) {
                    if (w == wid_) before += all;
                    all += wt[u][w];
                }
                const uint32_t k = before + __popc(m[u] & lt);
                if (((m[u] >> lane) & 1u) && k < v.cap_tile) tl[k] = jb + u * UT + tid;
                nt += all;
            }
            __syncthreads();
        }
        __syncthreads();  // io (and the tile, where the loop above did not run)
        if (nt > v.cap_tile) {
            if (tid == 0) atomicMax(&v.sc->overflow, nt);
            nt = v.cap_tile;
        }
        const uint32_t vm = __ballot_sync(0xffffffffu, io[lane].w != 0.f);  // the members
        uint32_t n_out[MPW] = {}, n_in[MPW] = {};
        uint32_t base_cnt = 0;
        const uint32_t ncand = nt * WCL;
        for (uint32_t k0 = 0; k0 < ncand; k0 += UT) {
            const uint32_t k = k0 + tid;
            uint32_t slot = INVALID_ID, mo = 0u, mi = 0u;
            if (k < ncand) {
                slot = tl[k / WCL] * WCL + (k % WCL);
                if (v.wid[slot] != INVALID_ID) {
                    const float3 o = xyz(v.wpos[4 * slot]);
#pragma unroll
                    for (int i = 0; i < GRPW; ++i) {
                        const float3 d = min_image_fast(o - xyz(io[i]), b);
                        const float d2 = dot3(d, d);
                        mo |= d2 < r2 ? 1u << i : 0u;
                        mi |= d2 < rin2 ? 1u << i : 0u;
                    }
                    // members below the candidate's slot (half lists)
                    const uint32_t below = slot - s_first;
                    const uint32_t lm = vm & (below >= GRPW ? 0xffffffffu : (1u << below) - 1u);
                    mo &= lm;
                    mi &= lm;
                }
            }
            const bool need = mo != 0u;
            const uint32_t mn = __ballot_sync(0xffffffffu, need);
            sh_out[tid] = mo;
            sh_in[tid] = mi;
            if (lane == 0) wn[wid_] = __popc(mn);
            __syncthreads();
            uint32_t loc = base_cnt + __popc(mn & lt), tn = 0;
#pragma unroll
            for (int w = 0; w < NWP; ++w) {
                if (w < wid_) loc += wn[w];
                tn += wn[w];
            }
            const bool fits = need && loc < v.cap_union;
            sh_loc[tid] = fits ? (uint16_t)loc : (uint16_t)0xFFFFu;
            if (fits) v.grp_uslot[(size_t)g * v.cap_union + loc] = slot;
            __syncthreads();
            base_cnt += tn;
            // the lists: members wid_ * MPW + q, 32 candidates at a time
            for (int c = 0; c < UT; c += 32) {
                if (k0 + c >= ncand) break;
                const uint32_t xo = sh_out[c + lane] >> (wid_ * MPW), xi = sh_in[c + lane] >> (wid_ * MPW);
                const uint16_t l = sh_loc[c + lane];
#pragma unroll
                for (int q = 0; q < MPW; ++q) {
                    const size_t row = (size_t)(s_first + wid_ * MPW + q) * v.cap_nb;
                    const bool ho = ((xo >> q) & 1u) && l != 0xFFFFu, hi = ((xi >> q) & 1u) && l != 0xFFFFu;
                    const uint32_t bo = __ballot_sync(0xffffffffu, ho), bi = __ballot_sync(0xffffffffu, hi);
                    const uint32_t po = n_out[q] + __popc(bo & lt), pi = n_in[q] + __popc(bi & lt);
                    if (ho && po < v.cap_nb) v.wnb[row + po] = l;
                    if (hi && pi < v.cap_nb) v.winb[row + pi] = l;
                    n_out[q] += __popc(bo);
                    n_in[q] += __popc(bi);
                }
            }
            __syncthreads();  // the masks are refilled by the next chunk
        }
        if (tid == 0) {
            v.grp_nloc[g] = min(base_cnt, v.cap_union);
            if (base_cnt > v.cap_union) atomicMax(&v.sc->overflow, base_cnt);
            atomicMax(&v.sc->union_max, base_cnt);
        }
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < MPW; ++q) {
                const uint32_t s = s_first + wid_ * MPW + q;
                v.wnb_n[s] = min(n_out[q], v.cap_nb);
                v.winb_n[s] = min(n_in[q], v.cap_nb);
                if (n_out[q] > v.cap_nb) atomicMax(&v.sc->overflow, n_out[q]);
            }
        }
        if (v.ww_split > 1u) {
            // where the parts of the union start in each pruned list
            const uint32_t nloc = min(base_cnt, v.cap_union);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < MPW; ++q) {
                const uint32_t s = s_first + wid_ * MPW + q;
                if ((uint32_t)lane < v.ww_split) {
                    const uint16_t* lst = v.winb + (size_t)s * v.cap_nb;
                    const uint32_t c = ww_cut(nloc, lane, v.ww_split);
                    uint32_t l0 = 0, l1 = min(n_in[q], v.cap_nb);
                    while (l0 < l1) {
                        const uint32_t m = (l0 + l1) >> 1;
                        if ((uint32_t)lst[m] < c) l0 = m + 1; else l1 = m;
                    }
                    v.winb_cut[(size_t)WW_SPLIT_MAX * s + lane] = (uint16_t)l0;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Pruning of the water-water lists (a dual pair list: Pall, Zhmurov,
// Bauer, Abraham, Lundborg, Gray, Hess, Lindahl, J. Chem. Phys. 153, 134110
// (2020)).  The rebuild's lists hold the molecule pairs with an O-O distance
// below r_ww = cutoff + 2 reach + buffer; the kernel walks these pruned to
// r_in = cutoff + 2 reach + prune buffer, which stay complete until some
// water has moved half the prune buffer since the prune.  The rebuild writes
// both; this kernel prunes again in between.  One CTA per group: the union's
// O positions are staged in shared memory (PR_CHUNK at a time) and a warp per
// water tests 32 of its entries at a time in order, the next 32 loading
// meanwhile, and compacts the hits with ballots (the pruned lists stay
// ascending).  Bound by the latency of the list reads: with 8 lanes per
// water a list of 100 was a chain of 13 loads, 33 us for 16 groups and 34 for
// 750; a warp per water takes 12 and 22.  The group's O positions are recorded
// for the next check.
// ---------------------------------------------------------------------------
constexpr int PRT = 256;
constexpr uint32_t PR_CHUNK = 1024;

DYN_KERNEL(__launch_bounds__(PRT), k_ww_prune, (, bool force), (, force)) {
    if (!(force || v.sc->need_prune)) return;
    __shared__ float4 uo[PR_CHUNK];
    const BoxDev b = *v.box;
    const float r2 = v.r_in * v.r_in;
    const uint32_t ng = (v.sc->n_wclus + GRPW / WCL - 1) / (GRPW / WCL);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    constexpr int MPW = GRPW / (PRT / 32);  // waters per warp
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t g = bk.idx; g < ng; g += bk.cnt) {
        const uint32_t nloc = v.grp_nloc[g];
        const uint32_t s0 = g * GRPW + wp * MPW;
        uint32_t n[MPW], k0[MPW] = {}, cnt[MPW] = {}, nx[MPW];
        // lane p counts the entries below the start of the union's part p
        const uint32_t my_cut = (uint32_t)lane < v.ww_split ? ww_cut(nloc, lane, v.ww_split) : 0u;
        uint32_t below[MPW] = {};
        float3 io[MPW];
#pragma unroll
        for (int q = 0; q < MPW; ++q) {
            const uint32_t s = s0 + q;
            n[q] = v.wid[s] != INVALID_ID ? v.wnb_n[s] : 0u;
            io[q] = xyz(v.wpos[4 * s]);
            nx[q] = (uint32_t)lane < n[q] ? (uint32_t)v.wnb[(size_t)s * v.cap_nb + lane] : 0xFFFFFFFFu;
        }
        for (uint32_t lo = 0; lo < nloc; lo += PR_CHUNK) {
            const uint32_t hi = min(nloc, lo + PR_CHUNK);
            for (uint32_t t = tid; t < hi - lo; t += PRT)
                uo[t] = v.wpos[4 * (size_t)v.grp_uslot[(size_t)g * v.cap_union + lo + t]];
            __syncthreads();
#pragma unroll
            for (int q = 0; q < MPW; ++q) {
                const uint16_t* in = v.wnb + (size_t)(s0 + q) * v.cap_nb;
                uint16_t* out = v.winb + (size_t)(s0 + q) * v.cap_nb;
                // this water's entries in [lo, hi): a prefix of what is left
                for (;;) {
                    const uint32_t idx = nx[q];
                    const bool here = idx < hi;
                    const uint32_t adv = __popc(__ballot_sync(0xffffffffu, here));
                    if (adv == 32u) {
                        const uint32_t k = k0[q] + 32u + lane;
                        nx[q] = k < n[q] ? (uint32_t)in[k] : 0xFFFFFFFFu;
                    }
                    bool hit = false;
                    if (here) {
                        const float3 d = min_image_fast(io[q] - xyz(uo[idx - lo]), b);
                        hit = dot3(d, d) < r2;
                    }
                    const uint32_t mh = __ballot_sync(0xffffffffu, hit);
                    if (hit) out[cnt[q] + __popc(mh & lt)] = (uint16_t)idx;
                    cnt[q] += __popc(mh);
                    for (uint32_t p = 1; p < v.ww_split; ++p) {
                        const uint32_t cut = __shfl_sync(0xffffffffu, my_cut, p);
                        const bool lower = hit & (idx < cut);
                        const uint32_t c = __popc(__ballot_sync(0xffffffffu, lower));
                        if ((uint32_t)lane == p) below[q] += c;
                    }
                    k0[q] += adv;
                    if (adv < 32u) {
                        // the rest of these 32 belongs to the next chunk
                        if (adv && hi < nloc) {
                            const uint32_t k = k0[q] + lane;
                            nx[q] = k < n[q] ? (uint32_t)in[k] : 0xFFFFFFFFu;
                        }
                        break;
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < MPW; ++q)
            if (lane == 0) v.winb_n[s0 + q] = cnt[q];
#pragma unroll
        for (int q = 0; q < MPW; ++q)
            if (v.ww_split > 1u && (uint32_t)lane < v.ww_split)
                v.winb_cut[(size_t)WW_SPLIT_MAX * (s0 + q) + lane] = (uint16_t)below[q];
        if (tid < GRPW) v.wprune[g * GRPW + tid] = v.wpos[4 * (g * GRPW + tid)];
    }
}

DYN_KERNEL(, k_prune_done, (, bool force), (, force)) {
    if (!(force || v.sc->need_prune)) return;
    v.sc->need_prune = 0u;
    v.sc->prunes += 1ull;
}

DYN_KERNEL(, k_rebuild_done, (, bool force), (, force)) {
    if (!rebuild_on(v, force)) return;
    v.sc->need_rebuild = 0u;
    v.sc->rebuilds += 1ull;
    // the rebuild wrote the pruned lists too
    v.sc->need_prune = 0u;
    v.sc->prunes += 1ull;
}

// Copies positions into cluster order and zeroes the atoms' and the
// waters' short-range force accumulators (every pair kernel adds to them),
// for an evaluation without a step; a step's first half does both.
DYN_KERNEL(, k_gather_atoms, (), ()) {
    const uint32_t t0 = bk.idx * blockDim.x + threadIdx.x, stride = bk.cnt * blockDim.x;
    for (uint32_t s = t0; s < v.na_cap; s += stride) {
        const uint32_t a = v.sidx[s];
        if (a != INVALID_ID) {
            v.spos[s] = v.apos[a];
            v.aforce[3 * (size_t)a + 0] = 0; v.aforce[3 * (size_t)a + 1] = 0; v.aforce[3 * (size_t)a + 2] = 0;
        }
    }
    int4* wf = reinterpret_cast<int4*>(v.wforce);  // 12 int64 = 6 int4 per slot
    for (uint32_t t = t0; t < 6 * v.nw_cap; t += stride) wf[t] = make_int4(0, 0, 0, 0);
}

inline int nblocks(uint64_t n, int threads, int cap = 148 * 8) {
    uint64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    return (int)(b < (uint64_t)cap ? b : cap);
}

}  // namespace

namespace dyn {

void launch_displacement_check(const Target& t) {
    t.launch(k_disp_check, k_disp_check_batch, [](const SysView& v) { return nblocks(v.nw_cap + v.na, 256); },
             256, 0);
}

void launch_rebuild(const Target& t, bool force) {
    const int T = 256;
    auto nmax = [](const SysView& v) { return v.nw_cap > v.na_cap ? v.nw_cap : v.na_cap; };
    t.launch(k_col_clear, k_col_clear_batch,
             [](const SysView& v) { return nblocks(std::max(std::max(v.ncol, v.ancol), v.na_cap), 256); }, T, 0, force);
    t.launch(k_col_assign, k_col_assign_batch, [&](const SysView& v) { return nblocks(nmax(v), 256); }, T, 0, force);
    t.launch(k_col_scan, k_col_scan_batch, [](const SysView&) { return 1; }, SCT, 0, force);
    t.launch(k_col_bucket, k_col_bucket_batch, [&](const SysView& v) { return nblocks(nmax(v), 256); }, T, 0, force);
    t.launch(k_col_rank, k_col_rank_batch,
             [](const SysView& v) { return nblocks(std::max<uint64_t>((uint64_t)(v.nw ? v.ncol : 1u) * RKT, v.na), RKT); },
             RKT, 0, force);
    t.launch(k_perm_copyback, k_perm_copyback_batch, [&](const SysView& v) { return nblocks(nmax(v), 256); }, T, 0,
             force);
    const int LT = 128;  // 4 warps per block, one i-cluster per warp
    t.launch(k_group_union, k_group_union_batch,
             [](const SysView& v) { return v.nw ? (int)std::min<uint32_t>(v.ngrp_cap, 148 * 8) : 0; }, UT, 0, force);
    t.launch(k_list_ws, k_list_ws_batch,
             [](const SysView& v) { return v.nw && v.na ? (int)std::min<uint32_t>(v.naclus_cap, 148 * 8) : 0; }, WLT, 0,
             force);
    t.launch(k_list_ss, k_list_ss_batch,
             [](const SysView& v) { return v.na ? nblocks((uint64_t)v.naclus_cap * 32, 128, 1 << 30) : 0; }, LT, 0,
             force);
    t.launch(k_items, k_items_batch, [](const SysView& v) { return v.na ? 2 : 0; }, IT_T, 0, force);
    t.launch(k_rebuild_done, k_rebuild_done_batch, [](const SysView&) { return 1; }, 1, 0, force);
}

void launch_prune(const Target& t, bool force) {
    t.launch(k_ww_prune, k_ww_prune_batch,
             [](const SysView& v) { return v.nw ? (int)std::min<uint32_t>(v.ngrp_cap, 148 * 8) : 0; }, PRT, 0, force);
    t.launch(k_prune_done, k_prune_done_batch, [](const SysView&) { return 1; }, 1, 0, force);
}

void launch_gather_atoms(const Target& t) {
    t.launch(k_gather_atoms, k_gather_atoms_batch,
             [](const SysView& v) { return nblocks(std::max<uint64_t>(v.na_cap, 6ull * v.nw_cap), 256); }, 256, 0);
}

}  // namespace dyn
