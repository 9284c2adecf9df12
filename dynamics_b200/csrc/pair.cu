// Short-range LJ + erfc-screened Coulomb over cluster pairs.
//
// Replaces the reference's one-thread-per-pair kernel over a flat list
// (src/cuda/cuda.cu:185-362) and its CPU twin (src/non_bonded.rs:258-412,
// 950-1057).  The physics is the reference CPU path's: LJ for r <= lj_cutoff
// between sites that carry LJ, erfc(alpha r)/r Coulomb for r < cutoff
// between charged sites, 1-2/1-3 exclusions, no intra-water pairs; 1-4 pairs
// are excluded here and evaluated (scaled) by k_pair14.
//
// Work decomposition.  Water-water: one CTA per 32-water i-group (or part of
// one), j sites staged in shared memory, the group's molecule lists dealt out
// over the threads (k_pair_ww_tile).  Water-atom: one warp per atom cluster
// and batch of the waters listed for it, a lane per water (k_pair_ws).
// Atom-atom: one warp per work item (an 8-atom i-cluster and up to ch_mix
// entries of its list); lane = (ii, jq) with ii = lane & 7 and jq = lane >> 3
// evaluates i-atom ii against j-atoms jq and jq + 4 of every j-cluster in the
// item (k_pair_ss).  All lists hold every pair once.  A water is moved as a
// whole: one min-image shift from its O serves all its sites, valid because
// the cutoff plus twice the O-H reach is below half the box.  Forces are
// summed in float32 registers as far as a thread's work goes and added to the
// int64 fixed-point accumulators with reductions; integer sums do not depend
// on order, so the result is deterministic.
#include <algorithm>
#include <cstring>
#include <vector>

#include "engine.cuh"

namespace {

constexpr int PT = 128;  // threads per block (4 warps)

// e_lj, e_c accumulate per-pair energies in float64 (energy steps only);
// w sums the virial of one list entry (a molecule pair, or an i-body
// against a j-cluster's atoms) in float32, and wd the entries' sums in
// float64, so no long float32 chain feeds the pressure
struct Acc3 {
    double e_lj, e_c;
    float w;
    double wd;
    __device__ __forceinline__ void flush_w() { wd += (double)w; w = 0.f; }
};

// erfc-screened Coulomb between site pi and site pj shifted by sh
// (d = pi - (pj - sh)), branch-free: force q q (r^-3 + g(r^2)) d with
// g(z) = 2 d/dz [erf(alpha sqrt z) / sqrt z] from the host-fitted polynomial
// in t = 2 r^2 / rc^2 - 1 (no square root needed for the argument); zero for
// r >= rc (src/cuda/cuda.cu:160-164).  On energy steps the energy
// qqe erfc(alpha r) / r is added in float64.
template <bool ENERGY>
__device__ __forceinline__ void coul(float3 pi, float3 pj, float3 sh, float qq, double qqe, const PairParams& P,
                                     float3& f, Acc3& a) {
    const float3 d = pi - (pj - sh);
    const float r2 = dot3(d, d);
    const float rinv = rsqrtf(r2);
    const float t = fmaf(r2, P.two_over_rc2, -1.0f);
    float g = P.poly_g[NPOLY_G - 1];
#pragma unroll
    for (int k = NPOLY_G - 2; k >= 0; --k) g = fmaf(g, t, P.poly_g[k]);
    float fs = qq * fmaf(rinv * rinv, rinv, g);
    fs = r2 < P.rc2 ? fs : 0.0f;
    f.x = fmaf(fs, d.x, f.x); f.y = fmaf(fs, d.y, f.y); f.z = fmaf(fs, d.z, f.z);
    a.w = fmaf(fs, r2, a.w);
    if (ENERGY && r2 < P.rc2) {
        // erfc(alpha r) / r in float32 from the force's r^2 and 1/r, scaled by
        // the float64 charge product and summed in float64: per-pair errors
        // of a few ulp with no common sign
        const float re = r2 * rinv;
        a.e_c += qqe * (double)(erfcf(P.alpha * re) * rinv);
    }
}

// 12-6 LJ (force_e_lj, src/forces.rs:10-21) between pi and pj shifted by sh,
// branch-free, r <= lj_cutoff; energy summed in float64.
template <bool ENERGY>
__device__ __forceinline__ void lj(float3 pi, float3 pj, float3 sh, float sig2, float eps, float ljc2,
                                   float scale, float3& f, Acc3& a) {
    const float3 d = pi - (pj - sh);
    const float r2 = dot3(d, d);
    const bool in = r2 <= ljc2;
    const float ir2 = __frcp_rn(in ? r2 : 1.0f);
    const float sr2 = sig2 * ir2;
    const float sr6 = sr2 * sr2 * sr2;
    float fs = scale * 24.0f * eps * fmaf(2.f, sr6 * sr6, -sr6) * ir2;
    fs = in ? fs : 0.0f;
    f.x = fmaf(fs, d.x, f.x); f.y = fmaf(fs, d.y, f.y); f.z = fmaf(fs, d.z, f.z);
    a.w = fmaf(fs, r2, a.w);
    if (ENERGY && in) {
        const double s6 = (double)sr6;
        a.e_lj += 4.0 * (double)scale * (double)eps * (s6 * s6 - s6);
    }
}

// Soft-core LJ of a pair between the alchemical molecule and the rest
// (Beutler et al., Chem. Phys. Lett. 222, 529 (1994), as
// alchemical_lj_soft_core_decouple, src/non_bonded.rs:883-941, with the
// reference's sc-alpha 0.5, power 1 and soft-core sigma >= 3 A,
// src/alchemical.rs:55-65): V = (1 - l) V_LJ(r_sc) with
// r_sc^6 = r^6 + 0.5 s^6 l, s = max(sigma, 3); force (1 - l) F_LJ(r_sc)
// (r / r_sc)^5; dV/dl = -V_LJ(r_sc) - (1 - l) F_LJ(r_sc) 0.5 s^6 / (6 r_sc^5),
// times dl/dlambda of the schedule (dlam) into dh.
template <bool ENERGY>
__device__ __forceinline__ void lj_soft(float3 pi, float3 pj, float3 sh, float sig, float eps, float ljc2,
                                        float lam, float dlam, float3& f, Acc3& a, double& dh) {
    const float3 d = pi - (pj - sh);
    const float r2 = dot3(d, d);
    if (!(r2 <= ljc2) || !(r2 > 0.f) || eps == 0.f) return;
    const float ss = fmaxf(sig, 3.0f), ss2 = ss * ss;
    const float ss6 = ss2 * ss2 * ss2;
    const float rsc6 = fmaf(0.5f * ss6, lam, r2 * r2 * r2);
    const float rsc = sqrtf(cbrtf(rsc6));
    const float inv_rsc = 1.0f / rsc;
    const float sr = sig * inv_rsc, sr2 = sr * sr;
    const float sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
    const float hf = 24.0f * eps * fmaf(2.0f, sr12, -sr6) * inv_rsc;
    const float he = 4.0f * eps * (sr12 - sr6);
    const float scale = 1.0f - lam;
    const float r = sqrtf(r2);
    const float q = r * inv_rsc, q2 = q * q;
    const float fs = hf * scale * (q2 * q2 * q) / r;
    f.x = fmaf(fs, d.x, f.x); f.y = fmaf(fs, d.y, f.y); f.z = fmaf(fs, d.z, f.z);
    a.w = fmaf(fs, r2, a.w);
    if (ENERGY) {
        const double rsc5 = (double)rsc6 / (double)rsc;
        a.e_lj += (double)scale * (double)he;
        dh += (double)dlam * (-(double)he - (double)scale * (double)hf * (0.5 * (double)ss6) / (6.0 * rsc5));
    }
}

__device__ __forceinline__ float3 shift_of(float3 d, const BoxDev& b) {
    return f3(-rintf(d.x * b.inv_ext[0]) * b.ext[0], -rintf(d.y * b.inv_ext[1]) * b.ext[1],
              -rintf(d.z * b.inv_ext[2]) * b.ext[2]);
}

__device__ __forceinline__ float red4(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 8);
    x += __shfl_xor_sync(0xffffffffu, x, 16);
    return x;
}

__device__ __forceinline__ void add_fix3(long long* p, float3 f) {
    fix_atomic_add(p + 0, fix_from_float(f.x));
    fix_atomic_add(p + 1, fix_from_float(f.y));
    fix_atomic_add(p + 2, fix_from_float(f.z));
}

template <bool ENERGY>
__device__ __forceinline__ void write_partials(const SysView& v, Blk bk, int region, double el,
                                               double ec, double w, double dh = 0.0) {
    double x[4] = {el, ec, w, dh};
    block_sum_d<4>(x);
    if (threadIdx.x == 0) {
        double* p = v.partials + ((size_t)region * v.max_blocks + bk.idx) * 4;
        p[0] = x[0]; p[1] = x[1]; p[2] = x[2]; p[3] = x[3];
    }
}

// ---------------------------------------------------------------------------
// Staging for the water-water kernel (k_pair_ww_tile, below): the sites of a
// range of a group's union, 64 bytes per water, into shared memory with
// asynchronous 16-byte copies.  Site k of union water u sits at 4 u + (k ^
// swizzle(u)): lanes that read the same site of scattered waters then spread
// over all eight 16-byte bank groups (unswizzled, a site falls into two of
// them, and the four loads per molecule pair were 9-way conflicts on
// average; bulk copies cannot write this order).
// ---------------------------------------------------------------------------
constexpr int WT = 256;  // threads per CTA
constexpr int JS = 13;   // words per union water of the j sums

__device__ __forceinline__ uint32_t tile_swizzle(uint32_t u) { return (u >> 1) & 3u; }

template <int T>
__device__ __forceinline__ void stage_chunk(const SysView& v, uint32_t g, uint32_t lo, uint32_t n, float4* tile,
                                            uint32_t* uslot, int tid) {
    const uint32_t* slots = v.grp_uslot + (size_t)g * v.cap_union + lo;
    for (uint32_t t = tid; t < 4 * n; t += T) {
        const uint32_t u = t >> 2, k = t & 3u;
        const uint32_t s = slots[u];
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(tile + 4 * u + (k ^ tile_swizzle(u))));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(v.wpos + 4 * (size_t)s + k) : "memory");
        if (k == 0) uslot[u] = s;
    }
}

// 1 / sqrt(x), the instruction behind rsqrtf; squared distances are never
// subnormal, so the flushing form needs no scaling around it
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void axpy3(float3& acc, float s, float3 d) {
    acc.x = fmaf(s, d.x, acc.x); acc.y = fmaf(s, d.y, acc.y); acc.z = fmaf(s, d.z, acc.z);
}

// Screened Coulomb of one site pair of a molecule pair (coul above; nj is the
// negated j position, moved to the image nearest the i-water): the pair
// force fs d is added to the i-site sum fi and to gj (the j site receives
// -gj).
template <bool ENERGY>
__device__ __forceinline__ void coul2(float3 pi, float3 nj, float qq, double qqe, const PairParams& P, float3& fi,
                                      float3& gj, Acc3& a) {
    const float3 d = pi + nj;
    const float r2 = dot3(d, d);
    const float rinv = rsqrt_ftz(r2);
    const float t = fmaf(r2, P.two_over_rc2, -1.0f);
    float g = P.poly_g[NPOLY_G - 1];
#pragma unroll
    for (int k = NPOLY_G - 2; k >= 0; --k) g = fmaf(g, t, P.poly_g[k]);
    float fs = qq * fmaf(rinv * rinv, rinv, g);
    fs = r2 < P.rc2 ? fs : 0.0f;
    axpy3(fi, fs, d);
    axpy3(gj, fs, d);
    a.w = fmaf(fs, r2, a.w);
    if (ENERGY && r2 < P.rc2) a.e_c += qqe * (double)(erfcf(P.alpha * (r2 * rinv)) * rinv);
}

// j-side forces of a union water are added to the CTA's int32 sums.  A
// component too large for them (|f| >= JFIX_MAX: 32 such contributions stay
// below 2^15 kcal/mol/A, the int32 range at 2^-16) takes its whole site out
// of the sums (sites with one are flagged), and the molecule pair is
// evaluated again by jforce_big, which adds the flagged sites' forces to the
// slot's int64 sums.  Which way a site goes depends only on its values, and
// both are integer sums, so the result stays deterministic.
constexpr float JFIX_SCALE = (float)(1 << WW_JFIX_SHIFT);
constexpr float JFIX_MAX = 1000.0f;

// The force -g on one site into its three sums; true if it did not fit.
__device__ __forceinline__ bool jforce_add3(int* p, float3 g) {
    const bool big = fmaxf(fmaxf(fabsf(g.x), fabsf(g.y)), fabsf(g.z)) >= JFIX_MAX;
    const float sc = big ? 0.0f : -JFIX_SCALE;
    atomicAdd(p + 0, __float2int_rn(g.x * sc));
    atomicAdd(p + 1, __float2int_rn(g.y * sc));
    atomicAdd(p + 2, __float2int_rn(g.z * sc));
    return big;
}

// The flagged sites (bit k: site k) of the j water in slot, whose negated
// sites nj are at the image nearest the i-water pi.
__device__ __noinline__ void jforce_big(const SysView& v, uint32_t slot, uint32_t sites, const float4* pi,
                                        const float4* pj, uint32_t sw, float3 n) {
    const BoxDev b = *v.box;
    const float q[3] = {OPC_Q_H, OPC_Q_H, OPC_Q_EP};
    for (int k = 0; k < 4; ++k) {
        if (!((sites >> k) & 1u)) continue;
        const float4 p0 = pj[k ^ sw];
        const float3 j = f3(-fmaf(n.x, b.ext[0], -p0.x), -fmaf(n.y, b.ext[1], -p0.y), -fmaf(n.z, b.ext[2], -p0.z));
        float3 f = f3(0.f, 0.f, 0.f);
        Acc3 a{0.0, 0.0, 0.f, 0.0};
        if (k == 0) lj<false>(xyz(pi[0]), j, f3(0.f, 0.f, 0.f), OPC_O_SIGMA * OPC_O_SIGMA, OPC_O_EPS, v.pp.ljc2, 1.0f, f, a);
        for (int i = 1; i < 4 && k; ++i)
            coul<false>(xyz(pi[i]), j, f3(0.f, 0.f, 0.f), q[i - 1] * q[k - 1], 0.0, v.pp, f, a);
        long long* p = v.wforce + (size_t)slot * 12 + 3 * k;
        fix_atomic_add(p + 0, fix_from_float(-f.x));
        fix_atomic_add(p + 1, fix_from_float(-f.y));
        fix_atomic_add(p + 2, fix_from_float(-f.z));
    }
}

// Per-warp partials (the atom pair kernels' warps run independent work
// items: no block barrier at the end); fixed shuffle order, so the sums are
// deterministic.  The region holds blocks x PT/32 entries.
template <bool ENERGY>
__device__ __forceinline__ void write_partials_warp(const SysView& v, Blk bk, int region, double el, double ec,
                                                    double w, double dh) {
    el = warp_sum_d(el); ec = warp_sum_d(ec); w = warp_sum_d(w); dh = warp_sum_d(dh);
    if ((threadIdx.x & 31) == 0) {
        const size_t e = (size_t)bk.idx * (blockDim.x >> 5) + (threadIdx.x >> 5);
        double* p = v.partials + ((size_t)region * v.max_blocks + e) * 4;
        p[0] = el; p[1] = ec; p[2] = w; p[3] = dh;
    }
}

// ---------------------------------------------------------------------------
// water(i) - water(j), tile form, half lists.  A unit of work is a 32-water
// i-group and one of ww_split equal ranges of its union (the waters its
// lists reach); a CTA per unit copies the range's sites to shared memory, at
// most union_chunk waters at a time (one chunk for most
// units).  The lists hold every water pair once (in the list of the lower
// slot), so their lengths vary several-fold across a group; the chunk's
// entries of all 32 lists are therefore dealt out as one sequence, an equal
// contiguous share per thread, whatever list they come from.  A thread keeps
// the i-water's forces in registers while its share stays in one list and
// adds them to the water forces (int64 reductions) when it moves to the
// next.  All 10 site pairs of a molecule pair use one min-image shift.  The
// j sites are taken one after another, so that only one site's j force is
// held at a time: it goes to int32 fixed-point sums in shared memory (12
// components, 13 words apart per water, so that the threads' adds spread over
// the banks and take fixed offsets), which are added to the union waters'
// forces with one coalesced run of int64 reductions per chunk.  The shares
// depend only on the lists, the split and the chunk size, and every sum
// across threads is an integer sum: the forces are the same bits run to run.
//
// 24,000 waters in 98 A: 2.2 M list entries.  What it waits for is the
// latency of the shared-memory gathers, the barriers around each unit and the
// last wave of units (3 CTAs per SM; the batch form, which holds the view's
// pointers in registers, spills there and runs 2: 64 systems 1244 us a step
// against 1312).  84 -> 71 us (80,000 waters 217 -> 185, 8,000 waters 57 ->
// 39, 512 waters 22 -> 17) by the swizzled tile (the gathers were 9-way bank
// conflicts, 63 % of the shared-memory wavefronts), j sums at fixed offsets,
// one check for large forces per molecule pair instead of a branch per site,
// image shifts by fused multiply-adds, and parts that stage, zero and flush
// their own range of the union only (a part used to handle all of it).  Two
// entries at a time in packed float32 registers ran 38 M instead of 46 M
// instructions but no faster: a third of its instructions duplicated
// coefficients into register pairs, at 2 CTAs per SM.
// ---------------------------------------------------------------------------
DYN_KERNEL_T2((bool ENERGY), (ENERGY), __launch_bounds__(WT, 3), __launch_bounds__(WT, 2), k_pair_ww_tile, (, const PairParams P), (, P)) {
    extern __shared__ __align__(128) float4 tile[];  // union_chunk waters x 4 float4, then the j sums
    __shared__ float4 ipos[GRPW * 4];   // the group's i-water sites
    __shared__ uint32_t woff[GRPW + 1]; // first share position of each list's chunk entries
    __shared__ uint32_t wbeg[GRPW];     // each list's first entry in the chunk
    __shared__ uint32_t wend[GRPW];     // ... and one past its last
    const int tid = threadIdx.x;
    const uint32_t nwc = v.sc->n_wclus;
    const uint32_t ng = (nwc + GRPW / WCL - 1) / (GRPW / WCL);
    const uint32_t chunk = v.union_chunk;
    int* jacc = reinterpret_cast<int*>(tile + 4 * (size_t)chunk);            // [chunk][JS], 12 used
    uint32_t* uslot = reinterpret_cast<uint32_t*>(jacc + JS * (size_t)chunk);  // [chunk] union entry -> slot
    const BoxDev b = *v.box;
    constexpr float qhh = OPC_Q_H * OPC_Q_H, qhm = OPC_Q_H * OPC_Q_EP, qmm = OPC_Q_EP * OPC_Q_EP;
    const double ehh = (double)OPC_Q_H * (double)OPC_Q_H, ehm = (double)OPC_Q_H * (double)OPC_Q_EP,
                 emm = (double)OPC_Q_EP * (double)OPC_Q_EP;
    Acc3 a{0.0, 0.0, 0.f, 0.0};
    const uint32_t split = v.ww_split;
    for (uint32_t q = bk.idx; q < ng * split; q += bk.cnt) {
        const uint32_t g = q / split, part = q - g * split;
        const uint32_t nloc = v.grp_nloc[g];
        const uint32_t plo = ww_cut(nloc, part, split), phi = ww_cut(nloc, part + 1, split);
        if (tid < GRPW * 4) ipos[tid] = v.wpos[(size_t)4 * g * GRPW + tid];  // nw_cap holds whole groups
        uint32_t wlen = 0;
        if (tid >= 32 && tid < 32 + GRPW) {
            // this part's entries of list w: [wend, wlen)
            const int w = tid - 32;
            const uint32_t s = g * GRPW + w;
            wlen = v.winb_n[s];
            uint32_t b0 = 0;
            if (split > 1) {
                const uint16_t* cut = v.winb_cut + (size_t)WW_SPLIT_MAX * s;
                if (part) b0 = cut[part];
                if (part + 1 < split) wlen = cut[part + 1];
            }
            wend[w] = b0;
        }
        for (uint32_t lo = plo; lo < phi; lo += chunk) {
            const uint32_t hi = min(phi, lo + chunk), nu = hi - lo;
            stage_chunk<WT>(v, g, lo, nu, tile, uslot, tid);
            if (tid >= 32 && tid < 32 + GRPW) {
                // the list entries of this chunk: from where the previous
                // chunk stopped to the first union index >= hi (lists ascend)
                const int w = tid - 32;
                const uint32_t b0 = wend[w];
                uint32_t l0 = b0, l1 = wlen;
                if (hi == phi) l0 = l1;
                const uint16_t* lst = v.winb + (size_t)(g * GRPW + w) * v.cap_nb;
                while (l0 < l1) {
                    const uint32_t m = (l0 + l1) >> 1;
                    if ((uint32_t)lst[m] < hi) l0 = m + 1; else l1 = m;
                }
                uint32_t x = l0 - b0;  // inclusive scan over the lists
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (w >= o) x += y;
                }
                wbeg[w] = b0;
                woff[w + 1] = x;
                if (w == 0) woff[0] = 0u;
                wend[w] = l0;
            }
            for (uint32_t t = tid; t < JS * nu; t += WT) jacc[t] = 0;  // the j sums start at zero
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // this thread's share of the entries
            const uint32_t total = woff[GRPW];
            const uint32_t e0 = (uint32_t)(((uint64_t)tid * total) / WT);
            const uint32_t e1 = (uint32_t)(((uint64_t)(tid + 1) * total) / WT);
            int w = 0;
            while (w < GRPW - 1 && woff[w + 1] <= e0) ++w;
            float3 iO = f3(0, 0, 0), iH0 = iO, iH1 = iO, iM = iO;
            float3 fO = iO, fH0 = iO, fH1 = iO, fM = iO;
            const uint16_t* lst = v.winb;
            uint32_t wstop = 0;  // share position where list w ends
            auto enter = [&](int wn) {
                w = wn;
                iO = xyz(ipos[4 * w + 0]); iH0 = xyz(ipos[4 * w + 1]);
                iH1 = xyz(ipos[4 * w + 2]); iM = xyz(ipos[4 * w + 3]);
                // lst[e] is the entry at list position wbeg[w] + (e - woff[w])
                lst = v.winb + ((size_t)(g * GRPW + w) * v.cap_nb + wbeg[w]) - woff[w];
                wstop = woff[w + 1];
            };
            auto leave = [&]() {
                long long* p = v.wforce + (size_t)(g * GRPW + w) * 12;
                add_fix3(p + 0, fO); add_fix3(p + 3, fH0); add_fix3(p + 6, fH1); add_fix3(p + 9, fM);
                fO = f3(0, 0, 0); fH0 = fO; fH1 = fO; fM = fO;
            };
            if (e0 < e1) enter(w);
            // the next entry's index is loaded one iteration ahead, so the
            // global-memory latency of the list overlaps the arithmetic
            uint32_t idx_next = e0 < e1 ? (uint32_t)lst[e0] : 0u;
            for (uint32_t e = e0; e < e1; ++e) {
                if (e >= wstop) {
                    leave();
                    int wn = w + 1;
                    while (woff[wn + 1] <= e) ++wn;
                    enter(wn);
                    idx_next = (uint32_t)lst[e];
                }
                const uint32_t u = idx_next - lo;
                if (e + 1 < e1 && e + 1 < wstop) idx_next = (uint32_t)lst[e + 1];
                const float4* jw = tile + 4 * u;
                const uint32_t sw = tile_swizzle(u);
                int* jf = jacc + JS * u;
                // negated j sites at the image nearest the i-water
                const float3 jO = xyz(jw[sw]);
                const float3 n = f3(-nearest_int(iO.x - jO.x, b.inv_ext[0]), -nearest_int(iO.y - jO.y, b.inv_ext[1]),
                                    -nearest_int(iO.z - jO.z, b.inv_ext[2]));
                auto image = [&](float3 p) {
                    return f3(fmaf(n.x, b.ext[0], -p.x), fmaf(n.y, b.ext[1], -p.y), fmaf(n.z, b.ext[2], -p.z));
                };
                uint32_t big = 0;  // sites whose force does not fit the int32 sums
                {
                    const float3 nj = image(jO);
                    float3 t = f3(0.f, 0.f, 0.f);
                    lj<ENERGY>(iO, f3(-nj.x, -nj.y, -nj.z), f3(0.f, 0.f, 0.f), OPC_O_SIGMA * OPC_O_SIGMA, OPC_O_EPS,
                               P.ljc2, 1.0f, t, a);
                    fO = fO + t;
                    if (jforce_add3(jf, t)) big |= 1u;
                }
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    const float3 nj = image(xyz(jw[k ^ sw]));
                    float3 gj = f3(0.f, 0.f, 0.f);
                    coul2<ENERGY>(iH0, nj, k == 3 ? qhm : qhh, k == 3 ? ehm : ehh, P, fH0, gj, a);
                    coul2<ENERGY>(iH1, nj, k == 3 ? qhm : qhh, k == 3 ? ehm : ehh, P, fH1, gj, a);
                    coul2<ENERGY>(iM, nj, k == 3 ? qmm : qhm, k == 3 ? emm : ehm, P, fM, gj, a);
                    if (jforce_add3(jf + 3 * k, gj)) big |= 1u << k;
                }
                if (big) jforce_big(v, uslot[u], big, ipos + 4 * w, jw, sw, n);
                a.flush_w();
            }
            if (e0 < e1) leave();
            __syncthreads();  // every j sum of the chunk is in
            // the chunk's sums -> the union waters' forces (2^-16 -> 2^-32
            // fixed point); consecutive union entries of a run are
            // consecutive slots, so the reductions are coalesced
            for (uint32_t t = tid; t < 12 * nu; t += WT) {
                const uint32_t u = t / 12, c = t - 12 * u;
                const int val = jacc[JS * u + c];
                if (val != 0)
                    fix_atomic_add(v.wforce + 12 * (size_t)uslot[u] + c,
                                   (long long)val * (1ll << (32 - WW_JFIX_SHIFT)));
            }
            __syncthreads();  // the tile and the sums are refilled by the next chunk or unit
        }
        __syncthreads();  // the i-water sites are refilled by the next unit
    }
    write_partials<ENERGY>(v, bk, REG_WW, ENERGY ? a.e_lj : 0.0, ENERGY ? a.e_c : 0.0, a.wd);
}


// Reduce-scatter over the 8 lanes that share jq (lane bits 0-2): N values
// per lane in, N/8 out; lane ii ends with the sums of values
// [ii N/8, (ii + 1) N/8).  The pairing order is fixed, so the result is
// deterministic.
template <int N>
__device__ __forceinline__ void reduce_scatter8(float (&x)[N], int ii) {
#pragma unroll
    for (int m = 4, h = N / 2; m >= 1; m >>= 1, h >>= 1) {
        const bool up = (ii & m) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float keep = up ? x[k + h] : x[k];
            const float send = up ? x[k] : x[k + h];
            x[k] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
}

__device__ __forceinline__ void add_fix(long long* p, float f) {
    if (f != 0.0f) fix_atomic_add(p, fix_from_float(f));
}

// j-atom data of one list entry for lane group jq: atoms jq and jq + 4 of
// cluster cj (position + charge, sigma/eps, home index or INVALID_ID)
struct JAtoms { float4 p0, p1; float2 l0, l1; uint32_t a0, a1; };
__device__ __forceinline__ JAtoms load_jatoms(const SysView& v, uint32_t cj, int jq) {
    const uint32_t s = cj * ACL + jq;
    return JAtoms{v.spos[s], v.spos[s + 4], v.slj[s], v.slj[s + 4], v.sidx[s], v.sidx[s + 4]};
}

// ---------------------------------------------------------------------------
// water - atom, each pair once.  One warp per work item: an atom cluster (up
// to 8 atoms) and 32 of the waters listed within the list radius of any of its
// atoms.  A lane takes one water and evaluates it against the cluster's atoms
// in turn (their data is the same for all lanes: one broadcast load each), so
// that the lanes' work is the listed waters and not the pairs of two bounding
// boxes.  The water's forces stay in registers over the atoms and are added
// once (12 int64 reductions); each lane keeps its share of the atoms' forces
// in shared memory (24 sums per lane, no conflicts), added up over the lanes
// in a fixed order at the end, one lane per component.  An atom beyond the
// cutoff plus the O-H reach of all 32 waters is skipped by a vote.
//
// Bound by issue (the energies take about as much as the forces, on every
// step by default) at 16 warps per SM.  24,000 waters and 5,000 atoms: 40 us
// and 18 M warp instructions, against 74 us and 40 M for pairs of an 8-water
// and an 8-atom cluster (few of whose 64 pairs are in range: the water
// clusters are 2.7 A thin in a column 10.8 A wide); 8,000 waters and 640 atoms
// 28 -> 16 us, 2,900 and 510 21 -> 15.  Two or four batches of 32 waters per
// item 43 and 45 us; 5 and 6 CTAs per SM 46 and 43.
// ---------------------------------------------------------------------------
DYN_KERNEL_T((bool ENERGY, bool ALCH), (ENERGY, ALCH), __launch_bounds__(PT, 4), k_pair_ws, (, const PairParams P), (, P)) {
    __shared__ float fa[PT / 32][3 * ACL][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint32_t nwarps = (bk.cnt * blockDim.x) >> 5;
    const uint32_t nit = v.sc->n_ws_items;
    const BoxDev b = *v.box;
    const float ljc2 = P.ljc2;
    double el = 0.0, ec = 0.0, dh = 0.0;
    Acc3 a{0.0, 0.0, 0.f, 0.0};
    for (uint32_t it = ((bk.idx * blockDim.x + threadIdx.x) >> 5); it < nit; it += nwarps) {
        const uint2 item = v.ws_item[it];
        const uint32_t ci = item.x, k0 = item.y;
        const bool vi = k0 + lane < v.ws_n[ci];
        const uint32_t s = v.ws_j[(size_t)ci * v.cap_ws + k0 + (vi ? lane : 0)];
        const uint32_t ai = lane < ACL ? v.sidx[ci * ACL + lane] : INVALID_ID;
        const uint32_t am = __ballot_sync(0xffffffffu, ai != INVALID_ID);
#pragma unroll
        for (int k = 0; k < 3 * ACL; ++k) fa[wp][k][lane] = 0.f;
        const float3 iO = xyz(v.wpos[4 * s + 0]), iH0 = xyz(v.wpos[4 * s + 1]);
        const float3 iH1 = xyz(v.wpos[4 * s + 2]), iM = xyz(v.wpos[4 * s + 3]);
        float3 fO = f3(0, 0, 0), fH0 = fO, fH1 = fO, fM = fO;
        for (uint32_t mm = am; mm; mm &= mm - 1u) {
            const int k = __ffs(mm) - 1;
            const float4 pj = v.spos[ci * ACL + k];
            const float2 lj_j = v.slj[ci * ACL + k];
            // the atom moved to the image nearest the water's O once
            const float3 jp = xyz(pj), z0 = f3(0.f, 0.f, 0.f);
            const float3 js = f3(fmaf(nearest_int(iO.x - jp.x, b.inv_ext[0]), b.ext[0], jp.x),
                                 fmaf(nearest_int(iO.y - jp.y, b.inv_ext[1]), b.ext[1], jp.y),
                                 fmaf(nearest_int(iO.z - jp.z, b.inv_ext[2]), b.ext[2], jp.z));
            const float3 dO = iO - js;
            if (!__any_sync(0xffffffffu, vi && dot3(dO, dO) < v.r_ws_skip2)) continue;
            if (!vi) continue;
            float3 fo = z0, f0 = z0, f1 = z0, fm = z0;
            const float sg = 0.5f * (OPC_O_SIGMA + lj_j.x);
            const float ep = sqrtf(OPC_O_EPS * lj_j.y);
            const double qe = (double)pj.w;
            const uint32_t aj = ALCH ? v.sidx[ci * ACL + k] : 0u;
            if (ALCH && aj >= v.alch_lo && aj < v.alch_hi) {
                // a water and an atom of the alchemical molecule
                lj_soft<ENERGY>(iO, js, z0, sg, ep, ljc2, v.alch_ll, v.alch_dll, fo, a, dh);
                Acc3 t{0.0, 0.0, 0.f, 0.0};
                coul<ENERGY>(iH0, js, z0, OPC_Q_H * pj.w, (double)OPC_Q_H * qe, P, f0, t);
                coul<ENERGY>(iH1, js, z0, OPC_Q_H * pj.w, (double)OPC_Q_H * qe, P, f1, t);
                coul<ENERGY>(iM, js, z0, OPC_Q_EP * pj.w, (double)OPC_Q_EP * qe, P, fm, t);
                const float cs = v.alch_cs;
                f0 = f0 * cs; f1 = f1 * cs; fm = fm * cs;
                a.w = fmaf(cs, t.w, a.w);
                if (ENERGY) { a.e_c += (double)cs * t.e_c; dh += (double)v.alch_dcs * t.e_c; }
            } else {
                lj<ENERGY>(iO, js, z0, sg * sg, ep, ljc2, 1.0f, fo, a);
                coul<ENERGY>(iH0, js, z0, OPC_Q_H * pj.w, (double)OPC_Q_H * qe, P, f0, a);
                coul<ENERGY>(iH1, js, z0, OPC_Q_H * pj.w, (double)OPC_Q_H * qe, P, f1, a);
                coul<ENERGY>(iM, js, z0, OPC_Q_EP * pj.w, (double)OPC_Q_EP * qe, P, fm, a);
            }
            a.flush_w();
            fO = fO + fo; fH0 = fH0 + f0; fH1 = fH1 + f1; fM = fM + fm;
            const float3 t = (fo + f0) + (f1 + fm);
            fa[wp][3 * k + 0][lane] -= t.x;
            fa[wp][3 * k + 1][lane] -= t.y;
            fa[wp][3 * k + 2][lane] -= t.z;
        }
        if (vi) {
            long long* p = v.wforce + (size_t)s * 12;
            add_fix3(p + 0, fO); add_fix3(p + 3, fH0); add_fix3(p + 6, fH1); add_fix3(p + 9, fM);
        }
        __syncwarp();
        // lane 3 k + c adds up component c of atom k (rotated: no bank conflicts)
        const uint32_t at = __shfl_sync(0xffffffffu, ai, lane / 3);
        if (lane < 3 * ACL && at != INVALID_ID) {
            float f = 0.f;
#pragma unroll 8
            for (int j = 0; j < 32; ++j) f += fa[wp][lane][(lane + j) & 31];
            add_fix(v.aforce + 3 * (size_t)at + lane % 3, f);
        }
        __syncwarp();
    }
    if (ENERGY) { el = a.e_lj; ec = a.e_c; }
    write_partials_warp<ENERGY>(v, bk, REG_WS, el, ec, a.wd, dh);
}

// ---------------------------------------------------------------------------
// atom(i) - atom(j), each pair once (cluster pairs with cj >= ci; the
// interaction mask from the list build holds jj > ii on the diagonal and
// drops exclusions); work items, prefetch and j-side atomics as above.
// ---------------------------------------------------------------------------
DYN_KERNEL_T((bool ENERGY, bool ALCH), (ENERGY, ALCH), __launch_bounds__(PT), k_pair_ss, (, const PairParams P), (, P)) {
    const int lane = threadIdx.x & 31;
    const int ii = lane & 7, jq = lane >> 3;
    const uint32_t nwarps = (bk.cnt * blockDim.x) >> 5;
    const uint32_t nit = v.sc->n_ss_items;
    const BoxDev b = *v.box;
    const float ljc2 = P.ljc2;
    double el = 0.0, ec = 0.0, ew = 0.0, dh = 0.0;
    for (uint32_t it = ((bk.idx * blockDim.x + threadIdx.x) >> 5); it < nit; it += nwarps) {
        const uint2 item = v.ss_item[it];
        const uint32_t ci = item.x, k0 = item.y;
        const uint32_t n = min(v.ss_n[ci], k0 + v.ch_mix) - k0;
        const uint32_t si = ci * ACL + ii;
        const uint32_t ai = v.sidx[si];
        const float4 pi = v.spos[si];
        const float2 lji = v.slj[si];
        float3 f = f3(0, 0, 0);
        Acc3 a{0.0, 0.0, 0.f, 0.0};
        const size_t row = (size_t)ci * v.cap_ss + k0;
        const uint32_t my_j = (uint32_t)lane < n ? v.ss_j[row + lane] : 0u;
        const unsigned long long my_m = (uint32_t)lane < n ? v.ss_mask[row + lane] : 0ull;
        JAtoms nx = load_jatoms(v, __shfl_sync(0xffffffffu, my_j, 0), jq);
        for (uint32_t k = 0; k < n; ++k) {
            const JAtoms cur = nx;
            const unsigned long long m = __shfl_sync(0xffffffffu, my_m, k);
            if (k + 1 < n) nx = load_jatoms(v, __shfl_sync(0xffffffffu, my_j, k + 1), jq);
            float jf[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int jj = jq + 4 * h;
                const float4 pj = h ? cur.p1 : cur.p0;
                const float2 ljj = h ? cur.l1 : cur.l0;
                float3 fp = f3(0, 0, 0);
                if ((m >> (ii * ACL + jj)) & 1ull) {
                    const float3 s = shift_of(xyz(pi) - xyz(pj), b);
                    const float sg = 0.5f * (lji.x + ljj.x);
                    const uint32_t aj = h ? cur.a1 : cur.a0;
                    if (ALCH && ((ai >= v.alch_lo && ai < v.alch_hi) != (aj >= v.alch_lo && aj < v.alch_hi))) {
                        // exactly one atom of the pair in the alchemical molecule
                        lj_soft<ENERGY>(xyz(pi), xyz(pj), s, sg, sqrtf(lji.y * ljj.y), ljc2, v.alch_ll, v.alch_dll,
                                        fp, a, dh);
                        Acc3 t{0.0, 0.0, 0.f, 0.0};
                        float3 fc = f3(0.f, 0.f, 0.f);
                        coul<ENERGY>(xyz(pi), xyz(pj), s, pi.w * pj.w, (double)pi.w * (double)pj.w, P, fc, t);
                        const float cs = v.alch_cs;
                        fp = fp + fc * cs;
                        a.w = fmaf(cs, t.w, a.w);
                        if (ENERGY) { a.e_c += (double)cs * t.e_c; dh += (double)v.alch_dcs * t.e_c; }
                    } else {
                        lj<ENERGY>(xyz(pi), xyz(pj), s, sg * sg, sqrtf(lji.y * ljj.y), ljc2, 1.0f, fp, a);
                        coul<ENERGY>(xyz(pi), xyz(pj), s, pi.w * pj.w, (double)pi.w * (double)pj.w, P, fp, a);
                    }
                }
                f = f + fp;
                jf[3 * h + 0] = -fp.x; jf[3 * h + 1] = -fp.y; jf[3 * h + 2] = -fp.z;
            }
            jf[6] = 0.f; jf[7] = 0.f;
            a.flush_w();
            // lane ii < 6 now holds component ii % 3 of atom jq + 4 (ii / 3)
            reduce_scatter8(jf, ii);
            if (ii < 6) {
                const uint32_t aj = ii < 3 ? cur.a0 : cur.a1;
                if (aj != INVALID_ID) add_fix(v.aforce + 3 * (size_t)aj + ii % 3, jf[0]);
            }
        }
        f = f3(red4(f.x), red4(f.y), red4(f.z));
        if (jq == 0 && ai != INVALID_ID) add_fix3(v.aforce + 3 * (size_t)ai, f);
        if (ENERGY) { el += a.e_lj; ec += a.e_c; }
        a.flush_w();
        ew += a.wd;
    }
    write_partials_warp<ENERGY>(v, bk, REG_SS, el, ec, ew, dh);
}

// ---------------------------------------------------------------------------
// 1-4 pairs: LJ x0.5, Coulomb x1/1.2 (src/non_bonded.rs:55-56,1014-1042)
// ---------------------------------------------------------------------------
DYN_KERNEL_T((bool ENERGY), (ENERGY), , k_pair14, (, const PairParams P), (, P)) {
    const BoxDev b = *v.box;
    double e_acc = 0.0, w_acc = 0.0;
    for (uint32_t k = bk.idx * blockDim.x + threadIdx.x; k < v.n14; k += bk.cnt * blockDim.x) {
        const uint2 p = v.p14[k];
        const float4 par = v.p14_par[k];  // sigma, eps, qq
        const float4 pa = v.apos[p.x], pb = v.apos[p.y];
        const float3 sh = shift_of(xyz(pa) - xyz(pb), b);
        float3 f = f3(0, 0, 0);
        Acc3 a{0.0, 0.0, 0.f, 0.0};
        lj<ENERGY>(xyz(pa), xyz(pb), sh, par.x * par.x, par.y, P.ljc2, 0.5f, f, a);
        float3 fc = f3(0, 0, 0);
        Acc3 ac{0.0, 0.0, 0.f, 0.0};
        coul<ENERGY>(xyz(pa), xyz(pb), sh, par.z, (double)pa.w * (double)pb.w, P, fc, ac);
        const float s = 0.833333333f;
        f = f + fc * s;
        add_fix3(v.aforce + 3 * (size_t)p.x, f);
        add_fix3(v.aforce + 3 * (size_t)p.y, f3(-f.x, -f.y, -f.z));
        if (ENERGY) e_acc += a.e_lj + ac.e_c / 1.2;
        w_acc += (double)a.w + (double)ac.w * s;
    }
    write_partials<ENERGY>(v, bk, REG_14, e_acc, 0.0, w_acc);
}

// Blocks of the atom pair kernels: one per 4 work items, at most one
// resident wave (4 blocks per SM; the kernels loop over the items), which
// also bounds the block partials the step finalisation sums.
inline int pblocks(const SysView& v, uint64_t warps) {
    uint64_t bl = (warps * 32 + PT - 1) / PT;
    if (bl < 1) bl = 1;
    // at most max_blocks / 4: the kernels write one partial per warp
    const uint64_t cap = std::min<uint64_t>(v.max_blocks / (PT / 32), 148u * 4u);
    return (int)(bl < cap ? bl : cap);
}

}  // namespace

namespace dyn {

int pair_blocks_ws(const SysView& v) { return pblocks(v, v.ws_item_cap); }

int ww_tile_blocks(const SysView& v) {
    const uint64_t n = (uint64_t)v.ngrp_cap * v.ww_split;
    return (int)(n < v.max_blocks ? n : v.max_blocks);
}

// per union water: 4 float4 positions, the j sums and its slot
size_t ww_tile_smem(const SysView& v) { return (size_t)v.union_chunk * WW_CHUNK_BYTES; }

// The limit is a property of the kernel, shared by every system in the
// process, so it is raised to the device maximum once rather than set to one
// system's chunk size (which would break systems with larger chunks).
int pair_ww_setup(const SysView& v) {
    int dev = 0, optin = 0;
    DYN_CUDA(cudaGetDevice(&dev));
    DYN_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const void* ks[4] = {(const void*)k_pair_ww_tile<true>, (const void*)k_pair_ww_tile<false>,
                         (const void*)k_pair_ww_tile_batch<true>, (const void*)k_pair_ww_tile_batch<false>};
    for (const void* k : ks) {
        cudaFuncAttributes fa;
        DYN_CUDA(cudaFuncGetAttributes(&fa, k));
        const int lim = optin - (int)fa.sharedSizeBytes;
        DYN_CHECK(ww_tile_smem(v) <= (size_t)lim, DYN_ERR_UNSUPPORTED, "water-water chunk exceeds shared memory");
        DYN_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
    }
    return DYN_OK;
}
int pair_blocks_ss(const SysView& v) { return pblocks(v, v.ss_item_cap); }
int pair14_blocks(const SysView& v) {
    uint64_t bl = (v.n14 + 255) / 256;
    if (bl < 1) bl = 1;
    return (int)(bl < v.max_blocks ? bl : v.max_blocks);
}

void launch_pairs(const Target& t, bool energy) {
    launch_pairs_water(t, energy);
    launch_pairs_atoms(t, energy);
}

// the alchemical variants wherever a system decouples a molecule
inline bool any_alch(const Target& t) {
    return t.any([](const SysView& v) { return v.alch_on != 0u; });
}

// The pair kernels take the cutoffs and the force polynomial by value, so
// that they read them as constants also where their SysView lies in global
// memory (a batch): one launch for every distinct set among the systems, which
// is one unless a batch's members differ in cutoff or alpha.
template <typename KP, typename KB, typename G>
void launch_pair_kernel(const Target& t, KP kp, KB kb, G grid, int threads, size_t smem) {
    std::vector<PairParams> sets;
    auto same = [](const PairParams& a, const PairParams& b) { return std::memcmp(&a, &b, sizeof(PairParams)) == 0; };
    if (t.v) sets.push_back(t.v->pp);
    else
        for (uint32_t i = 0; i < batch_size(t.b); ++i) {
            const PairParams& p = batch_view(t.b, i).pp;
            if (std::none_of(sets.begin(), sets.end(), [&](const PairParams& q) { return same(p, q); }))
                sets.push_back(p);
        }
    for (const PairParams& p : sets)
        t.launch(kp, kb, [&](const SysView& v) { return same(v.pp, p) ? grid(v) : 0; }, threads, smem, p);
}

void launch_pairs_atoms(const Target& t, bool energy) {
    auto ss = [](const SysView& v) { return v.na ? pair_blocks_ss(v) : 0; };
    const bool al = any_alch(t);
    if (energy && al) launch_pair_kernel(t, k_pair_ss<true, true>, k_pair_ss_batch<true, true>, ss, PT, 0);
    else if (energy) launch_pair_kernel(t, k_pair_ss<true, false>, k_pair_ss_batch<true, false>, ss, PT, 0);
    else if (al) launch_pair_kernel(t, k_pair_ss<false, true>, k_pair_ss_batch<false, true>, ss, PT, 0);
    else launch_pair_kernel(t, k_pair_ss<false, false>, k_pair_ss_batch<false, false>, ss, PT, 0);
}

void launch_pairs_ww(const Target& t, bool energy) {
    const size_t sm = t.max_over([](const SysView& v) { return v.nw ? ww_tile_smem(v) : (size_t)0; });
    // water-water short-range energy is part of the potential only with
    // DYN_FLAG_FULL_ENERGY (the reference leaves it out,
    // src/non_bonded.rs:335-342), so other energy steps skip it
    auto eww = [energy](const SysView& v) { return energy && (v.flags & DYN_FLAG_FULL_ENERGY); };
    launch_pair_kernel(t, k_pair_ww_tile<true>, k_pair_ww_tile_batch<true>,
                       [&](const SysView& v) { return v.nw && eww(v) ? ww_tile_blocks(v) : 0; }, WT, sm);
    launch_pair_kernel(t, k_pair_ww_tile<false>, k_pair_ww_tile_batch<false>,
                       [&](const SysView& v) { return v.nw && !eww(v) ? ww_tile_blocks(v) : 0; }, WT, sm);
}

void launch_pairs_water(const Target& t, bool energy) {
    launch_pairs_ww(t, energy);
    launch_pairs_ws(t, energy);
}

void launch_pairs_ws(const Target& t, bool energy) {
    auto ws = [](const SysView& v) { return v.nw && v.na ? pair_blocks_ws(v) : 0; };
    const bool al = any_alch(t);
    if (energy && al) launch_pair_kernel(t, k_pair_ws<true, true>, k_pair_ws_batch<true, true>, ws, PT, 0);
    else if (energy) launch_pair_kernel(t, k_pair_ws<true, false>, k_pair_ws_batch<true, false>, ws, PT, 0);
    else if (al) launch_pair_kernel(t, k_pair_ws<false, true>, k_pair_ws_batch<false, true>, ws, PT, 0);
    else launch_pair_kernel(t, k_pair_ws<false, false>, k_pair_ws_batch<false, false>, ws, PT, 0);
}

void launch_pair14(const Target& t, bool energy) {
    auto g = [](const SysView& v) { return v.n14 ? pair14_blocks(v) : 0; };
    if (energy) launch_pair_kernel(t, k_pair14<true>, k_pair14_batch<true>, g, 256, 0);
    else launch_pair_kernel(t, k_pair14<false>, k_pair14_batch<false>, g, 256, 0);
}

}  // namespace dyn
