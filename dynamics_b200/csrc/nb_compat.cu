// Layer 1 of the C ABI: a drop-in for src/gpu_interface.rs.
//
// The reference uploads 33 bytes of per-pair metadata (15 arrays) and
// evaluates one pair per thread with float atomics
// (src/cuda/cuda.cu:185-362).  Here the same flat pair list is re-packed to
// 20 bytes per pair (two 32-bit words holding index, body code and flag,
// (sigma, eps) and the product q_t q_s), evaluated one pair per thread with
// the reference's float32 pair math, and accumulated into 64-bit fixed-point
// forces, so results are bit-identical run to run.  The pair-list build
// (dyn_nb_build_pairs) replaces the reference's O(N^2) host rebuild with a
// GPU brute-force scan in the reference's exact float32 arithmetic.
// Pairs flagged alchemical (DYN_PAIR_ALCH, or marked by dyn_nb_mark_alch)
// take the reference's soft-core LJ and scaled Coulomb on the staged
// decoupling schedule (nonbonded_force_alchemical_kernel,
// src/cuda/cuda.cu:367-566; f_nonbonded_cpu, src/non_bonded.rs:950-1057).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace {

// packed pair words: w.x = target index (bits 0-26) | alchemical (27) |
// body (28-30) | scale14 (31); w.y = source index (0-27) | body | symmetric
constexpr uint32_t IDX_MASK = 0x0FFFFFFFu;
constexpr uint32_t TGT_MASK = 0x07FFFFFFu;
constexpr uint32_t ALCH_BIT = 0x08000000u;
constexpr int NB_PART = 3;  // virial, energy, dH/dlambda per block
constexpr int NB_BLOCK = 256;
constexpr int NB_MAX_BLOCKS = 148 * 8;

}  // namespace

struct dyn_nb_s {
    cudaStream_t stream = nullptr;
    uint32_t n_dyn = 0, n_water = 0;
    float rc = 10.f, alpha = 0.3f, ljc = 0.f;
    // dyn, O, M, H0, H1, one after another: off[body] + 3 i + component of n_comp
    size_t off[5] = {}, n_comp = 0;
    float* d_pos = nullptr;
    long long* d_f = nullptr;      // fixed-point forces, then virial, energy, dH/dlambda (double)
    float4* d_sphere = nullptr;    // [n_water] centre and radius of each water's sites
    double* d_partials = nullptr;  // [2 * NB_MAX_BLOCKS * NB_PART]
    uint64_t n_alch = 0;           // installed pairs with the alchemical bit
    // device memory of dyn_nb_build_pairs, kept between calls: its inputs and
    // row counts, and the lists of (row, neighbour) pairs
    struct Area { char* p = nullptr; size_t cap = 0; };
    Area scratch, lists;
    // the installed list ends in the ten flat entries of each of these water
    // pairs (in lists): every built list, and a set one in the same order
    uint64_t n_ww = 0;
    const uint32_t* d_wwi = nullptr; const uint32_t* d_wwj = nullptr;
    uint64_t n_pairs = 0, cap_pairs = 0;
    uint2* d_pidx = nullptr;       // packed target/source words
    float2* d_plj = nullptr;       // sigma, eps
    float* d_pqq = nullptr;        // q_t * q_s
    float* h_pos = nullptr;        // pinned staging
    double* h_f = nullptr;
    uint32_t n_of(int a) const { return a == 0 ? n_dyn : n_water; }
};

// ---------------------------------------------------------------------------
// pair evaluation
// ---------------------------------------------------------------------------

__device__ __forceinline__ float3 ld_pos(const float* const* pos, uint32_t body, uint32_t i) {
    // body 0 = atom array, 1..4 = water O, M, H0, H1 arrays
    const float* a = pos[body];
    return f3(a[3 * i + 0], a[3 * i + 1], a[3 * i + 2]);
}

__device__ __forceinline__ float round_half_away(float q) {
    const float t = truncf(q);
    const float fr = __fsub_rn(q, t);
    return fabsf(fr) >= 0.5f ? t + copysignf(1.0f, q) : t;
}

struct PosPtrs { const float* p[5]; };
struct ForcePtrs { long long* f[5]; };

// The staged decoupling schedule of one lambda (staged_decoupling_schedule,
// src/alchemical.rs:77-100): Coulomb scale and its lambda derivative over
// lambda 0..0.5, then the soft-core LJ lambda and its derivative over 0.5..1.
struct AlchSched { float cs, dcs, ll, dll; };

AlchSched alch_schedule(double lambda) {
    float l = (float)lambda;
    l = std::min(1.0f, std::max(0.0f, l));
    if (l < 0.5f) return {1.0f - 2.0f * l, -2.0f, 0.0f, 0.0f};
    return {0.0f, 0.0f, 2.0f * l - 1.0f, 2.0f};
}

// Beutler soft-core LJ of a decoupled pair (alchemical_lj_soft_core_decouple,
// src/non_bonded.rs:883-941; sc-alpha 0.5, power 1, soft-core sigma >= 3 A,
// src/alchemical.rs:55-65): V = (1 - l) V_LJ(r_sc), r_sc^6 = r^6 + 0.5 s^6 l.
// Returns the force magnitude along the pair direction (F_LJ(r_sc) (1 - l)
// (r / r_sc)^5), the energy and dV/dl = -V_LJ(r_sc) - (1 - l) F_LJ(r_sc)
// 0.5 s^6 / (6 r_sc^5).  r2 = 0 gives the energy at contact and no force.
__device__ __forceinline__ void soft_core(float r2, float sig, float eps, float lam, float& fmag,
                                          float& e, float& dvdl) {
    fmag = 0.f; e = 0.f; dvdl = 0.f;
    if (eps == 0.f || !isfinite(eps) || !isfinite(sig)) return;
    const float ss = fmaxf(sig, 3.0f), ss2 = ss * ss;
    const float ss6 = ss2 * ss2 * ss2;
    const float rsc6 = fmaf(0.5f * ss6, lam, r2 * r2 * r2);
    if (!(rsc6 > 0.f) || !isfinite(rsc6)) return;
    const float rsc = sqrtf(cbrtf(rsc6));
    const float inv_rsc = 1.0f / rsc;
    const float sr = sig * inv_rsc, sr2 = sr * sr;
    const float sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
    const float hf = 24.0f * eps * fmaf(2.0f, sr12, -sr6) * inv_rsc;
    const float he = 4.0f * eps * (sr12 - sr6);
    const float scale = 1.0f - lam;
    const float q = sqrtf(r2) * inv_rsc, q2 = q * q;
    fmag = hf * scale * (q2 * q2 * q);
    e = he * scale;
    dvdl = -he - scale * hf * (0.5f * ss6) / (6.0f * (rsc6 * inv_rsc));
}

// CPU_SEM = false: the reference CUDA kernel's conventions
//   (src/cuda/cuda.cu:239-316, alchemical form 367-566): rint min-image by
//   multiplication, r^2 < 1e-16 skip, no LJ cutoff, energy only for atom
//   targets.
// CPU_SEM = true: f_nonbonded_cpu's conventions (src/non_bonded.rs:967-1054):
//   min-image by division with ties away from zero, r^2 < 1e-12 skip (an
//   alchemical pair there keeps its soft-core contact energy), LJ only for
//   r <= lj_cutoff, energy when either body is an atom.
// ALCH: pairs with the alchemical bit take soft-core LJ at the schedule's LJ
//   lambda and Coulomb times its scale; their dH/dlambda is summed.
struct PairConsts {
    float3 ext, inv_ext;
    float3 half;   // displacements below it are their own nearest image
    float rc, alpha, ljc;
    uint32_t ovr;
};

template <bool CPU_SEM>
__device__ __forceinline__ float image1(float d, float ext, float inv_ext, float half) {
    // |d| < half = 0.4999 extents: the quotient rounds to zero and d stays
    if (fabsf(d) < half) return d;
    if (CPU_SEM) return __fsub_rn(d, __fmul_rn(round_half_away(__fdiv_rn(d, ext)), ext));
    return d - rintf(d * inv_ext) * ext;
}

// One pair with displacement d (nearest image) and r2 = |d|^2: its force on
// the target is d times the returned value; e and dh receive its energy and
// dH/dlambda.
template <bool CPU_SEM, bool ALCH>
__device__ __forceinline__ float pair_eval(float r2, float sigma, float eps, float qq, bool scale14, bool alch,
                                           const PairConsts& c, const AlchSched& al, float& e, float& dh) {
    e = 0.f;
    dh = 0.f;
    const bool lj_off = c.ovr & DYN_OVR_LJ_DISABLED;
    const bool co_off = c.ovr & DYN_OVR_COULOMB_DISABLED;
    if (r2 < (CPU_SEM ? 1e-12f : 1e-16f)) {
        if (CPU_SEM && ALCH && alch && !lj_off && eps != 0.f) {
            float fs;
            soft_core(0.f, sigma, eps, al.ll, fs, e, dh);
            if (scale14) { e *= 0.5f; dh *= 0.5f; }
            dh *= al.dll;
        }
        return 0.f;
    }
    const float inv_r = rsqrtf(r2);
    const float r = r2 * inv_r;
    float fmag = 0.f;
    if (!lj_off && eps != 0.f && (!CPU_SEM || r <= c.ljc)) {
        float fl, el;
        if (ALCH && alch) {
            soft_core(r2, sigma, eps, al.ll, fl, el, dh);
            dh *= al.dll;
        } else {
            const float sr = sigma * inv_r;
            const float sr2 = sr * sr;
            const float sr6 = sr2 * sr2 * sr2;
            const float sr12 = sr6 * sr6;
            fl = 24.0f * eps * fmaf(2.f, sr12, -sr6) * inv_r;
            el = 4.f * eps * (sr12 - sr6);
        }
        if (scale14) { fl *= 0.5f; el *= 0.5f; dh *= 0.5f; }
        fmag += fl; e += el;
    }
    if (!co_off && qq != 0.f && r < c.rc) {
        const float ar = c.alpha * r;
        const float ec = erfcf(ar);
        const float ex = expf(-(ar * ar));
        float fc = qq * fmaf(ec, inv_r * inv_r, 2.0f * c.alpha * ex * INV_SQRT_PI_F * inv_r);
        float eco = qq * inv_r * ec;
        if (scale14) { fc *= 0.833333333f; eco *= 0.833333333f; }
        if (ALCH && alch) {
            fmag += fc * al.cs; e += eco * al.cs;
            dh += eco * al.dcs;
        } else {
            fmag += fc; e += eco;
        }
    }
    return fmag * inv_r;
}

__device__ __forceinline__ void write_nb_partials(double w, double e, double h, double* __restrict__ partials) {
    double v[NB_PART] = {w, e, h};
    block_sum_d<NB_PART>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < NB_PART; ++k) partials[NB_PART * blockIdx.x + k] = v[k];
}

__device__ __forceinline__ double virial_of(float3 d, float3 f) {
    return (double)d.x * (double)f.x + (double)d.y * (double)f.y + (double)d.z * (double)f.z;
}

// The general kernel: any flat pair list, one pair per thread.  Pairs beyond
// the cutoffs (most of a list with the reference's 4 A skin) add nothing and
// skip their six 64-bit reductions, which bound the kernel.
template <bool CPU_SEM, bool ALCH>
__global__ void __launch_bounds__(NB_BLOCK) nb_pair_kernel(
    PosPtrs pos, ForcePtrs out, const uint2* __restrict__ pidx, const float2* __restrict__ plj,
    const float* __restrict__ pqq, uint64_t n, PairConsts c, AlchSched al, double* __restrict__ partials) {
    double w_acc = 0.0, e_acc = 0.0, h_acc = 0.0;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 w = pidx[p];
        const uint32_t bt = (w.x >> 28) & 7u, bs = (w.y >> 28) & 7u;
        const uint32_t it = w.x & TGT_MASK, is = w.y & IDX_MASK;
        const bool scale14 = w.x >> 31, sym = w.y >> 31;
        const float3 pt = ld_pos(pos.p, bt, it);
        const float3 ps = ld_pos(pos.p, bs, is);
        float3 d = pt - ps;
        d.x = image1<CPU_SEM>(d.x, c.ext.x, c.inv_ext.x, c.half.x);
        d.y = image1<CPU_SEM>(d.y, c.ext.y, c.inv_ext.y, c.half.y);
        d.z = image1<CPU_SEM>(d.z, c.ext.z, c.inv_ext.z, c.half.z);
        const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
        const float2 lj = plj[p];
        float e, dh;
        const float fs = pair_eval<CPU_SEM, ALCH>(r2, lj.x, lj.y, pqq[p], scale14, ALCH && (w.x & ALCH_BIT), c, al, e, dh);
        if (CPU_SEM ? (bt == 0 || bs == 0) : (bt == 0)) e_acc += (double)e;
        if (ALCH) h_acc += (double)dh;
        if (fs == 0.f && isfinite(r2)) continue;
        const float3 f = d * fs;
        w_acc += virial_of(d, f);
        long long* ft = out.f[bt] + 3 * (size_t)it;
        fix_atomic_add(ft + 0, fix_from_float(f.x));
        fix_atomic_add(ft + 1, fix_from_float(f.y));
        fix_atomic_add(ft + 2, fix_from_float(f.z));
        if (sym) {
            long long* fsrc = out.f[bs] + 3 * (size_t)is;
            fix_atomic_add(fsrc + 0, -fix_from_float(f.x));
            fix_atomic_add(fsrc + 1, -fix_from_float(f.y));
            fix_atomic_add(fsrc + 2, -fix_from_float(f.z));
        }
    }
    write_nb_partials(w_acc, e_acc, h_acc, partials);
}

// Bounding spheres of the waters: the midpoint of the hydrogens and the
// largest distance of a site from it, with room for the rounding of this and
// of the distances compared with it.  Waters of any shape, also one broken
// over the box's faces, whose sphere is then as large as the box.
__global__ void nb_sphere_kernel(PosPtrs pos, uint32_t n, float3 ext, float4* __restrict__ sphere) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 h0 = ld_pos(pos.p, 3, i), h1 = ld_pos(pos.p, 4, i);
        const float3 c = (h0 + h1) * 0.5f;
        float r2 = 0.f, big = fmaxf(ext.x, fmaxf(ext.y, ext.z));
        bool finite = true;
        for (int b = 1; b < 5; ++b) {
            const float3 x = ld_pos(pos.p, b, i), d = x - c;
            const float d2 = dot3(d, d);
            finite = finite && isfinite(d2);
            r2 = fmaxf(r2, d2);
            big = fmaxf(big, fmaxf(fabsf(x.x), fmaxf(fabsf(x.y), fabsf(x.z))));
        }
        sphere[i] = make_float4(c.x, c.y, c.z, finite ? sqrtf(r2) * 1.000001f + 2e-6f * big : INFINITY);
    }
}

// The water-water part of a list in setup_pairs' order, from its
// molecule pairs (8 bytes each) instead of their ten flat entries (200 bytes).
// A warp takes 32 run consecutive molecule pairs, which mostly share the
// first water, and its lanes equal contiguous shares of them: every site pair
// is evaluated and rounded to fixed point as by the general kernel, the first
// water's forces are summed in 64-bit registers until it changes and the
// second's per molecule pair, so the sums are the same integers.  With an LJ
// cutoff (CPU_SEM) no force reaches beyond the cutoffs, and only the molecule
// pairs whose bounding spheres come that near are shared out: bound by issue,
// and two thirds of a list with skin lie beyond, but a warp in which one lane's
// pair is in reach evaluates for all.  1.4 M molecule pairs of 7,800 waters
// (13 A list, 9 A cutoff): 116 us, 176 without the selection, 942 as 14 M flat
// entries with six reductions each.  Runs of 16 where that leaves two waves of
// threads, shorter ones below (89,000 molecule pairs in runs of 8 left most of
// the SMs without work: 58 us).
constexpr uint64_t WW_RUN = 16, WW_THREADS = 148 * 1024;
inline uint32_t ww_run(uint64_t n) { return (uint32_t)std::max<uint64_t>(1, std::min(WW_RUN, n / WW_THREADS)); }

template <bool CPU_SEM>
__global__ void __launch_bounds__(NB_BLOCK) nb_ww_kernel(PosPtrs pos, ForcePtrs out, const uint32_t* __restrict__ wi,
                                                         const uint32_t* __restrict__ wj, uint64_t n, uint32_t run,
                                                         const float4* __restrict__ sphere, PairConsts c,
                                                         double* __restrict__ partials) {
    __shared__ uint16_t near[CPU_SEM ? NB_BLOCK * WW_RUN : 1];  // a warp's selected pairs
    // sites in setup_pairs' order O, M, H0, H1 = bodies 1..4
    const float q[4] = {0.f, OPC_Q_EP, OPC_Q_H, OPC_Q_H};
    const AlchSched none{1.f, 0.f, 0.f, 0.f};
    double w_acc = 0.0;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, piece = 32u * run;
    uint16_t* sel = near + (CPU_SEM ? warp * piece : 0u);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * run;
    // k0: the warp's first pair, the same in all its lanes
    for (uint64_t k0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + warp) * piece; k0 < n; k0 += stride) {
        uint32_t cnt = k0 + piece < n ? piece : (uint32_t)(n - k0);
        if (CPU_SEM) {
            const float reach = fmaxf(c.rc, c.ljc);
            uint32_t m = 0;
            for (uint32_t t = lane; t < piece; t += 32) {
                bool in = false;
                if (t < cnt) {
                    const float4 a = sphere[wi[k0 + t]], b = sphere[wj[k0 + t]];
                    float3 d = f3(a.x - b.x, a.y - b.y, a.z - b.z);
                    d.x -= rintf(d.x * c.inv_ext.x) * c.ext.x;
                    d.y -= rintf(d.y * c.inv_ext.y) * c.ext.y;
                    d.z -= rintf(d.z * c.inv_ext.z) * c.ext.z;
                    const float d2 = dot3(d, d), l = reach + a.w + b.w;
                    // not finite: evaluated, as without the selection
                    in = !(d2 > l * l) || !isfinite(d2);
                }
                const uint32_t mask = __ballot_sync(0xffffffffu, in);
                if (in) sel[m + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)t;
                m += __popc(mask);
            }
            cnt = m;
            __syncwarp();
        }
        const uint32_t t0 = lane * cnt / 32u, t1 = (lane + 1u) * cnt / 32u;
        uint32_t cur = 0xFFFFFFFFu;
        float3 pi[4];
        long long fi[12];
        bool any_i = false;
        auto flush = [&]() {
            if (any_i)
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        if (fi[3 * s + x]) fix_atomic_add(out.f[s + 1] + 3 * (size_t)cur + x, fi[3 * s + x]);
        };
        for (uint32_t t2 = t0; t2 < t1; ++t2) {
            const uint64_t k = k0 + (CPU_SEM ? (uint32_t)sel[t2] : t2);
            const uint32_t i = wi[k], j = wj[k];
            if (i != cur) {
                flush();
                cur = i;
                any_i = false;
#pragma unroll
                for (int s = 0; s < 4; ++s) pi[s] = ld_pos(pos.p, s + 1, i);
#pragma unroll
                for (int x = 0; x < 12; ++x) fi[x] = 0;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float3 pj = ld_pos(pos.p, t + 1, j);
                long long fj[3] = {0, 0, 0};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    if ((s == 0) != (t == 0)) continue;  // O-O (LJ) and the charged sites' pairs
                    float3 d = pi[s] - pj;
                    d.x = image1<CPU_SEM>(d.x, c.ext.x, c.inv_ext.x, c.half.x);
                    d.y = image1<CPU_SEM>(d.y, c.ext.y, c.inv_ext.y, c.half.y);
                    d.z = image1<CPU_SEM>(d.z, c.ext.z, c.inv_ext.z, c.half.z);
                    const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
                    float e, dh;
                    const float fs = pair_eval<CPU_SEM, false>(r2, OPC_O_SIGMA, s == 0 ? OPC_O_EPS : 0.f,
                                                               s == 0 ? 0.f : __fmul_rn(q[s], q[t]), false, false, c,
                                                               none, e, dh);
                    if (fs == 0.f && isfinite(r2)) continue;
                    const float3 f = d * fs;
                    w_acc += virial_of(d, f);
                    const long long x = fix_from_float(f.x), y = fix_from_float(f.y), z = fix_from_float(f.z);
                    fi[3 * s + 0] += x; fi[3 * s + 1] += y; fi[3 * s + 2] += z;
                    fj[0] -= x; fj[1] -= y; fj[2] -= z;
                    any_i = true;
                }
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    if (fj[x]) fix_atomic_add(out.f[t + 1] + 3 * (size_t)j + x, fj[x]);
            }
        }
        flush();
        __syncwarp();  // the selection is refilled
    }
    write_nb_partials(w_acc, 0.0, 0.0, partials);
}

// Sums block partials in a fixed order (deterministic).
//
// Block 0 sums the blocks' partials into the scalars behind the n force
// components; the others turn those from fixed point into float64 in place,
// so that one copy takes the whole result to the host in the caller's type
// (six copies before, then a conversion per component on one host core: 303
// -> 229 us for a list of 512 waters and its forces, 398 -> 389 us for the
// forces of 14 M pairs).
__global__ void nb_finalize_kernel(const double* __restrict__ partials, int nblocks, long long* f, uint32_t n) {
    if (blockIdx.x > 0) {
        for (uint32_t k = (blockIdx.x - 1) * blockDim.x + threadIdx.x; k < n; k += (gridDim.x - 1) * blockDim.x)
            f[k] = __double_as_longlong((double)f[k] * DYN_FIX_INV);
        return;
    }
    double* scalars = reinterpret_cast<double*>(f + n);
    double v[NB_PART] = {0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
        for (int k = 0; k < NB_PART; ++k) v[k] += partials[NB_PART * b + k];
    block_sum_d<NB_PART>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < NB_PART; ++k) scalars[k] = v[k];
}

// Marks the installed pairs that cross the boundary of the atom range
// [lo, hi) as alchemical, as setup_pairs does for the alchemical molecule
// (src/non_bonded.rs:581-612): atom-atom pairs with exactly one end inside,
// atom-water pairs whose atom is inside; water-water pairs never.  Clears
// the bit on every other pair and counts the marked ones.
__global__ void mark_alch_kernel(uint64_t n, uint32_t lo, uint32_t hi, uint2* __restrict__ pidx,
                                 unsigned long long* __restrict__ count) {
    uint32_t c = 0;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        uint2 w = pidx[p];
        const uint32_t bt = (w.x >> 28) & 7u, bs = (w.y >> 28) & 7u;
        const uint32_t it = w.x & TGT_MASK, is = w.y & IDX_MASK;
        const bool in_t = bt == 0 && it >= lo && it < hi;
        const bool in_s = bs == 0 && is >= lo && is < hi;
        const bool a = in_t != in_s;
        w.x = a ? (w.x | ALCH_BIT) : (w.x & ~ALCH_BIT);
        pidx[p] = w;
        c += a;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
}

__global__ void pack_pairs_kernel(uint64_t n, const uint32_t* __restrict__ tgt,
                                  const uint32_t* __restrict__ src, const float* __restrict__ sig,
                                  const float* __restrict__ eps, const float* __restrict__ qt,
                                  const float* __restrict__ qs, const uint8_t* __restrict__ bt,
                                  const uint8_t* __restrict__ bs, const uint8_t* __restrict__ fl,
                                  uint2* __restrict__ pidx, float2* __restrict__ plj,
                                  float* __restrict__ pqq) {
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t f = fl[p];
        uint2 w;
        w.x = (tgt[p] & TGT_MASK) | ((uint32_t)(bt[p] & 7u) << 28) |
              ((f & DYN_PAIR_SCALE14) ? 0x80000000u : 0u) | ((f & DYN_PAIR_ALCH) ? ALCH_BIT : 0u);
        w.y = (src[p] & IDX_MASK) | ((uint32_t)(bs[p] & 7u) << 28) | ((f & DYN_PAIR_SYMMETRIC) ? 0x80000000u : 0u);
        pidx[p] = w;
        plj[p] = make_float2(sig[p], (f & DYN_PAIR_LJ) ? eps[p] : 0.f);
        pqq[p] = (f & DYN_PAIR_COULOMB) ? __fmul_rn(qt[p], qs[p]) : 0.f;
    }
}

// ---------------------------------------------------------------------------
// reference-exact neighbour lists (src/neighbors.rs:180-281) + setup_pairs
// ---------------------------------------------------------------------------

// SimBox::min_image in float32, no contraction (src/barostat.rs:162-170).
__device__ __forceinline__ float mi1(float dv, float e) {
    return __fsub_rn(dv, __fmul_rn(round_half_away(__fdiv_rn(dv, e)), e));
}
__device__ __forceinline__ float dist2_ref(float3 a, float3 b, float3 ext) {
    const float x = mi1(__fsub_rn(a.x, b.x), ext.x);
    const float y = mi1(__fsub_rn(a.y, b.y), ext.y);
    const float z = mi1(__fsub_rn(a.z, b.z), ext.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
}
// SimBox::wrap (src/barostat.rs:141-157): rem_euclid then + lo.
__device__ __forceinline__ float wrap1(float p, float lo, float e) {
    float r = fmodf(__fsub_rn(p, lo), e);
    if (r < 0.f) r = __fadd_rn(r, fabsf(e));
    return __fadd_rn(r, lo);
}

__global__ void wrap_o_kernel(uint32_t nw, const float* __restrict__ o, float3 lo, float3 ext,
                              float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nw) return;
    out[3 * i + 0] = wrap1(o[3 * i + 0], lo.x, ext.x);
    out[3 * i + 1] = wrap1(o[3 * i + 1], lo.y, ext.y);
    out[3 * i + 2] = wrap1(o[3 * i + 2], lo.z, ext.z);
}

__device__ __forceinline__ bool in_sorted(const uint32_t* a, uint32_t n, uint32_t v) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        if (a[m] < v) lo = m + 1; else hi = m;
    }
    return lo < n && a[lo] == v;
}

struct ListArgs {
    const float* outer;    // [3*n_outer]
    const float* inner;    // [3*n_inner]
    uint32_t n_outer, n_inner;
    int mode;              // 0 std-std (half, j>i), 1 std-water, 2 water-water (half)
    float thr;             // (cutoff+skin)^2
    float3 ext;
    const uint8_t* is_static;
    const uint8_t* bonded_only;
    const uint32_t* ex_off; const uint32_t* ex_idx;   // exclusions CSR (std-std)
    const uint32_t* s14_off; const uint32_t* s14_idx; // 1-4 CSR
};

// One warp per outer row; inner indices are scanned in ascending order and
// compacted with ballots, so rows come out sorted, as in the reference.
// PASS 0 counts pairs per row; PASS 1 writes them at row offsets.
template <int PASS>
__global__ void ref_list_kernel(ListArgs a, uint32_t* __restrict__ row_count,
                                const uint64_t* __restrict__ row_off, uint32_t* __restrict__ out_i,
                                uint32_t* __restrict__ out_j, uint8_t* __restrict__ out_s14) {
    const int lane = threadIdx.x & 31;
    const uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= a.n_outer) return;
    const float3 pi = f3(a.outer[3 * row], a.outer[3 * row + 1], a.outer[3 * row + 2]);
    const uint32_t j0 = (a.mode == 1) ? 0u : row + 1;
    uint32_t cnt = 0;
    uint64_t base = PASS ? row_off[row] : 0;
    for (uint32_t jb = j0; jb < a.n_inner; jb += 32) {
        const uint32_t j = jb + lane;
        bool hit = false;
        bool s14 = false;
        if (j < a.n_inner) {
            const float3 pj = f3(a.inner[3 * j], a.inner[3 * j + 1], a.inner[3 * j + 2]);
            bool skip = false;
            if (a.mode == 0) {
                if (a.is_static && a.is_static[row] && a.is_static[j]) skip = true;
            }
            if (!skip) hit = dist2_ref(pi, pj, a.ext) < a.thr;
            if (hit && a.mode == 0) {
                // setup_pairs filters (src/non_bonded.rs:572-580)
                if (a.bonded_only && (a.bonded_only[row] || a.bonded_only[j])) hit = false;
                if (hit && a.ex_off &&
                    in_sorted(a.ex_idx + a.ex_off[row], a.ex_off[row + 1] - a.ex_off[row], j))
                    hit = false;
                if (hit && a.s14_off)
                    s14 = in_sorted(a.s14_idx + a.s14_off[row], a.s14_off[row + 1] - a.s14_off[row], j);
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (PASS && hit) {
            const uint32_t k = cnt + __popc(m & ((1u << lane) - 1u));
            out_i[base + k] = row;
            out_j[base + k] = j;
            if (out_s14) out_s14[base + k] = s14;
        }
        cnt += __popc(m);
    }
    if (!PASS && lane == 0) row_count[row] = cnt;
}

// Exclusive sums of the rows' counts and their total, a block per list.
struct ScanArgs { const uint32_t* cnt[3]; uint64_t* off[3]; uint32_t n[3]; uint64_t* total; };
constexpr int SCAN_T = 1024;
__global__ void __launch_bounds__(SCAN_T) scan_rows_kernel(ScanArgs a) {
    __shared__ uint64_t ws[SCAN_T / 32];
    const uint32_t* cnt = a.cnt[blockIdx.x];
    uint64_t* off = a.off[blockIdx.x];
    const uint32_t n = a.n[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t base = 0;
    for (uint64_t c0 = 0; c0 < n; c0 += SCAN_T) {
        const uint64_t c = c0 + threadIdx.x;
        const uint64_t k = c < n ? cnt[c] : 0u;
        uint64_t x = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[w] = x;
        __syncthreads();
        if (w == 0) {
            uint64_t t = ws[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            ws[lane] = t;
        }
        __syncthreads();
        if (c < n) off[c] = base + (w ? ws[w - 1] : 0u) + x - k;
        base += ws[SCAN_T / 32 - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) { off[n] = base; a.total[blockIdx.x] = base; }
}

// The flat SoA of setup_pairs from the three lists of (row, neighbour)
// pairs, one flat entry per thread so that the writes are contiguous: 0.9 M
// entries in 5 us; a thread per row, whose lanes wrote 200 bytes apart, took
// 698 us for the water part and 260 for the water-atom part.
struct EmitArgs {
    uint64_t n_ss, n_sw, n_ww;  // list entries
    const uint32_t* ss_i; const uint32_t* ss_j; const uint8_t* ss_s14;
    const uint32_t* sw_i; const uint32_t* sw_j;
    const uint32_t* ww_i; const uint32_t* ww_j;
    const float* q; const float* sig; const float* eps;
};

// water site codes in setup_pairs' iteration order O, M, H0, H1
__device__ __forceinline__ float site_q(uint32_t s) {
    return s == DYN_BODY_W_O ? 0.f : (s == DYN_BODY_W_M ? OPC_Q_EP : OPC_Q_H);
}

__global__ void __launch_bounds__(NB_BLOCK) emit_pairs_kernel(EmitArgs a, uint2* __restrict__ pidx,
                                                              float2* __restrict__ plj, float* __restrict__ pqq) {
    const uint64_t base_sw = a.n_ss, base_ww = base_sw + 4 * a.n_sw, n = base_ww + 10 * a.n_ww;
    for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (uint64_t)gridDim.x * blockDim.x) {
        uint2 w;
        float2 lj;
        float qq;
        if (o >= base_ww) {
            // O-O, then M, H0, H1 against M, H0, H1
            const uint64_t k = (o - base_ww) / 10u;
            const uint32_t t = (uint32_t)((o - base_ww) - 10u * k);
            const uint32_t s0 = t ? DYN_BODY_W_M + (t - 1) / 3u : DYN_BODY_W_O;
            const uint32_t s1 = t ? DYN_BODY_W_M + (t - 1) % 3u : DYN_BODY_W_O;
            w = make_uint2(a.ww_i[k] | (s0 << 28), a.ww_j[k] | (s1 << 28) | 0x80000000u);
            lj = make_float2(OPC_O_SIGMA, t ? 0.f : OPC_O_EPS);
            qq = t ? __fmul_rn(site_q(s0), site_q(s1)) : 0.f;
        } else if (o >= base_sw) {
            const uint64_t k = (o - base_sw) >> 2;
            const uint32_t s = DYN_BODY_W_O + (uint32_t)((o - base_sw) & 3u);
            const uint32_t i = a.sw_i[k];
            w = make_uint2(i, a.sw_j[k] | (s << 28) | 0x80000000u);
            // water_std row of LjTables (src/non_bonded.rs:139-145)
            lj = make_float2(__fmul_rn(0.5f, __fadd_rn(a.sig[i], OPC_O_SIGMA)),
                             s == DYN_BODY_W_O ? __fsqrt_rn(__fmul_rn(a.eps[i], OPC_O_EPS)) : 0.f);
            qq = s == DYN_BODY_W_O ? 0.f : __fmul_rn(a.q[i], site_q(s));
        } else {
            const uint32_t i = a.ss_i[o], j = a.ss_j[o];
            w = make_uint2(i | (a.ss_s14[o] ? 0x80000000u : 0u), j | 0x80000000u);
            // combine_lj_params (src/non_bonded.rs:1081-1086)
            lj = make_float2(__fmul_rn(0.5f, __fadd_rn(a.sig[i], a.sig[j])), __fsqrt_rn(__fmul_rn(a.eps[i], a.eps[j])));
            qq = __fmul_rn(a.q[i], a.q[j]);
        }
        pidx[o] = w;
        plj[o] = lj;
        pqq[o] = qq;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

template <typename T>
int dalloc(T** p, size_t n) {
    if (n == 0) n = 1;
    cudaError_t e = cudaMalloc((void**)p, n * sizeof(T));
    if (e != cudaSuccess) return dyn::cuda_fail(e, "cudaMalloc");
    return DYN_OK;
}
template <typename T>
int halloc(T** p, size_t n) {
    if (n == 0) n = 1;
    cudaError_t e = cudaMallocHost((void**)p, n * sizeof(T));
    if (e != cudaSuccess) return dyn::cuda_fail(e, "cudaMallocHost");
    return DYN_OK;
}

int ensure_pair_capacity(dyn_nb_s* h, uint64_t n) {
    if (n <= h->cap_pairs) return DYN_OK;
    cudaFree(h->d_pidx); cudaFree(h->d_plj); cudaFree(h->d_pqq);
    h->d_pidx = nullptr; h->d_plj = nullptr; h->d_pqq = nullptr; h->cap_pairs = 0;
    int rc;
    if ((rc = dalloc(&h->d_pidx, n)) || (rc = dalloc(&h->d_plj, n)) || (rc = dalloc(&h->d_pqq, n)))
        return rc;
    h->cap_pairs = n;
    return DYN_OK;
}

void build_csr(uint32_t n, uint64_t m, const uint32_t* pairs, std::vector<uint32_t>& off,
               std::vector<uint32_t>& idx) {
    // symmetric CSR of (i, j) pairs, each row sorted ascending
    std::vector<std::vector<uint32_t>> rows(n);
    for (uint64_t k = 0; k < m; ++k) {
        const uint32_t i = pairs[2 * k], j = pairs[2 * k + 1];
        if (i < n && j < n) { rows[i].push_back(j); rows[j].push_back(i); }
    }
    off.assign(n + 1, 0);
    idx.clear();
    for (uint32_t i = 0; i < n; ++i) {
        std::sort(rows[i].begin(), rows[i].end());
        rows[i].erase(std::unique(rows[i].begin(), rows[i].end()), rows[i].end());
        off[i + 1] = off[i] + (uint32_t)rows[i].size();
        idx.insert(idx.end(), rows[i].begin(), rows[i].end());
    }
}

// Whether the ten entries from o on are one water pair as setup_pairs writes
// it (emit_pairs_kernel): O-O with the water's LJ, then M, H0, H1 against M,
// H0, H1 with their charges, all symmetric.
bool is_water_pair(uint64_t o, const uint32_t* tgt, const uint32_t* src, const float* sigma, const float* eps,
                   const float* q_tgt, const float* q_src, const uint8_t* body_tgt, const uint8_t* body_src,
                   const uint8_t* flags) {
    const float q[3] = {OPC_Q_EP, OPC_Q_H, OPC_Q_H};
    for (uint32_t t = 0; t < 10; ++t) {
        const uint64_t p = o + t;
        const uint32_t s0 = t ? (t - 1) / 3u : 0u, s1 = t ? (t - 1) % 3u : 0u;
        if (tgt[p] != tgt[o] || src[p] != src[o] || body_tgt[p] != (t ? DYN_BODY_W_M + s0 : DYN_BODY_W_O) ||
            body_src[p] != (t ? DYN_BODY_W_M + s1 : DYN_BODY_W_O) ||
            flags[p] != (DYN_PAIR_SYMMETRIC | (t ? DYN_PAIR_COULOMB : DYN_PAIR_LJ)))
            return false;
        if (t ? q_tgt[p] * q_src[p] != q[s0] * q[s1] : sigma[p] != OPC_O_SIGMA || eps[p] != OPC_O_EPS) return false;
    }
    return true;
}

// Device memory of a handle that grows as calls need more and is kept.
int ensure(dyn_nb_s::Area& a, size_t bytes) {
    if (bytes <= a.cap) return DYN_OK;
    if (a.p) cudaFree(a.p);
    a.p = nullptr;
    a.cap = 0;
    const cudaError_t e = cudaMalloc((void**)&a.p, bytes);
    if (e != cudaSuccess) return dyn::cuda_fail(e, "cudaMalloc");
    a.cap = bytes;
    return DYN_OK;
}

// Takes n elements from an area laid out front to back (256-byte aligned);
// with base = nullptr only the size is counted.
template <typename T>
T* carve(char* base, size_t& used, size_t n) {
    T* p = base ? (T*)(base + used) : nullptr;
    used += (std::max<size_t>(n, 1) * sizeof(T) + 255) / 256 * 256;
    return p;
}

}  // namespace

extern "C" int dyn_nb_create(void* stream, uint32_t n_dyn, uint32_t n_water, float cutoff_ewald,
                             float alpha_ewald, float lj_cutoff, dyn_nb_t* out) {
    DYN_CHECK(out != nullptr, DYN_ERR_INVALID, "dyn_nb_create: out is NULL");
    DYN_CHECK(cutoff_ewald > 0.f && alpha_ewald > 0.f, DYN_ERR_INVALID,
              "dyn_nb_create: cutoff and alpha must be > 0");
    DYN_CHECK(n_dyn < (1u << 27) && n_water < (1u << 27), DYN_ERR_INVALID,
              "dyn_nb_create: fewer than 2^27 atoms / waters");
    *out = nullptr;
    dyn_nb_s* h = new dyn_nb_s();
    h->stream = (cudaStream_t)stream;
    h->n_dyn = n_dyn; h->n_water = n_water;
    h->rc = cutoff_ewald; h->alpha = alpha_ewald; h->ljc = lj_cutoff;
    int rc = DYN_OK;
    for (int a = 0; a < 5; ++a) {
        const size_t n3 = 3 * (size_t)h->n_of(a);
        h->off[a] = h->n_comp;
        h->n_comp += n3;
    }
    if (rc == DYN_OK) rc = dalloc(&h->d_pos, h->n_comp);
    if (rc == DYN_OK) rc = dalloc(&h->d_f, h->n_comp + NB_PART);
    if (rc == DYN_OK) rc = halloc(&h->h_pos, h->n_comp);
    if (rc == DYN_OK) rc = halloc(&h->h_f, h->n_comp + NB_PART);
    if (rc == DYN_OK) rc = dalloc(&h->d_sphere, n_water);
    if (rc == DYN_OK) rc = dalloc(&h->d_partials, 2 * NB_PART * NB_MAX_BLOCKS);
    if (rc != DYN_OK) {
        dyn_nb_destroy(h);
        return rc;
    }
    *out = h;
    return DYN_OK;
}

extern "C" int dyn_nb_destroy(dyn_nb_t h) {
    if (!h) return DYN_OK;
    if (h->stream) cudaStreamSynchronize(h->stream); else cudaDeviceSynchronize();
    cudaFree(h->d_pos); cudaFree(h->d_f);
    cudaFreeHost(h->h_pos); cudaFreeHost(h->h_f);
    cudaFree(h->d_sphere); cudaFree(h->d_partials);
    cudaFree(h->d_pidx); cudaFree(h->d_plj); cudaFree(h->d_pqq);
    cudaFree(h->scratch.p); cudaFree(h->lists.p);
    delete h;
    return DYN_OK;
}

extern "C" int dyn_nb_set_pairs(dyn_nb_t h, uint64_t n, const uint32_t* tgt, const uint32_t* src,
                                const float* sigma, const float* eps, const float* q_tgt,
                                const float* q_src, const uint8_t* body_tgt,
                                const uint8_t* body_src, const uint8_t* flags) {
    DYN_CHECK(h, DYN_ERR_INVALID, "dyn_nb_set_pairs: NULL handle");
    if (n > 0)
        DYN_CHECK(tgt && src && sigma && eps && q_tgt && q_src && body_tgt && body_src && flags,
                  DYN_ERR_INVALID, "dyn_nb_set_pairs: NULL array");
    for (uint64_t p = 0; p < n; ++p) {
        const uint32_t bt = body_tgt[p], bs = body_src[p];
        if (bt > 4 || bs > 4) return dyn::fail(DYN_ERR_INVALID, "dyn_nb_set_pairs: body code > 4");
        if (tgt[p] >= (bt ? h->n_water : h->n_dyn) || src[p] >= (bs ? h->n_water : h->n_dyn))
            return dyn::fail(DYN_ERR_INVALID, "dyn_nb_set_pairs: pair index out of range");
    }
    int rc = ensure_pair_capacity(h, n);
    if (rc) return rc;
    h->n_pairs = n;
    h->n_alch = 0;
    h->n_ww = 0;
    for (uint64_t p = 0; p < n; ++p) h->n_alch += (flags[p] & DYN_PAIR_ALCH) != 0;
    if (n == 0) return DYN_OK;
    // stage through temporary device buffers, then pack
    void* tmp = nullptr;
    const size_t bytes = n * (4 + 4 + 4 + 4 + 4 + 4 + 1 + 1 + 1);
    DYN_CUDA(cudaMalloc(&tmp, bytes));
    char* b = (char*)tmp;
    uint32_t* dt = (uint32_t*)b; b += 4 * n;
    uint32_t* ds = (uint32_t*)b; b += 4 * n;
    float* dsg = (float*)b; b += 4 * n;
    float* dep = (float*)b; b += 4 * n;
    float* dqt = (float*)b; b += 4 * n;
    float* dqs = (float*)b; b += 4 * n;
    uint8_t* dbt = (uint8_t*)b; b += n;
    uint8_t* dbs = (uint8_t*)b; b += n;
    uint8_t* dfl = (uint8_t*)b;
    cudaStream_t st = h->stream;
    cudaMemcpyAsync(dt, tgt, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(ds, src, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dsg, sigma, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dep, eps, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dqt, q_tgt, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dqs, q_src, 4 * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dbt, body_tgt, n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dbs, body_src, n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dfl, flags, n, cudaMemcpyHostToDevice, st);
    const int blocks = (int)std::min<uint64_t>((n + 255) / 256, 148 * 16);
    pack_pairs_kernel<<<blocks, 256, 0, st>>>(n, dt, ds, dsg, dep, dqt, dqs, dbt, dbs, dfl,
                                              h->d_pidx, h->d_plj, h->d_pqq);
    DYN_CUDA(cudaGetLastError());
    DYN_CUDA(cudaStreamSynchronize(st));
    cudaFree(tmp);
    // the water pairs a list in setup_pairs' order ends with are evaluated by
    // molecule, as those of a built list
    uint64_t nww = 0;
    while (10 * (nww + 1) <= n &&
           is_water_pair(n - 10 * (nww + 1), tgt, src, sigma, eps, q_tgt, q_src, body_tgt, body_src, flags))
        ++nww;
    if (nww) {
        std::vector<uint32_t> wi(nww), wj(nww);
        for (uint64_t k = 0; k < nww; ++k) {
            const uint64_t o = n - 10 * (nww - k);
            wi[k] = tgt[o];
            wj[k] = src[o];
        }
        uint32_t *di = nullptr, *dj = nullptr;
        auto lay = [&](char* base) {
            size_t u = 0;
            di = carve<uint32_t>(base, u, nww);
            dj = carve<uint32_t>(base, u, nww);
            return u;
        };
        if ((rc = ensure(h->lists, lay(nullptr))) != DYN_OK) return rc;
        lay(h->lists.p);
        DYN_CUDA(cudaMemcpyAsync(di, wi.data(), 4 * nww, cudaMemcpyHostToDevice, st));
        DYN_CUDA(cudaMemcpyAsync(dj, wj.data(), 4 * nww, cudaMemcpyHostToDevice, st));
        DYN_CUDA(cudaStreamSynchronize(st));
        h->d_wwi = di;
        h->d_wwj = dj;
        h->n_ww = nww;
    }
    return DYN_OK;
}

extern "C" int dyn_nb_get_pairs(dyn_nb_t h, uint64_t n, uint32_t* tgt, uint32_t* src,
                                float* sigma, float* eps, float* q_tgt, float* q_src,
                                uint8_t* body_tgt, uint8_t* body_src, uint8_t* flags) {
    DYN_CHECK(h, DYN_ERR_INVALID, "dyn_nb_get_pairs: NULL handle");
    DYN_CHECK(n <= h->n_pairs, DYN_ERR_INVALID, "dyn_nb_get_pairs: n exceeds installed pairs");
    if (n == 0) return DYN_OK;
    std::vector<uint2> idx(n);
    std::vector<float2> lj(n);
    std::vector<float> qq(n);
    cudaStream_t st = h->stream;
    DYN_CUDA(cudaMemcpyAsync(idx.data(), h->d_pidx, n * sizeof(uint2), cudaMemcpyDeviceToHost, st));
    DYN_CUDA(cudaMemcpyAsync(lj.data(), h->d_plj, n * sizeof(float2), cudaMemcpyDeviceToHost, st));
    DYN_CUDA(cudaMemcpyAsync(qq.data(), h->d_pqq, n * sizeof(float), cudaMemcpyDeviceToHost, st));
    DYN_CUDA(cudaStreamSynchronize(st));
    for (uint64_t p = 0; p < n; ++p) {
        const uint32_t bt = (idx[p].x >> 28) & 7u, bs = (idx[p].y >> 28) & 7u;
        if (tgt) tgt[p] = idx[p].x & TGT_MASK;
        if (src) src[p] = idx[p].y & IDX_MASK;
        if (body_tgt) body_tgt[p] = (uint8_t)bt;
        if (body_src) body_src[p] = (uint8_t)bs;
        if (sigma) sigma[p] = lj[p].x;
        if (eps) eps[p] = lj[p].y;
        if (q_tgt) q_tgt[p] = qq[p];   // the product q_t q_s is what is stored
        if (q_src) q_src[p] = 1.0f;
        if (flags) {
            uint8_t f = 0;
            if (idx[p].x >> 31) f |= DYN_PAIR_SCALE14;
            if (idx[p].y >> 31) f |= DYN_PAIR_SYMMETRIC;
            if (idx[p].x & ALCH_BIT) f |= DYN_PAIR_ALCH;
            if (lj[p].y != 0.f) f |= DYN_PAIR_LJ;
            // setup_pairs sets calc_coulomb for every pair but water O ones
            const bool o_t = bt == DYN_BODY_W_O, o_s = bs == DYN_BODY_W_O;
            if (!(o_t || o_s)) f |= DYN_PAIR_COULOMB;
            flags[p] = f;
        }
    }
    return DYN_OK;
}

extern "C" int dyn_nb_build_pairs(dyn_nb_t h, const float* pos_dyn, const float* pos_w_o,
                                  const float* atom_q, const float* atom_sigma,
                                  const float* atom_eps, const uint8_t* is_static,
                                  const uint8_t* bonded_only, uint64_t n_excl,
                                  const uint32_t* excl, uint64_t n_pair14, const uint32_t* pair14,
                                  const float box_lo[3], const float box_hi[3], float skin,
                                  uint64_t* n_pairs_out) {
    DYN_CHECK(h && box_lo && box_hi, DYN_ERR_INVALID, "dyn_nb_build_pairs: NULL argument");
    DYN_CHECK(h->n_dyn == 0 || (pos_dyn && atom_q && atom_sigma && atom_eps), DYN_ERR_INVALID,
              "dyn_nb_build_pairs: atom arrays required");
    DYN_CHECK(h->n_water == 0 || pos_w_o, DYN_ERR_INVALID, "dyn_nb_build_pairs: water O required");
    DYN_CHECK(skin >= 0.f, DYN_ERR_INVALID, "dyn_nb_build_pairs: skin < 0");
    const uint32_t ns = h->n_dyn, nw = h->n_water;
    cudaStream_t st = h->stream;
    // float32 exactly as the reference: extent = hi - lo, thr = (c+s)*(c+s)
    float ext_h[3], lo_h[3];
    for (int k = 0; k < 3; ++k) {
        lo_h[k] = box_lo[k];
        volatile float e = box_hi[k] - box_lo[k];
        ext_h[k] = e;
        DYN_CHECK(ext_h[k] > 0.f, DYN_ERR_INVALID, "dyn_nb_build_pairs: box extent must be > 0");
    }
    volatile float cs = h->rc + skin;
    const float thr = cs * cs;
    const float3 ext = make_float3(ext_h[0], ext_h[1], ext_h[2]);
    // exclusion / 1-4 CSR
    std::vector<uint32_t> ex_off, ex_idx, s_off, s_idx;
    build_csr(ns, n_excl, excl, ex_off, ex_idx);
    build_csr(ns, n_pair14, pair14, s_off, s_idx);
#define TRY(x) do { const int _r = (x); if (_r != DYN_OK) return _r; } while (0)
    // the inputs, packed on the host and copied in one go, then the rows'
    // counts and offsets
    struct Lay {
        float *atoms, *wo_raw, *q, *sig, *eps, *wo;
        uint32_t *exo, *exi, *so, *si, *cnt[3];
        uint8_t *st, *bonly;
        uint64_t *off[3], *total;
    } L{};
    const uint32_t rows[3] = {ns, ns, nw};
    auto lay = [&](char* base, size_t& in_bytes) {
        size_t u = 0;
        L.atoms = carve<float>(base, u, 3 * (size_t)ns);
        L.wo_raw = carve<float>(base, u, 3 * (size_t)nw);
        L.q = carve<float>(base, u, ns);
        L.sig = carve<float>(base, u, ns);
        L.eps = carve<float>(base, u, ns);
        L.exo = carve<uint32_t>(base, u, ex_off.size());
        L.exi = carve<uint32_t>(base, u, ex_idx.size());
        L.so = carve<uint32_t>(base, u, s_off.size());
        L.si = carve<uint32_t>(base, u, s_idx.size());
        L.st = carve<uint8_t>(base, u, ns);
        L.bonly = carve<uint8_t>(base, u, ns);
        in_bytes = u;
        L.wo = carve<float>(base, u, 3 * (size_t)nw);
        for (int k = 0; k < 3; ++k) L.cnt[k] = carve<uint32_t>(base, u, rows[k]);
        for (int k = 0; k < 3; ++k) L.off[k] = carve<uint64_t>(base, u, rows[k] + 1);
        L.total = carve<uint64_t>(base, u, 3);
        return u;
    };
    size_t in_bytes = 0;
    TRY(ensure(h->scratch, lay(nullptr, in_bytes)));
    std::vector<char> in(in_bytes);
    lay(in.data(), in_bytes);
    auto put = [](void* dst, const void* src, size_t n) { if (n && src) std::memcpy(dst, src, n); };
    put(L.atoms, pos_dyn, 12 * (size_t)ns);
    put(L.wo_raw, pos_w_o, 12 * (size_t)nw);
    put(L.q, atom_q, 4 * (size_t)ns);
    put(L.sig, atom_sigma, 4 * (size_t)ns);
    put(L.eps, atom_eps, 4 * (size_t)ns);
    put(L.exo, ex_off.data(), 4 * ex_off.size());
    put(L.exi, ex_idx.data(), 4 * ex_idx.size());
    put(L.so, s_off.data(), 4 * s_off.size());
    put(L.si, s_idx.data(), 4 * s_idx.size());
    put(L.st, is_static, ns);
    put(L.bonly, bonded_only, ns);
    lay(h->scratch.p, in_bytes);
    DYN_CUDA(cudaMemcpyAsync(h->scratch.p, in.data(), in_bytes, cudaMemcpyHostToDevice, st));
    if (nw) {
        wrap_o_kernel<<<(nw + 255) / 256, 256, 0, st>>>(nw, L.wo_raw, make_float3(lo_h[0], lo_h[1], lo_h[2]), ext, L.wo);
        DYN_CUDA(cudaGetLastError());
    }
    // std-std, std-water, water-water
    ListArgs la[3];
    for (int k = 0; k < 3; ++k) {
        la[k] = ListArgs{};
        la[k].thr = thr; la[k].ext = ext; la[k].mode = k;
        la[k].outer = k == 2 ? L.wo : L.atoms;
        la[k].inner = k == 0 ? L.atoms : L.wo;
        la[k].n_outer = rows[k];
        la[k].n_inner = k == 0 ? ns : nw;
    }
    la[0].is_static = is_static ? L.st : nullptr;
    la[0].bonded_only = bonded_only ? L.bonly : nullptr;
    la[0].ex_off = L.exo; la[0].ex_idx = L.exi; la[0].s14_off = L.so; la[0].s14_idx = L.si;
    const int threads = 256;
    auto blocks = [&](int k) { return (unsigned)(((uint64_t)rows[k] * 32 + threads - 1) / threads); };
    ScanArgs sa{};
    for (int k = 0; k < 3; ++k) {
        if (rows[k]) ref_list_kernel<0><<<blocks(k), threads, 0, st>>>(la[k], L.cnt[k], nullptr, nullptr, nullptr, nullptr);
        sa.cnt[k] = L.cnt[k]; sa.off[k] = L.off[k]; sa.n[k] = rows[k];
    }
    sa.total = L.total;
    scan_rows_kernel<<<3, SCAN_T, 0, st>>>(sa);
    DYN_CUDA(cudaGetLastError());
    uint64_t tot[3] = {};
    DYN_CUDA(cudaMemcpyAsync(tot, L.total, sizeof(tot), cudaMemcpyDeviceToHost, st));
    DYN_CUDA(cudaStreamSynchronize(st));
    const uint64_t total = tot[0] + 4 * tot[1] + 10 * tot[2];
    // nothing is installed while the list's memory is replaced
    h->n_pairs = 0;
    h->n_ww = 0;
    h->n_alch = 0;
    uint32_t *li[3], *lj[3];
    uint8_t* s14 = nullptr;
    auto lay_lists = [&](char* base) {
        size_t u = 0;
        for (int k = 0; k < 3; ++k) { li[k] = carve<uint32_t>(base, u, tot[k]); lj[k] = carve<uint32_t>(base, u, tot[k]); }
        s14 = carve<uint8_t>(base, u, tot[0]);
        return u;
    };
    TRY(ensure(h->lists, lay_lists(nullptr)));
    lay_lists(h->lists.p);
    TRY(ensure_pair_capacity(h, total));
    for (int k = 0; k < 3; ++k)
        if (rows[k])
            ref_list_kernel<1><<<blocks(k), threads, 0, st>>>(la[k], nullptr, L.off[k], li[k], lj[k], k == 0 ? s14 : nullptr);
    EmitArgs ea{};
    ea.n_ss = tot[0]; ea.n_sw = tot[1]; ea.n_ww = tot[2];
    ea.ss_i = li[0]; ea.ss_j = lj[0]; ea.ss_s14 = s14;
    ea.sw_i = li[1]; ea.sw_j = lj[1];
    ea.ww_i = li[2]; ea.ww_j = lj[2];
    ea.q = L.q; ea.sig = L.sig; ea.eps = L.eps;
    if (total) {
        const int eb = (int)std::min<uint64_t>((total + NB_BLOCK - 1) / NB_BLOCK, 148 * 16);
        emit_pairs_kernel<<<eb, NB_BLOCK, 0, st>>>(ea, h->d_pidx, h->d_plj, h->d_pqq);
    }
    DYN_CUDA(cudaGetLastError());
    DYN_CUDA(cudaStreamSynchronize(st));
    h->n_pairs = total;
    h->n_ww = tot[2];
    h->d_wwi = li[2];
    h->d_wwj = lj[2];
    if (n_pairs_out) *n_pairs_out = total;
#undef TRY
    return DYN_OK;
}

namespace {

int nb_forces(dyn_nb_t h, const float* pos_dyn, const float* pos_w_o,
                             const float* pos_w_m, const float* pos_w_h0, const float* pos_w_h1,
                             const float cell_extent[3], uint32_t override_bits, double* f_dyn,
                             double* f_w_o, double* f_w_m, double* f_w_h0, double* f_w_h1,
                             double* virial, double* energy, double lambda, double* dh_dl) {
    DYN_CHECK(h && cell_extent, DYN_ERR_INVALID, "dyn_nb_forces: NULL argument");
    const float* in[5] = {pos_dyn, pos_w_o, pos_w_m, pos_w_h0, pos_w_h1};
    double* outp[5] = {f_dyn, f_w_o, f_w_m, f_w_h0, f_w_h1};
    for (int a = 0; a < 5; ++a)
        if (h->n_of(a) > 0)
            DYN_CHECK(in[a] != nullptr, DYN_ERR_INVALID, "dyn_nb_forces: NULL position array");
    for (int k = 0; k < 3; ++k)
        DYN_CHECK(cell_extent[k] > 0.f, DYN_ERR_INVALID, "dyn_nb_forces: extent must be > 0");
    cudaStream_t st = h->stream;
    // upload_positions (src/gpu_interface.rs:414-455) via pinned staging
    for (int a = 0; a < 5; ++a) {
        const size_t n3 = 3 * (size_t)h->n_of(a);
        if (!n3) continue;
        std::memcpy(h->h_pos + h->off[a], in[a], n3 * sizeof(float));
    }
    if (h->n_comp)
        DYN_CUDA(cudaMemcpyAsync(h->d_pos, h->h_pos, h->n_comp * sizeof(float), cudaMemcpyHostToDevice, st));
    // zero_forces_and_accums (src/gpu_interface.rs:635-645)
    DYN_CUDA(cudaMemsetAsync(h->d_f, 0, (h->n_comp + NB_PART) * sizeof(long long), st));
    const float3 ext = make_float3(cell_extent[0], cell_extent[1], cell_extent[2]);
    // the reference computes the reciprocal extent on the host in float32
    const float3 inv_ext = make_float3(1.0f / ext.x, 1.0f / ext.y, 1.0f / ext.z);
    // the flat entries but the water pairs of a built list, which are taken
    // by molecule
    const uint64_t n_flat = h->n_pairs - 10 * h->n_ww;
    auto nblk = [](uint64_t n) {
        return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + NB_BLOCK - 1) / NB_BLOCK, NB_MAX_BLOCKS));
    };
    const int blocks = nblk(n_flat);
    PosPtrs pp;
    ForcePtrs fp;
    for (int a = 0; a < 5; ++a) { pp.p[a] = h->d_pos + h->off[a]; fp.f[a] = h->d_f + h->off[a]; }
    PairConsts pc{};
    pc.ext = ext;
    pc.inv_ext = inv_ext;
    pc.half = make_float3(0.4999f * ext.x, 0.4999f * ext.y, 0.4999f * ext.z);
    pc.rc = h->rc; pc.alpha = h->alpha; pc.ljc = h->ljc;
    pc.ovr = override_bits;
    // the alchemical kernel runs when any installed pair is alchemical, as
    // force_nonbonded_gpu picks it (src/gpu_interface.rs:488-499)
    const AlchSched al = alch_schedule(lambda);
    const bool cpu = h->ljc > 0.f, alch = h->n_alch > 0;
    auto kern = cpu ? (alch ? nb_pair_kernel<true, true> : nb_pair_kernel<true, false>)
                    : (alch ? nb_pair_kernel<false, true> : nb_pair_kernel<false, false>);
    kern<<<blocks, NB_BLOCK, 0, st>>>(pp, fp, h->d_pidx, h->d_plj, h->d_pqq, n_flat, pc, al, h->d_partials);
    DYN_CUDA(cudaGetLastError());
    int all_blocks = blocks;
    if (h->n_ww) {
        const uint32_t run = ww_run(h->n_ww);
        const int wb = nblk((h->n_ww + run - 1) / run);
        auto wk = cpu ? nb_ww_kernel<true> : nb_ww_kernel<false>;
        if (cpu)
            nb_sphere_kernel<<<nblk(h->n_water), NB_BLOCK, 0, st>>>(pp, h->n_water, ext, h->d_sphere);
        wk<<<wb, NB_BLOCK, 0, st>>>(pp, fp, h->d_wwi, h->d_wwj, h->n_ww, run, h->d_sphere, pc,
                                      h->d_partials + (size_t)NB_PART * blocks);
        DYN_CUDA(cudaGetLastError());
        all_blocks += wb;
    }
    const int fb = 1 + (int)std::min<size_t>((h->n_comp + 255) / 256, 148 * 8);
    nb_finalize_kernel<<<fb, 256, 0, st>>>(h->d_partials, all_blocks, h->d_f, (uint32_t)h->n_comp);
    DYN_CUDA(cudaGetLastError());
    DYN_CUDA(cudaMemcpyAsync(h->h_f, h->d_f, (h->n_comp + NB_PART) * sizeof(double), cudaMemcpyDeviceToHost, st));
    DYN_CUDA(cudaStreamSynchronize(st));
    for (int a = 0; a < 5; ++a) {
        const size_t n3 = 3 * (size_t)h->n_of(a);
        if (outp[a] && n3) std::memcpy(outp[a], h->h_f + h->off[a], n3 * sizeof(double));
    }
    const double* sums = h->h_f + h->n_comp;
    if (virial) *virial = sums[0];
    if (energy) *energy = sums[1];
    if (dh_dl) *dh_dl = alch ? sums[2] : 0.0;
    return DYN_OK;
}

}  // namespace

extern "C" int dyn_nb_forces(dyn_nb_t h, const float* pos_dyn, const float* pos_w_o,
                             const float* pos_w_m, const float* pos_w_h0, const float* pos_w_h1,
                             const float cell_extent[3], uint32_t override_bits, double* f_dyn,
                             double* f_w_o, double* f_w_m, double* f_w_h0, double* f_w_h1,
                             double* virial, double* energy) {
    return nb_forces(h, pos_dyn, pos_w_o, pos_w_m, pos_w_h0, pos_w_h1, cell_extent, override_bits,
                     f_dyn, f_w_o, f_w_m, f_w_h0, f_w_h1, virial, energy, 0.0, nullptr);
}

extern "C" int dyn_nb_forces_alch(dyn_nb_t h, const float* pos_dyn, const float* pos_w_o,
                                  const float* pos_w_m, const float* pos_w_h0,
                                  const float* pos_w_h1, const float cell_extent[3],
                                  uint32_t override_bits, double lambda_alch, double* f_dyn,
                                  double* f_w_o, double* f_w_m, double* f_w_h0, double* f_w_h1,
                                  double* virial, double* energy, double* dh_dl) {
    DYN_CHECK(std::isfinite(lambda_alch), DYN_ERR_INVALID, "dyn_nb_forces_alch: lambda is not finite");
    return nb_forces(h, pos_dyn, pos_w_o, pos_w_m, pos_w_h0, pos_w_h1, cell_extent, override_bits,
                     f_dyn, f_w_o, f_w_m, f_w_h0, f_w_h1, virial, energy, lambda_alch, dh_dl);
}

extern "C" int dyn_nb_mark_alch(dyn_nb_t h, uint32_t atom_begin, uint32_t atom_end,
                                uint64_t* n_marked) {
    DYN_CHECK(h, DYN_ERR_INVALID, "dyn_nb_mark_alch: NULL handle");
    DYN_CHECK(atom_begin <= atom_end && atom_end <= h->n_dyn, DYN_ERR_INVALID,
              "dyn_nb_mark_alch: range outside the atoms");
    cudaStream_t st = h->stream;
    unsigned long long* d_cnt = nullptr;
    DYN_CUDA(cudaMalloc(&d_cnt, sizeof(unsigned long long)));
    cudaError_t e = cudaMemsetAsync(d_cnt, 0, sizeof(unsigned long long), st);
    if (e == cudaSuccess && h->n_pairs) {
        const int blocks = (int)std::min<uint64_t>((h->n_pairs + 255) / 256, 148 * 8);
        mark_alch_kernel<<<blocks, 256, 0, st>>>(h->n_pairs, atom_begin, atom_end, h->d_pidx, d_cnt);
        e = cudaGetLastError();
    }
    unsigned long long c = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&c, d_cnt, sizeof(c), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_cnt);
    if (e != cudaSuccess) return dyn::cuda_fail(e, "dyn_nb_mark_alch");
    h->n_alch = c;
    if (n_marked) *n_marked = c;
    return DYN_OK;
}
