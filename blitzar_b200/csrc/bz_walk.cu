// Warp-cooperative group tree walk (the force hot path).
//
// One warp owns a group of at most 32 consecutive Morton-sorted targets (a run of sibling
// subtrees cut from the octree, bz_groups.cu).  It walks the tree once for the whole group: each
// step takes the children of the four nodes opened last (one per lane), tests them against the
// group's bounding box, and sorts them with warp votes into
//   - pruned (beyond the short-range cutoff),
//   - accepted multipoles  -> appended to a shared-memory node list,
//   - leaves to sum directly -> appended to a shared-memory leaf list,
//   - opened internal nodes -> pushed on a shared-memory stack as (first child, child count),
//     placed by a vote (pushing the children themselves took a shuffle scan and a loop).
// Full lists are flushed: the lanes share the evaluation of every target against each listed
// node (LaneMap), and leaf particles are pulled into a shared-memory tile with cp.async.bulk
// (global -> shared, completing on an mbarrier, into this CTA only) and summed with FP32 pair
// arithmetic.  Per-flush partial sums are folded into the running force with a two-sum
// (compensated accumulation).
//
// Decisions are computed with round-to-nearest intrinsics (no contraction) so that the set
// of accepted nodes and direct leaves is bit-identical to the oracle's; the reference's
// per-particle stackless walk is engine/physics/octree/cuda/force/OctGpu.inl:100-228 and the
// TreePM pair law with the Gaussian split is engine/physics/core/cuda/prelude/
// CudForceKernels.inl:62-89.
#include "bz_common.cuh"
#include "bz_kernels.h"

#include <cuda_fp16.h>

#include <type_traits>

namespace bz {

namespace {

constexpr int kWarps = 4;
constexpr int kStack = 128;       // shared-memory part of the traversal stack
constexpr int kSpill = 8192;      // per-warp global spill area (oldest entries)
constexpr int kList = 64;         // leaf list
constexpr int kNodes = 128;       // accepted nodes evaluated per flush
constexpr int kTile = 128;        // staged leaf particles
// ... of a walk that only filters, where a lane sums the sources inside its own cutoff and a tile
// takes as long as the lane with the most of them: 1.86 times the mean over 128 sources, 1.35 times
// over 256 (256^3 walk 7.0 -> 6.45 ms).  A flush falls due early enough that most fit one tile (192
// listed: 6.45, 256: 6.53).
constexpr int kFilterTile = 256;
constexpr int kFilterFlush = 192;
constexpr int kMaskPitch = 40;  // a target's word q lies 8 banks past its word q - 1
constexpr int kFlushParticles = 256;  // listed leaf particles that trigger a flush
constexpr int kIndexBits = 26;
constexpr int kIndexMask = (1 << kIndexBits) - 1;
constexpr int kPerPairImage = 64;  // leaf code: periodic image chosen per pair

constexpr int kNoShift = 21;       // shift code of the central image on all three axes

template <bool QUAD, bool FILTER> struct __align__(16) WarpSmem {
    static constexpr int kSources = FILTER ? kFilterTile : kTile;
    // a leaf flush and a node flush never overlap: they share their staging area
    union {
        struct {
            float4 tile[kSources];
            unsigned mask[kSources / 32 + 1][kMaskPitch];  // per-lane in-cutoff bits of the tile
            uint4 brow[FILTER ? 32 : 1];  // cutoff filter: FP16 rows of 32 of the tile's sources
        };
        struct {
            // accepted nodes, two to an entry so that packed FP32 instructions take both:
            // {x x y y}, {z z m m}, {xx xx xy xy}, {xz xz yy yy}, {yz yz zz zz}
            float4 nd[QUAD ? 5 : 2][kNodes / 2];
            float2 nd_tr[QUAD ? kNodes / 2 : 1];  // tr(Q) eps^2 (Newtonian) or -tr(Q) / 2 (split)
        };
    };
    uint4 arow[FILTER ? 32 : 1];  // cutoff filter: FP16 rows of the targets
    float4 frame;     // ... centre of the group, scale (0: too wide for FP16, scalar filter)
    float4 tgt[32];   // the group's targets (slots past its size repeat the first)
    // sorted index of each tile source (potentials, pairs recorded); FILTER: its list entry
    std::conditional_t<FILTER, unsigned char, int> tidx[kSources];
    unsigned stack[kStack];  // opened nodes: first child | (children - 1) << kIndexBits
    int nlist[kNodes + 32];
    int lstart[kList];
    int lcount[kList];
    unsigned char lcode[kList];
    union {
        int lnode[kList];
        int lpre[kList];  // particles listed before the entry (once the nodes have been looked at)
    };
    unsigned long long bar;
};

// How the 32 lanes share the evaluation of a group's gn targets against a staged list of
// sources or nodes: lane = slice x T + slot with T target slots and S = 32 / T slices.  A lane
// takes every S-th entry of the list for the targets slot, slot + T, ... (kChunk of them at a
// time, so that one shared-memory read of an entry serves kChunk interactions), and the
// slices' sums are combined once a flush.  With one target a lane instead, groups of fewer than
// 32 targets leave lanes idle on every entry, and groups cut from an octree hold 18 (Plummer
// 65k) to 23 (Hernquist 4M) of 32 on average, mostly a single particle in the outskirts of a
// small system (1272 of the 1423 groups of Plummer 4096).  T = 4 rounds gn up to a multiple of 4.
//
// The kernel is bound by the issue and the FP32 pipe (Hernquist 1M: DRAM idle, FMA pipes 60 %
// busy).  Measured per walk, one target a lane -> this mapping with two nodes or sources in
// each packed FP32 instruction, 128 nodes a flush, and opened nodes instead of children on the
// stack: Plummer 4096 0.233 -> 0.103 ms, Plummer 65k 0.64 -> 0.39 ms, Hernquist 4M 49.7 -> 36.4
// ms, an adaptive ensemble substep of 96 clusters 1.12 -> 0.58 ms on average, isolated TreePM of
// 1M (with the leaves wholly inside the cutoff summed without the filter) 6.87 -> 4.37 ms.  Four targets a
// chunk (more code than the instruction cache holds: 42.6 ms at 4M) and scalar instructions
// (40.0 ms) were slower.
constexpr int kSlots = 4;
constexpr int kChunk = 2;

struct LaneMap {
    int slot, slice, nslices, rows;  // rows: targets a slot serves
    __device__ LaneMap(int gn, bool sliced)
    {
        const int lane = threadIdx.x & 31;
        // log2 of the slots: 1 or 2 targets take as many, more take kSlots; a (nearly) full group
        // has no lanes to win and takes one target a lane, which needs no sums over slices
        // (all-full lattice groups, 128^3 CIC TreePM: 2.26 ms against 2.84; Hernquist 4M 36.4
        // against 36.7)
        const int sh = !sliced || gn > 28 ? 5 : (gn < 3 ? gn - 1 : 2);
        slot = lane & ((1 << sh) - 1);
        slice = lane >> sh;
        nslices = 32 >> sh;
        rows = sh == 2 ? (gn + kSlots - 1) / kSlots : 1;
    }
};

// erfc(u) ~= t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) e^{-u^2},  t = 1/(1 + p u)
// (Abramowitz & Stegun 7.1.26, |error| <= 1.5e-7).
__device__ __forceinline__ float erfc_as(float u, float e)
{
    const float t = rcp_approx(fmaf(0.3275911f, u, 1.0f));
    float p = 1.061405429f;
    p = fmaf(p, t, -1.453152027f);
    p = fmaf(p, t, 1.421413741f);
    p = fmaf(p, t, -0.284496736f);
    p = fmaf(p, t, 0.254829592f);
    return t * p * e;
}

constexpr float kTwoOverSqrtPi = 1.1283791670955126f;
constexpr float kFourOverSqrtPi = 2.2567583341910252f;
constexpr float kEightOverSqrtPi = 4.5135166683820503f;

struct SplitK {
    float inv2rs;  // 1 / (2 r_s)
    float cexp;    // -log2(e) / (4 r_s^2): e^{-u^2} = 2^{s^2 cexp}
    float pk;      // 0.3275911 / (2 r_s): A&S t = 1 / (1 + p u)
    float c2;      // (2/sqrt(pi)) / (2 r_s): 2u/sqrt(pi) = s c2
};

__device__ __forceinline__ float ex2_approx(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two FP32 values in one 64-bit register pair: one packed instruction does both.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float lo(F2 a)
{
    return __uint_as_float(static_cast<unsigned>(a.v));
}
__device__ __forceinline__ float hi(F2 a)
{
    return __uint_as_float(static_cast<unsigned>(a.v >> 32));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 rsqrt2(F2 a) { return f2(rsqrt_approx(lo(a)), rsqrt_approx(hi(a))); }

template <bool SPLIT, bool POT>
__device__ __forceinline__ void pair_pp(const float4 s, float tx, float ty, float tz,
                                        const WalkParams& p, float inv2rs, bool cut, bool self,
                                        float& fx, float& fy, float& fz, float& fp)
{
    const float dx = s.x - tx, dy = s.y - ty, dz = s.z - tz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float s2 = r2 + p.eps2;
    float m = s.w;
    if (cut && r2 > p.rcut2)
        m = 0.0f;
    float rinv = rsqrt_approx(s2);
    if (s2 <= p.min_dist2) {
        m = 0.0f;
        rinv = 0.0f;
    }
    const float rinv2 = rinv * rinv;
    float f = m * rinv * rinv2;
    if (SPLIT) {
        const float u = s2 * rinv * inv2rs;
        const float e = __expf(-u * u);
        const float ec = erfc_as(u, e);
        const float w = fmaf(kTwoOverSqrtPi * u, e, ec);
        f *= w;
        if (POT && !self)
            fp = fmaf(-m * ec, rinv, fp);
    } else {
        if (POT && !self)
            fp = fmaf(-m, rinv, fp);
    }
    fx = fmaf(f, dx, fx);
    fy = fmaf(f, dy, fy);
    fz = fmaf(f, dz, fz);
}

// Force-only pair for softening above the minimum-distance floor (no zero-distance guard
// needed): the split weight w = e^{-u^2} (t P(t) + 2u/sqrt(pi)) with the A&S 7.1.26 erfc and
// all scale factors folded into precomputed constants.
// Returns 1 when the pair lies inside the cutoff (or no cutoff is applied), else 0.
template <bool SPLIT>
__device__ __forceinline__ unsigned pair_fast(const float4 s, float tx, float ty, float tz, float eps2,
                                              float rcut2, bool cut, const SplitK& k, float& fx,
                                              float& fy, float& fz)
{
    const float dx = s.x - tx, dy = s.y - ty, dz = s.z - tz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float s2 = r2 + eps2;
    const bool outside = cut && r2 > rcut2;
    const float m = outside ? 0.0f : s.w;
    const float rinv = rsqrt_approx(s2);
    float mw = m;
    if (SPLIT) {
        const float sd = s2 * rinv;
        const float e = ex2_approx(s2 * k.cexp);
        const float t = rcp_approx(fmaf(sd, k.pk, 1.0f));
        float q = 1.061405429f;
        q = fmaf(q, t, -1.453152027f);
        q = fmaf(q, t, 1.421413741f);
        q = fmaf(q, t, -0.284496736f);
        q = fmaf(q, t, 0.254829592f);
        mw = m * (e * fmaf(t, q, sd * k.c2));
    }
    const float f = mw * (rinv * rinv * rinv);
    fx = fmaf(f, dx, fx);
    fy = fmaf(f, dy, fy);
    fz = fmaf(f, dz, fz);
    return outside ? 0u : 1u;
}

template <bool SPLIT, bool QUAD, bool POT>
__device__ __forceinline__ void pair_pn(const float4 mo, const float4 qa, const float2 qb,
                                        float tx, float ty, float tz, const WalkParams& p,
                                        float inv2rs, float& fx, float& fy, float& fz, float& fp)
{
    const float dx = mo.x - tx, dy = mo.y - ty, dz = mo.z - tz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float s2 = r2 + p.eps2;
    float rinv = rsqrt_approx(s2);
    float m = mo.w;
    if (s2 <= p.min_dist2) {
        rinv = 0.0f;
        m = 0.0f;
    }
    const float rinv2 = rinv * rinv;
    float D0, D1, D2 = 0.0f, D3 = 0.0f;
    if (SPLIT) {
        const float u = s2 * rinv * inv2rs;
        const float e = __expf(-u * u);
        const float ec = erfc_as(u, e);
        const float h = fmaf(kTwoOverSqrtPi * u, e, ec);
        D0 = ec * rinv;
        D1 = h * rinv * rinv2;
        if (QUAD) {
            const float u2 = u * u;
            const float k = fmaf(kFourOverSqrtPi * u2 * u, e, 3.0f * h);
            const float l = fmaf(kEightOverSqrtPi * u2 * u2 * u, e, 5.0f * k);
            D2 = k * rinv2 * rinv2 * rinv;
            D3 = l * rinv2 * rinv2 * rinv2 * rinv;
        }
    } else {
        D0 = rinv;
        D1 = rinv * rinv2;
        if (QUAD) {
            D2 = 3.0f * D1 * rinv2;
            D3 = 5.0f * D2 * rinv2;
        }
    }
    float c0 = m * D1;
    if (QUAD) {
        const float qdx = fmaf(qa.x, dx, fmaf(qa.y, dy, qa.z * dz));
        const float qdy = fmaf(qa.y, dx, fmaf(qa.w, dy, qb.x * dz));
        const float qdz = fmaf(qa.z, dx, fmaf(qb.x, dy, qb.y * dz));
        const float dqd = fmaf(dx, qdx, fmaf(dy, qdy, dz * qdz));
        const float tr = qa.x + qa.w + qb.y;
        if (m == 0.0f) {
            D1 = D2 = D3 = 0.0f;
        }
        c0 = fmaf(0.5f * D3, dqd, fmaf(-0.5f * D2, tr, c0));
        fx = fmaf(c0, dx, fmaf(-D2, qdx, fx));
        fy = fmaf(c0, dy, fmaf(-D2, qdy, fy));
        fz = fmaf(c0, dz, fmaf(-D2, qdz, fz));
        if (POT)
            fp += fmaf(-m, D0, fmaf(0.5f * D1, tr, -0.5f * D2 * dqd));
    } else {
        fx = fmaf(c0, dx, fx);
        fy = fmaf(c0, dy, fy);
        fz = fmaf(c0, dz, fz);
        if (POT)
            fp = fmaf(-m, D0, fp);
    }
}

// Force-only Newtonian quadrupole interaction of two nodes at a time, with the traceless second
// moment Q' = Q - tr(Q)/3 I.  With softening the trace does not drop out of the expansion; written
// with Q' the acceleration is (m/s^3 + 15/2 (dQ'd + trm)/s^7) d - 3 Q'd/s^5 with s^2 = r^2 + eps^2
// and trm = -tr(Q) eps^2/3, algebraically the same as the traceful form (the m/s^3 + (15/2 dQd/s^7 -
// 3/2 tr/s^5)) d - 3 Qd/s^5 of pair_pn).  Used only when eps^2 exceeds the minimum distance^2,
// so the minimum-distance guard of pair_pn can never trigger.
// The potential's expansion collapses the same way: -m/s - 3/2 (dQ'd + trm)/s^5, negated in np.
// nx, ny, nz: the target's negated position; q = -3 Q' (xx xy xz yy yz zz), trm scaled by -3 too.
template <bool POT>
__device__ __forceinline__ void pair_pn_newton2(F2 x, F2 y, F2 z, F2 m, const F2* q, F2 trm, F2 nx,
                                                F2 ny, F2 nz, F2 eps2, F2& fx, F2& fy, F2& fz, F2& np)
{
    const F2 dx = add2(x, nx), dy = add2(y, ny), dz = add2(z, nz);
    const F2 rinv = rsqrt2(fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2))));
    const F2 a = mul2(rinv, rinv);  // 1/r^2
    const F2 b = mul2(rinv, a);     // 1/r^3
    const F2 t5 = mul2(b, a);       // 1/r^5
    const F2 qx = fma2(q[0], dx, fma2(q[1], dy, mul2(q[2], dz)));
    const F2 qy = fma2(q[1], dx, fma2(q[3], dy, mul2(q[4], dz)));
    const F2 qz = fma2(q[2], dx, fma2(q[4], dy, mul2(q[5], dz)));
    const F2 dqd = fma2(dx, qx, fma2(dy, qy, fma2(dz, qz, trm)));
    const F2 c0 = mul2(b, fma2(mul2(a, mul2(a, dqd)), f2(-2.5f), m));
    fx = fma2(c0, dx, fma2(t5, qx, fx));
    fy = fma2(c0, dy, fma2(t5, qy, fy));
    fz = fma2(c0, dz, fma2(t5, qz, fz));
    if (POT)
        np = fma2(m, rinv, fma2(mul2(t5, f2(-0.5f)), dqd, np));
}

// Force-only quadrupole interaction with the split kernel of two nodes at a time, softening above
// the minimum-distance floor.  pair_pn's expansion with its powers of 1/s factored out:
//   f = b (m h + a (l a dQd / 2 - k tr / 2)) d - k a b Q d,   a = 1/s^2, b = 1/s^3.
// nx, ny, nz: the target's negated position; q = -Q (xx xy xz yy yz zz), htr = -tr(Q) / 2.
__device__ __forceinline__ void pair_pn_split2(F2 x, F2 y, F2 z, F2 m, const F2* q, F2 htr, F2 nx, F2 ny,
                                               F2 nz, F2 eps2, float inv2rs, F2& fx, F2& fy, F2& fz)
{
    const F2 dx = add2(x, nx), dy = add2(y, ny), dz = add2(z, nz);
    const F2 s2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2)));
    const F2 rinv = rsqrt2(s2);
    const F2 a = mul2(rinv, rinv);
    const F2 b = mul2(rinv, a);
    const F2 u = mul2(mul2(s2, rinv), f2(inv2rs));
    const F2 u2 = mul2(u, u);
    const F2 g = mul2(u2, f2(-1.4426950408889634f));
    const F2 e = f2(ex2_approx(lo(g)), ex2_approx(hi(g)));
    const F2 v = fma2(u, f2(0.3275911f), f2(1.0f));
    const F2 t = f2(rcp_approx(lo(v)), rcp_approx(hi(v)));
    F2 ec = f2(1.061405429f);
    ec = fma2(ec, t, f2(-1.453152027f));
    ec = fma2(ec, t, f2(1.421413741f));
    ec = fma2(ec, t, f2(-0.284496736f));
    ec = fma2(ec, t, f2(0.254829592f));
    ec = mul2(mul2(ec, t), e);
    const F2 w1 = mul2(u, e), w3 = mul2(u2, w1), w5 = mul2(u2, w3);
    const F2 h = fma2(w1, f2(kTwoOverSqrtPi), ec);
    const F2 k = fma2(w3, f2(kFourOverSqrtPi), mul2(h, f2(3.0f)));
    const F2 nl = fma2(w5, f2(-0.5f * kEightOverSqrtPi), mul2(k, f2(-2.5f)));  // -l / 2
    const F2 qx = fma2(q[0], dx, fma2(q[1], dy, mul2(q[2], dz)));
    const F2 qy = fma2(q[1], dx, fma2(q[3], dy, mul2(q[4], dz)));
    const F2 qz = fma2(q[2], dx, fma2(q[4], dy, mul2(q[5], dz)));
    const F2 dqd = fma2(dx, qx, fma2(dy, qy, mul2(dz, qz)));
    const F2 c0 = mul2(b, fma2(a, fma2(mul2(nl, a), dqd, mul2(k, htr)), mul2(m, h)));
    const F2 c2 = mul2(k, mul2(a, b));
    fx = fma2(c0, dx, fma2(c2, qx, fx));
    fy = fma2(c0, dy, fma2(c2, qy, fy));
    fz = fma2(c0, dz, fma2(c2, qz, fz));
}

// As pair_fast without a cutoff, for two sources at a time; POT: np collects mp / s, mp the masses
// that count for the potential (not the target's own).
template <bool SPLIT, bool POT>
__device__ __forceinline__ void pair_fast2(F2 x, F2 y, F2 z, F2 m, F2 mp, F2 nx, F2 ny, F2 nz, F2 eps2,
                                           const SplitK& k, F2& fx, F2& fy, F2& fz, F2& np)
{
    const F2 dx = add2(x, nx), dy = add2(y, ny), dz = add2(z, nz);
    const F2 s2 = add2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))), eps2);
    const F2 rinv = rsqrt2(s2);
    F2 mw = m;
    if (SPLIT) {
        const F2 sd = mul2(s2, rinv);
        const F2 g = mul2(s2, f2(k.cexp));
        const F2 e = f2(ex2_approx(lo(g)), ex2_approx(hi(g)));
        const F2 u = fma2(sd, f2(k.pk), f2(1.0f));
        const F2 t = f2(rcp_approx(lo(u)), rcp_approx(hi(u)));
        F2 q = f2(1.061405429f);
        q = fma2(q, t, f2(-1.453152027f));
        q = fma2(q, t, f2(1.421413741f));
        q = fma2(q, t, f2(-0.284496736f));
        q = fma2(q, t, f2(0.254829592f));
        mw = mul2(m, mul2(e, fma2(t, q, mul2(sd, f2(k.c2)))));
    }
    const F2 f = mul2(mw, mul2(rinv, mul2(rinv, rinv)));
    fx = fma2(f, dx, fx);
    fy = fma2(f, dy, fy);
    fz = fma2(f, dz, fz);
    if (POT)
        np = fma2(mp, rinv, np);
}

struct Acc {
    float s[4];
    float e[4];
    __device__ void zero()
    {
        for (int i = 0; i < 4; ++i)
            s[i] = e[i] = 0.0f;
    }
    __device__ void add(int i, float v)
    {
        float ss, ee;
        two_sum(s[i], v, ss, ee);
        s[i] = ss;
        e[i] += ee;
    }
    __device__ float total(int i) const { return s[i] + e[i]; }
};

template <int N> struct IntC {
    static constexpr int value = N;
};

__device__ __forceinline__ float shift_of(int code, int axis, float box)
{
    return box * static_cast<float>(((code >> (2 * axis)) & 3) - 1);
}

// Sums of one pass over a staged list: R targets of this lane's slot, C components.
template <int R, int C> struct Rows {
    float tx[R], ty[R], tz[R], f[C][R];
    template <class W> __device__ __forceinline__ void load(const W& w, const LaneMap& lm, int row0)
    {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const float4 t = w.tgt[lm.slot + kSlots * (row0 + k)];
            tx[k] = t.x;
            ty[k] = t.y;
            tz[k] = t.z;
#pragma unroll
            for (int c = 0; c < C; ++c)
                f[c][k] = 0.0f;
        }
    }
    // Adds the slices' sums; lane j = slice * slots + slot adds those of target j to acc.  (Two
    // rows only go with kSlots slots, a single one with any number.)
    __device__ __forceinline__ void fold(const LaneMap& lm, int row0, Acc& acc)
    {
        if constexpr (R == 2) {
            // the first exchange leaves a lane with the row of its slice's parity
            const bool odd = lm.slice & 1;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                float v = (odd ? f[c][1] : f[c][0]) +
                          __shfl_xor_sync(kFullMask, odd ? f[c][0] : f[c][1], kSlots);
                v += __shfl_xor_sync(kFullMask, v, 2 * kSlots);
                v += __shfl_xor_sync(kFullMask, v, 4 * kSlots);
                acc.add(c, (lm.slice & ~1) == row0 ? v : 0.0f);
            }
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                float v = f[c][0];
                for (int o = 16; o >= 32 / lm.nslices; o >>= 1)
                    v += __shfl_xor_sync(kFullMask, v, o);
                acc.add(c, lm.slice == row0 ? v : 0.0f);
            }
        }
    }
};

// The walks that slice: all but the short-range walk without quadrupoles (a node-size cap or
// multipole_order 1), which the per-lane cutoff filter dominates: its few node terms do not pay
// for the registers of the chunks.
template <bool SPLIT, bool QUAD> constexpr bool walk_sliced() { return !SPLIT || QUAD; }
// Walks whose leaves all go through the cutoff filter (in larger tiles, on the tensor cores).
template <bool SPLIT, bool QUAD, bool POT> constexpr bool walk_filters() { return SPLIT && !QUAD && !POT; }

// Calls body with every chunk of at most kChunk rows: body(std::integral_constant<R>, row0).
template <bool SLICED, class F> __device__ __forceinline__ void for_rows(const LaneMap& lm, F body)
{
    if constexpr (!SLICED) {
        body(IntC<1>{}, 0);
    } else
    for (int row0 = 0; row0 < lm.rows; row0 += kChunk) {
        if (lm.rows - row0 >= kChunk)
            body(IntC<kChunk>{}, row0);
        else
            body(IntC<1>{}, row0);
    }
}

// Evaluates the first m <= kNodes listed nodes for the group's targets.
template <bool PERIODIC, bool SPLIT, bool QUAD, bool POT, class W>
__device__ __forceinline__ void flush_nodes(W& w, int m, const TreeArrays& t,
                                            const WalkParams& p, float inv2rs, const LaneMap& lm,
                                            Acc& acc)
{
    const int lane = threadIdx.x & 31;
    // quadrupoles with eps^2 > min distance^2 are evaluated two nodes at a time (with the split
    // kernel, forces only); the Newtonian ones in the traceless form
    const bool packed = QUAD && !(POT && SPLIT) && p.eps2 > p.min_dist2;
    const int pairs = (m + 1) >> 1;
    if ((m & 1) && lane == 0)
        w.nlist[m] = w.nlist[m - 1];  // an odd list's last node is paired with itself, massless
    __syncwarp();
    for (int i = lane; i < pairs; i += 32) {
        float v[2][11];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = w.nlist[2 * i + h];
            const int k = e & kIndexMask;
            float4 mo = t.mono[k];
            if (PERIODIC) {
                const int code = static_cast<int>(static_cast<unsigned>(e) >> kIndexBits);
                mo.x -= shift_of(code, 0, p.box);
                mo.y -= shift_of(code, 1, p.box);
                mo.z -= shift_of(code, 2, p.box);
            }
            v[h][0] = mo.x;
            v[h][1] = mo.y;
            v[h][2] = mo.z;
            v[h][3] = mo.w;
            if (QUAD) {
                const float4 qa = t.quadA[k];
                const float2 qb = t.quadB[k];
                v[h][4] = qa.x;
                v[h][5] = qa.y;
                v[h][6] = qa.z;
                v[h][7] = qa.w;
                v[h][8] = qb.x;
                v[h][9] = qb.y;
                if (packed) {
                    const float tr = qa.x + qa.w + qb.y;
                    const float c = SPLIT ? -1.0f : -3.0f, off = SPLIT ? 0.0f : tr;
                    v[h][4] = fmaf(c, qa.x, off);
                    v[h][5] = c * qa.y;
                    v[h][6] = c * qa.z;
                    v[h][7] = fmaf(c, qa.w, off);
                    v[h][8] = c * qb.x;
                    v[h][9] = fmaf(c, qb.y, off);
                    v[h][10] = SPLIT ? -0.5f * tr : tr * p.eps2;
                }
            }
        }
        if (2 * i + 1 == m) {
#pragma unroll
            for (int c = 3; c < 11; ++c)
                v[1][c] = 0.0f;
        }
#pragma unroll
        for (int c = 0; c < (QUAD ? 5 : 2); ++c)
            w.nd[c][i] = make_float4(v[0][2 * c], v[1][2 * c], v[0][2 * c + 1], v[1][2 * c + 1]);
        if (packed)
            w.nd_tr[i] = make_float2(v[0][10], v[1][10]);
    }
    __syncwarp();
    for_rows<walk_sliced<SPLIT, QUAD>()>(lm, [&](auto rc, int row0) {
        constexpr int R = decltype(rc)::value;
        Rows<R, POT ? 4 : 3> rows;
        rows.load(w, lm, row0);
        float none = 0.0f;
        if (packed) {
            F2 nx[R], ny[R], nz[R], fx[R], fy[R], fz[R], np[R];
            const F2 eps2 = f2(p.eps2);
#pragma unroll
            for (int k = 0; k < R; ++k) {
                nx[k] = f2(-rows.tx[k]);
                ny[k] = f2(-rows.ty[k]);
                nz[k] = f2(-rows.tz[k]);
                fx[k] = fy[k] = fz[k] = np[k] = f2(0.0f);
            }
#pragma unroll 1
            for (int j = lm.slice; j < pairs; j += lm.nslices) {
                const ulonglong2* nd = reinterpret_cast<const ulonglong2*>(&w.nd[0][j]);
                constexpr int st = QUAD ? kNodes / 2 : 0;  // (packed implies QUAD)
                const ulonglong2 a = nd[0], b = nd[st], c = nd[2 * st], d = nd[3 * st], e = nd[4 * st];
                const F2 tr{*reinterpret_cast<const unsigned long long*>(&w.nd_tr[QUAD ? j : 0])};
                const F2 q[6] = {{c.x}, {c.y}, {d.x}, {d.y}, {e.x}, {e.y}};
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    if (SPLIT)
                        pair_pn_split2({a.x}, {a.y}, {b.x}, {b.y}, q, tr, nx[k], ny[k], nz[k], eps2, inv2rs,
                                       fx[k], fy[k], fz[k]);
                    else
                        pair_pn_newton2<POT>({a.x}, {a.y}, {b.x}, {b.y}, q, tr, nx[k], ny[k], nz[k], eps2, fx[k],
                                             fy[k], fz[k], np[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < R; ++k) {
                rows.f[0][k] = lo(fx[k]) + hi(fx[k]);
                rows.f[1][k] = lo(fy[k]) + hi(fy[k]);
                rows.f[2][k] = lo(fz[k]) + hi(fz[k]);
                if (POT)
                    rows.f[POT ? 3 : 0][k] = -(lo(np[k]) + hi(np[k]));
            }
        } else {
#pragma unroll 1
            for (int j = lm.slice; j < pairs; j += lm.nslices) {
                const float4 a = w.nd[0][j], b = w.nd[1][j];
                const float4 c = QUAD ? w.nd[QUAD ? 2 : 0][j] : make_float4(0, 0, 0, 0);
                const float4 d = QUAD ? w.nd[QUAD ? 3 : 0][j] : make_float4(0, 0, 0, 0);
                const float4 e = QUAD ? w.nd[QUAD ? 4 : 0][j] : make_float4(0, 0, 0, 0);
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    pair_pn<SPLIT, QUAD, POT>(make_float4(a.x, a.z, b.x, b.z), make_float4(c.x, c.z, d.x, d.z),
                                              make_float2(e.x, e.z), rows.tx[k], rows.ty[k], rows.tz[k], p,
                                              inv2rs, rows.f[0][k], rows.f[1][k], rows.f[2][k],
                                              POT ? rows.f[POT ? 3 : 0][k] : none);
                    pair_pn<SPLIT, QUAD, POT>(make_float4(a.y, a.w, b.y, b.w), make_float4(c.y, c.w, d.y, d.w),
                                              make_float2(e.y, e.w), rows.tx[k], rows.ty[k], rows.tz[k], p,
                                              inv2rs, rows.f[0][k], rows.f[1][k], rows.f[2][k],
                                              POT ? rows.f[POT ? 3 : 0][k] : none);
                }
            }
        }
        __syncwarp();
        rows.fold(lm, row0, acc);
    });
    __syncwarp();
}

// ---- cutoff filter on the tensor cores -----------------------------------------------------
// Which of 128 tile sources lie inside each of the 32 targets' cutoff spheres: the signs of
//   D = |s|^2 - 2 s t + |t|^2 - r^2 = [-2t, 1, 1, Thi, Tlo] . [s, Shi, Slo, 1, 1],
// a 32 x 128 x 8 product (mma m16n8k8, FP16 operands, FP32 sums), s and t in units of r_cut / 8
// from the group's centre.  S = |s|^2 of the ROUNDED s and T = |t|^2 - r^2 are split into two FP16
// parts, so D is the exact distance test of the rounded points up to 2^-22 of S and T; r carries
// the rounding of both points.  The marked set therefore contains every pair inside the cutoff
// (and about 0.5 % more), and the pair law's own FP32 test decides the rest, so the sums are those
// of the scalar filter, which spends nine instructions on each listed pair (5 to 7 listed for each
// evaluated one).  Measured: 256^3 walk 7.54 -> 7.27 ms, the 64^3 box 0.176 -> 0.171 ms.  The walks
// with quadrupoles keep the scalar filter: they filter few leaves (near ones go unfiltered, far
// ones as nodes) and lost more to the registers (128^3 CIC 2.26 -> 2.41 ms).
constexpr float kFilterScale = 8.0f;
constexpr float kFilterMaxExtent = 64.0f;  // of the group's half box, scaled: T and S stay far below 65504

__device__ __forceinline__ unsigned pack_h2(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&h);
}

// One FP16 row: {x, y, z, hi, lo, one, one, 0} of the point x, y, z; returns the rounded point's
// square norm through n2.
__device__ __forceinline__ float round_point(float& x, float& y, float& z)
{
    x = __half2float(__float2half_rn(x));
    y = __half2float(__float2half_rn(y));
    z = __half2float(__float2half_rn(z));
    return fmaf(x, x, fmaf(y, y, z * z));
}

template <class W>
__device__ __forceinline__ void filter_group(W& w, const float4 me, const float* gc, const float* ghalf, float rcut)
{
    const int lane = threadIdx.x & 31;
    const float sc = kFilterScale / rcut;
    const float ext = fmaxf(ghalf[0], fmaxf(ghalf[1], ghalf[2])) * sc;
    // position errors in scaled units: FP16 rounding of both points (sqrt(3) 2^-11 of their
    // coordinates, at most ext and ext + 8), FP32 rounding of the subtraction
    const float far = fmaxf(fabsf(gc[0]), fmaxf(fabsf(gc[1]), fabsf(gc[2])));
    const float d = 0.001f * (2.0f * ext + kFilterScale) + 1.0e-6f * sc * far;
    const float r = kFilterScale + d;
    const float r2 = r * r + 1.2e-5f * (2.0f * ext + kFilterScale) * (2.0f * ext + kFilterScale);
    float x = (me.x - gc[0]) * sc, y = (me.y - gc[1]) * sc, z = (me.z - gc[2]) * sc;
    const float t = round_point(x, y, z) - r2;
    const float hi = __half2float(__float2half_rn(t));
    w.arow[lane] = make_uint4(pack_h2(-2.0f * x, -2.0f * y), pack_h2(-2.0f * z, 1.0f), pack_h2(1.0f, hi),
                              pack_h2(t - hi, 0.0f));
    // (a NaN or infinite extent fails the comparison too)
    if (lane == 0)
        w.frame = make_float4(gc[0], gc[1], gc[2], ext <= kFilterMaxExtent && d < kFilterScale ? sc : 0.0f);
}

// Fills w.mask for the tile's sources base .. base + 127 (of nb): bit b of word q of target j is
// source 32 q + b.
template <class W> __device__ __forceinline__ void filter_tile(W& w, int base, int nb, const float4 frame)
{
    const int lane = threadIdx.x & 31;
    const int row = lane >> 2, q = lane & 3;
    const unsigned* ar = reinterpret_cast<const unsigned*>(w.arow);
    unsigned a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        a[i] = ar[(row + 8 * i) * 4 + q];
    unsigned m[4] = {0u, 0u, 0u, 0u};
    // column n of n-tile t of part h is source 32 (n / 2) + 8 h + 2 t + n % 2
    const int col = base + 32 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);
#pragma unroll 1
    for (int h = 3; h >= 0; --h) {
        uint4 v = make_uint4(0u, pack_h2(0.0f, 30000.0f), 0u, 0u);  // past the end: never inside
        if (col + 8 * h < nb) {
            const float4 s4 = w.tile[col + 8 * h];
            float x = (s4.x - frame.x) * frame.w, y = (s4.y - frame.y) * frame.w, z = (s4.z - frame.z) * frame.w;
            const float s2 = round_point(x, y, z);
            const float hi = __half2float(__float2half_rn(s2));
            v = make_uint4(pack_h2(x, y), pack_h2(z, hi), pack_h2(s2 - hi, 1.0f), pack_h2(1.0f, 0.0f));
        }
        w.brow[lane] = v;
        __syncwarp();
        unsigned b[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                     : "r"(smem_u32(w.brow) + lane * 16)
                     : "memory");
#pragma unroll
        for (int t = 3; t >= 0; --t) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float c[4];
                asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
                    "{%7, %7, %7, %7};"
                    : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                    : "r"(a[2 * i]), "r"(a[2 * i + 1]), "r"(b[t]), "f"(0.0f));
                m[2 * i] = __funnelshift_l(__float_as_uint(c[1]), m[2 * i], 1);
                m[2 * i] = __funnelshift_l(__float_as_uint(c[0]), m[2 * i], 1);
                m[2 * i + 1] = __funnelshift_l(__float_as_uint(c[3]), m[2 * i + 1], 1);
                m[2 * i + 1] = __funnelshift_l(__float_as_uint(c[2]), m[2 * i + 1], 1);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w.mask[(base >> 5) + q][row + 8 * i] = m[i];
    __syncwarp();
}

template <bool PERIODIC, bool SPLIT, bool POT, bool SLICED, bool FILTER, class W>
__device__ __forceinline__ void flush_leaves(W& w, int first, int nl, bool sure, const float4* __restrict__ pos4,
                                             const TreeArrays& t, const WalkParams& p,
                                             float inv2rs, bool cut, float tx, float ty, float tz,
                                             int self_index, Acc& acc, uint32_t& phase, int* err,
                                             const WalkOutputs& o, int pair_row, int& npair,
                                             unsigned& evald, const LaneMap& lm)
{
    // pairs closer than rcorr are recorded for the learned correction (pair_row < 0: a lane
    // without a target records nothing)
    const bool rec = o.pair_src != nullptr && p.rcorr2 > 0.0f;
    auto record = [&](float4 s4, int gidx) {
        const float dx = s4.x - tx, dy = s4.y - ty, dz = s4.z - tz;
        if (pair_row >= 0 && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= p.rcorr2) {
            if (npair < kPairSlots)
                o.pair_src[static_cast<size_t>(pair_row) * kPairSlots + npair] = gidx;
            ++npair;
        }
    };
    const int lane = threadIdx.x & 31;
    // Force-only evaluation above the minimum-distance floor runs the per-lane cutoff filter
    const bool fast = !POT && p.eps2 > p.min_dist2;
    cut = cut && !sure;  // every pair of these leaves lies inside the cutoff
    if (cut && !fast) {
        // Drop leaves that no target of this warp can reach: a leaf whose (shifted) box is
        // farther than the cutoff from every lane's target holds no pair inside the cutoff.
        // (With the per-lane filter this costs more than it saves: the filter drops the same
        // sources exactly.)
        // Lane j loads the boxes of list entries j and j + 32 in one round (no serial chain
        // of loads); each box is then broadcast by shuffle and tested against every target.
        float4 lo[2], hi[2];
        bool ppi[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = lane + 32 * h;
            lo[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            hi[h] = lo[h];
            ppi[h] = false;
            if (j < nl) {
                const int code = w.lcode[first + j];
                ppi[h] = PERIODIC && code == kPerPairImage;
                const int k = w.lnode[first + j];
                const float4 b0 = t.box0[k];
                const float4 b1 = t.box1[k];
                float sxo = 0.0f, syo = 0.0f, szo = 0.0f;
                if (PERIODIC && !ppi[h]) {
                    sxo = shift_of(code, 0, p.box);
                    syo = shift_of(code, 1, p.box);
                    szo = shift_of(code, 2, p.box);
                }
                lo[h] = make_float4(b0.x - sxo, b0.y - syo, b0.z - szo, 0.0f);
                hi[h] = make_float4(b1.x - sxo, b1.y - syo, b1.z - szo, 0.0f);
            }
        }
        const float lim2 = p.rcut2 * 1.0001f;
        int keep = 0;
        for (int j = 0; j < nl; ++j) {
            const int h = j >> 5, src = j & 31;
            const float bx0 = __shfl_sync(kFullMask, h ? lo[1].x : lo[0].x, src);
            const float by0 = __shfl_sync(kFullMask, h ? lo[1].y : lo[0].y, src);
            const float bz0 = __shfl_sync(kFullMask, h ? lo[1].z : lo[0].z, src);
            const float bx1 = __shfl_sync(kFullMask, h ? hi[1].x : hi[0].x, src);
            const float by1 = __shfl_sync(kFullMask, h ? hi[1].y : hi[0].y, src);
            const float bz1 = __shfl_sync(kFullMask, h ? hi[1].z : hi[0].z, src);
            const bool pp = __shfl_sync(kFullMask, h ? ppi[1] : ppi[0], src);
            bool need = true;
            if (!pp) {
                const float ddx = fmaxf(fmaxf(bx0 - tx, tx - bx1), 0.0f);
                const float ddy = fmaxf(fmaxf(by0 - ty, ty - by1), 0.0f);
                const float ddz = fmaxf(fmaxf(bz0 - tz, tz - bz1), 0.0f);
                need = fmaf(ddx, ddx, fmaf(ddy, ddy, ddz * ddz)) <= lim2;
            }
            if (__any_sync(kFullMask, need)) {
                if (lane == 0 && keep != j) {
                    w.lstart[first + keep] = w.lstart[first + j];
                    w.lcount[first + keep] = w.lcount[first + j];
                    w.lcode[first + keep] = w.lcode[first + j];
                    w.lnode[first + keep] = w.lnode[first + j];
                }
                ++keep;
            }
        }
        __syncwarp();
        nl = keep;
        if (nl == 0)
            return;
    }
    // exclusive prefix of the leaf sizes (list holds at most 64 entries)
    const int c0 = lane < nl ? w.lcount[first + lane] : 0;
    const int c1 = lane + 32 < nl ? w.lcount[first + lane + 32] : 0;
    const int i0 = warp_incl_scan(c0);
    const int t0 = __shfl_sync(kFullMask, i0, 31);
    const int i1 = warp_incl_scan(c1) + t0;
    const int total = __shfl_sync(kFullMask, i1, 31);
    if (lane < nl)
        w.lpre[first + lane] = i0 - c0;
    if (lane + 32 < nl)
        w.lpre[first + lane + 32] = i1 - c1;
    __syncwarp();
    SplitK sk;
    sk.inv2rs = inv2rs;
    sk.cexp = -1.4426950408889634f * inv2rs * inv2rs;
    sk.pk = 0.3275911f * inv2rs;
    sk.c2 = kTwoOverSqrtPi * inv2rs;
    int jfirst = 0;
    constexpr int kSources = W::kSources;
    for (int cbase = 0; cbase < total; cbase += kSources) {
        const int cend = min(cbase + kSources, total);
        // make earlier generic-proxy reads of the tile visible before the async writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0)
            mbar_arrive_expect_tx(&w.bar, static_cast<uint32_t>(cend - cbase) * 16u);
        __syncwarp();
        // each lane copies the tile parts of its leaves and notes whether they need a periodic
        // image shift or per-pair images
        bool shifted = false, pairimg = false;
        for (int j = lane; j < nl; j += 32) {
            const int lo = max(w.lpre[first + j], cbase);
            const int hi = min(w.lpre[first + j] + w.lcount[first + j], cend);
            if (hi > lo) {
                bulk_g2s(&w.tile[lo - cbase], pos4 + (w.lstart[first + j] + (lo - w.lpre[first + j])),
                         static_cast<uint32_t>(hi - lo) * 16u, &w.bar);
                if (PERIODIC) {
                    const int code = w.lcode[first + j];
                    pairimg = pairimg || code == kPerPairImage;
                    shifted = shifted || (code != kNoShift && code != kPerPairImage);
                }
                if (rec || POT)
                    for (int q = lo; q < hi; ++q)
                        w.tidx[q - cbase] = FILTER ? j : w.lstart[first + j] + (q - w.lpre[first + j]);
            }
        }
        const bool any_shift = PERIODIC && __any_sync(kFullMask, shifted);
        const bool per_pair = PERIODIC && __any_sync(kFullMask, pairimg);
        if (rec || POT)
            __syncwarp();
        mbar_wait_bounded(&w.bar, phase, err);
        phase ^= 1u;
        // Periodic images: the lane that copied a shifted leaf moves its sources into the
        // group's image in place (leaves summed with per-pair images keep their stored
        // positions).  Tiles without shifted leaves, most of them, skip this.
        if (any_shift) {
            for (int j = lane; j < nl; j += 32) {
                const int lo = max(w.lpre[first + j], cbase);
                const int hi = min(w.lpre[first + j] + w.lcount[first + j], cend);
                const int code = w.lcode[first + j];
                if (hi <= lo || code == kNoShift || code == kPerPairImage)
                    continue;
                const float shx = shift_of(code, 0, p.box), shy = shift_of(code, 1, p.box),
                            shz = shift_of(code, 2, p.box);
                for (int q = lo; q < hi; ++q) {
                    float4& s4 = w.tile[q - cbase];
                    s4.x = __fsub_rn(s4.x, shx);
                    s4.y = __fsub_rn(s4.y, shy);
                    s4.z = __fsub_rn(s4.z, shz);
                }
            }
            __syncwarp();
        }
        const int nb = cend - cbase;
        if (!per_pair && !rec && !(fast && cut)) {
            // every listed source of the tile goes through the pair law, two at a time (the tile
            // filled up with massless sources to whole pairs for every slice)
            evald += nb;
            const int npad = (nb + 2 * lm.nslices - 1) & ~(2 * lm.nslices - 1);
            const bool packed = SLICED && !cut && !(POT && SPLIT) && p.eps2 > p.min_dist2;
            if (packed) {
                for (int j = nb + lane; j < npad; j += 32) {
                    w.tile[j] = make_float4(tx, ty, tz, 0.0f);
                    if constexpr (POT)
                        w.tidx[j] = -1;
                }
                __syncwarp();
            }
            for_rows<SLICED>(lm, [&](auto rc, int row0) {
                constexpr int R = decltype(rc)::value;
                Rows<R, POT ? 4 : 3> rows;
                rows.load(w, lm, row0);
                float none = 0.0f;
                const int t0 = self_index - lane + lm.slot + kSlots * row0;
                if (packed) {
                    F2 nx[R], ny[R], nz[R], fx[R], fy[R], fz[R], np[R];
                    const F2 eps2 = f2(p.eps2);
#pragma unroll
                    for (int k = 0; k < R; ++k) {
                        nx[k] = f2(-rows.tx[k]);
                        ny[k] = f2(-rows.ty[k]);
                        nz[k] = f2(-rows.tz[k]);
                        fx[k] = fy[k] = fz[k] = np[k] = f2(0.0f);
                    }
#pragma unroll 1
                    for (int j = lm.slice; j < npad; j += 2 * lm.nslices) {
                        const float4 s0 = w.tile[j], s1 = w.tile[j + lm.nslices];
                        const int i0 = POT ? w.tidx[j] : 0, i1 = POT ? w.tidx[j + lm.nslices] : 0;
                        const F2 x = f2(s0.x, s1.x), y = f2(s0.y, s1.y), z = f2(s0.z, s1.z), m = f2(s0.w, s1.w);
#pragma unroll
                        for (int k = 0; k < R; ++k) {
                            const int own = t0 + kSlots * k;
                            const F2 mp = POT ? f2(i0 == own ? 0.0f : s0.w, i1 == own ? 0.0f : s1.w) : m;
                            pair_fast2<SPLIT, POT>(x, y, z, m, mp, nx[k], ny[k], nz[k], eps2, sk, fx[k], fy[k], fz[k],
                                                   np[k]);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < R; ++k) {
                        rows.f[0][k] = lo(fx[k]) + hi(fx[k]);
                        rows.f[1][k] = lo(fy[k]) + hi(fy[k]);
                        rows.f[2][k] = lo(fz[k]) + hi(fz[k]);
                        if (POT)
                            rows.f[POT ? 3 : 0][k] = -(lo(np[k]) + hi(np[k]));
                    }
                } else {
#pragma unroll 1
                    for (int j = lm.slice; j < nb; j += lm.nslices) {
                        const float4 s4 = w.tile[j];
                        const int src = POT ? w.tidx[j] : 0;
#pragma unroll
                        for (int k = 0; k < R; ++k)
                            pair_pp<SPLIT, POT>(s4, rows.tx[k], rows.ty[k], rows.tz[k], p, inv2rs, cut,
                                                POT && src == t0 + kSlots * k, rows.f[0][k], rows.f[1][k],
                                                rows.f[2][k], POT ? rows.f[POT ? 3 : 0][k] : none);
                    }
                }
                __syncwarp();
                rows.fold(lm, row0, acc);
            });
            __syncwarp();
            continue;
        }
        float fx = 0.0f, fy = 0.0f, fz = 0.0f, fp = 0.0f;
        if (fast && cut && !per_pair) {
            // Cutoff filter: each lane marks the tile sources inside its own cutoff sphere
            // (the same r^2 expression as the pair law, so the set is exact), then sums only
            // those.  Skipped pairs contribute exactly zero in the unfiltered sum, so the
            // result is bit-identical to summing every listed source in tile order.
            const int nw = (nb + 31) >> 5;
            // r2 <= rcut2 exactly when r2 - next_float(rcut2) is negative (a float difference
            // has the exact sign), so the sign bit is the mask bit: one funnel shift appends it
            const float rc2n = __uint_as_float(__float_as_uint(p.rcut2) + 1u);
            // the walks that only filter mark on the tensor cores; then a marked pair takes the
            // pair law's own distance test
            const float4 frame = FILTER ? w.frame : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (FILTER && frame.w > 0.0f) {
                filter_tile(w, 0, nb, frame);
                if (nb > 128)
                    filter_tile(w, 128, nb, frame);
            }
            for (int wd = 0; frame.w == 0.0f && wd < nw; ++wd) {
                const int qb = wd << 5;
                unsigned m = 0u;
                if (qb + 32 <= nb) {
                    // highest source first, shifting the mask left (short loop body)
#pragma unroll 8
                    for (int b = 31; b >= 0; --b) {
                        const float4 s4 = w.tile[qb + b];
                        const float dx = s4.x - tx, dy = s4.y - ty, dz = s4.z - tz;
                        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        m = __funnelshift_l(__float_as_uint(__fsub_rn(r2, rc2n)), m, 1);
                    }
                } else {
                    for (int b = 0; qb + b < nb; ++b) {
                        const float4 s4 = w.tile[qb + b];
                        const float dx = s4.x - tx, dy = s4.y - ty, dz = s4.z - tz;
                        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        if (r2 <= p.rcut2)
                            m |= 1u << b;
                    }
                }
                w.mask[wd][lane] = m;
            }
            if constexpr (FILTER) {
                // This lane's words with a mark, moved together, a zero word behind them; each
                // word's place in the tile, four bits a word.  The lanes then stay in step: no lane
                // looks for its next word while the others wait (256^3 walk 7.26 -> 7.0 ms at 128
                // sources a tile).
                unsigned order = 0u;
                int used = 0;
                for (int wd = 0; wd < nw; ++wd) {
                    const unsigned v = w.mask[wd][lane];
                    if (v != 0u) {
                        w.mask[used][lane] = v;
                        order |= static_cast<unsigned>(wd) << (4 * used);
                        ++used;
                    }
                }
                w.mask[used][lane] = 0u;
                unsigned m = w.mask[0][lane], mnext = w.mask[1][lane];
                int at = 1;
                while (m != 0u) {
                    const int b = static_cast<int>((order & 15u) << 5) + __ffs(m) - 1;
                    m &= m - 1u;
                    const float4 s4 = w.tile[b];
                    const bool last = m == 0u;
                    m = last ? mnext : m;
                    order = last ? order >> 4 : order;
                    at += last && mnext != 0u ? 1 : 0;
                    mnext = w.mask[at][lane];
                    evald += pair_fast<SPLIT>(s4, tx, ty, tz, p.eps2, p.rcut2, true, sk, fx, fy, fz);
                    if (rec) {
                        const int j = first + w.tidx[b];
                        record(s4, w.lstart[j] + (cbase + b - w.lpre[j]));
                    }
                }
            } else {
                // (few leaves are filtered here: 1 % of an isolated TreePM pass is lost to the above)
                int wd = 0;
                unsigned m = w.mask[0][lane];
                for (;;) {
                    while (m == 0u && ++wd < nw)
                        m = w.mask[wd][lane];
                    if (m == 0u)
                        break;
                    const int b = (wd << 5) + __ffs(m) - 1;
                    m &= m - 1u;
                    const float4 s4 = w.tile[b];
                    evald += pair_fast<SPLIT>(s4, tx, ty, tz, p.eps2, p.rcut2, false, sk, fx, fy, fz);
                    if (rec)
                        record(s4, w.tidx[b]);
                }
            }
            __syncwarp();
            // (jfirst, the first leaf the unfiltered path below must look at, is left behind
            // here: that path skips the leaves that end before its tile)
        } else {
            for (int j = jfirst; j < nl; ++j) {
                const int pre = w.lpre[first + j];
                if (pre >= cend)
                    break;
                const int lo = max(pre, cbase);
                const int hi = min(pre + w.lcount[first + j], cend);
                if (hi <= lo)
                    continue;
                const int gsrc0 = w.lstart[first + j] + (lo - pre);
                const int off = lo - cbase;
                const int cntp = hi - lo;
                evald += cntp;  // every listed source goes through the pair law here
                if (PERIODIC && w.lcode[first + j] == kPerPairImage) {
                    // rare slow path: nearest image chosen per pair
                    const float inv_box = 1.0f / p.box;
                    for (int q = 0; q < cntp; ++q) {
                        float4 s4 = w.tile[off + q];
                        s4.x = tx + (s4.x - tx - p.box * rintf((s4.x - tx) * inv_box));
                        s4.y = ty + (s4.y - ty - p.box * rintf((s4.y - ty) * inv_box));
                        s4.z = tz + (s4.z - tz - p.box * rintf((s4.z - tz) * inv_box));
                        pair_pp<SPLIT, POT>(s4, tx, ty, tz, p, inv2rs, cut,
                                            POT && gsrc0 + q == self_index, fx, fy, fz, fp);
                        if (rec)
                            record(s4, gsrc0 + q);
                    }
                    if (pre + w.lcount[first + j] <= cend)
                        jfirst = j + 1;
                    continue;
                }
                if (fast) {
                    for (int q = 0; q < cntp; ++q)
                        pair_fast<SPLIT>(w.tile[off + q], tx, ty, tz, p.eps2, p.rcut2, cut, sk, fx, fy, fz);
                } else {
                    for (int q = 0; q < cntp; ++q)
                        pair_pp<SPLIT, POT>(w.tile[off + q], tx, ty, tz, p, inv2rs, cut,
                                            POT && gsrc0 + q == self_index, fx, fy, fz, fp);
                }
                if (rec)
                    for (int q2 = 0; q2 < cntp; ++q2)
                        record(w.tile[off + q2], gsrc0 + q2);
                if (pre + w.lcount[first + j] <= cend)
                    jfirst = j + 1;
            }
        }
        acc.add(0, fx);
        acc.add(1, fy);
        acc.add(2, fz);
        if (POT)
            acc.add(3, fp);
        __syncwarp();
    }
}

// Resident blocks an SM that the walk is compiled for (4: 128 registers, 5: 96, 6: 80).  The
// sliced evaluation keeps two nodes, two targets and their sums in packed registers: 4 blocks
// hold them without spills (Hernquist 4M: 36.4 ms at 4, 37.4 at 5; isolated TreePM 1M: 4.35 at 4,
// 4.45 at 5, 4.99 at 6).  The walk that only filters takes the warps that its tile leaves room for
// (6 blocks, 80 registers: 256^3 6.45 ms, 5: 6.81).
template <bool SPLIT, bool QUAD, bool POT> constexpr int walk_min_blocks()
{
    return walk_filters<SPLIT, QUAD, POT>() ? 6 : 4;
}

// Persistent kernel: each warp takes groups from a global queue until none are left.  The
// traversal stack lives in shared memory; when it would overflow, its oldest half is spilled
// to a per-warp-slot global area and refilled when the shared part runs dry.
template <bool PERIODIC, bool SPLIT, bool QUAD, bool POT>
__global__ void __launch_bounds__(kWarps * 32, walk_min_blocks<SPLIT, QUAD, POT>()) k_walk(const float4* __restrict__ pos4, int n,
                                                       TreeArrays t, const int* __restrict__ gstart,
                                                       const int* __restrict__ groot,
                                                       const int* __restrict__ ngroups_ptr,
                                                       const int* __restrict__ gorder,
                                                       const int* __restrict__ gordered,
                                                       WalkParams p_in, float inv_box,
                                                       WalkOutputs o, unsigned* queue,
                                                       int* spill_base, int* err)
{
    // The isolated TreePM's split scale and cutoff follow its mesh cell, which the device
    // recomputes from the particles' bounds for every evaluation: read them here.
    WalkParams p = p_in;
    if (!PERIODIC && SPLIT && p_in.iso != nullptr) {
        p.rsplit = p_in.iso->rsplit;
        p.rcut2 = p_in.iso->rcut2;
        p.max_node_size = p_in.iso->max_node_size;
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr bool FILTER = walk_filters<SPLIT, QUAD, POT>();
    using Smem = WarpSmem<QUAD, FILTER>;
    Smem& w = reinterpret_cast<Smem*>(smem_raw)[warp];
    int* spill = spill_base + static_cast<size_t>(blockIdx.x * kWarps + warp) * kSpill;
    const int ngroups = *ngroups_ptr;
    const bool ordered = *gordered != 0;
    if (lane == 0)
        mbar_init(&w.bar, 1);
    fence_mbar_init();
    __syncwarp();
    constexpr bool SLICED = walk_sliced<SPLIT, QUAD>();
    // (adaptive steps: force-only walks of the octree solver)
    const bool adaptive = !PERIODIC && !SPLIT && !POT && p.active != nullptr;
    const bool cut = p.rcut2 > 0.0f;
    const float inv2rs = SPLIT ? 0.5f / p.rsplit : 0.0f;
    const float rcut = __fsqrt_rn(p.rcut2);
    const float half_box = __fmul_rn(0.5f, p.box);
    const unsigned lt = lanemask_lt();
    uint32_t phase = 0;

    for (;;) {
        int g = 0;
        if (lane == 0)
            g = static_cast<int>(atomicAdd(queue, 1u));
        g = __shfl_sync(kFullMask, g, 0);
        if (g >= ngroups)
            break;
        if (ordered)
            g = gorder[g];
        const int g0 = gstart[g];
        const int members = gstart[g + 1] - g0;
        const float4 member = pos4[lane < members ? g0 + lane : g0];
        // The targets this warp evaluates, one owner lane each: the group's members or, in
        // adaptive substeps, those of them that close their step (a group without one is not
        // walked).  Boxes and decisions are the whole group's either way.  (96 clusters, six levels, a
        // block of 32 substeps: walks 19.6 -> 16.9 ms.)
        int gn = members, ti = g0 + lane;
        float4 me = member;
        if (adaptive) {
            const unsigned closing = __ballot_sync(kFullMask, lane < members && p.active[g0 + lane] != 0);
            if (closing == 0u)
                continue;
            gn = __popc(closing);
            unsigned m = closing;
            for (int skip = lane < gn ? lane : 0; skip > 0; --skip)
                m &= m - 1u;
            const int src = __ffs(m) - 1;  // the closing member of this lane's rank
            ti = g0 + src;
            me.x = __shfl_sync(kFullMask, member.x, src);
            me.y = __shfl_sync(kFullMask, member.y, src);
            me.z = __shfl_sync(kFullMask, member.z, src);
            me.w = __shfl_sync(kFullMask, member.w, src);
        }
        const bool valid = lane < gn;
        const LaneMap lanes(gn, SLICED);
        w.tgt[lane] = me;
        float gmin[3] = {member.x, member.y, member.z}, gmax[3] = {member.x, member.y, member.z};
#pragma unroll
        for (int a = 0; a < 3; ++a)
            for (int off = 16; off > 0; off >>= 1) {
                gmin[a] = fminf(gmin[a], __shfl_xor_sync(kFullMask, gmin[a], off));
                gmax[a] = fmaxf(gmax[a], __shfl_xor_sync(kFullMask, gmax[a], off));
            }
        float gc[3], ghalf[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            gc[a] = __fmul_rn(0.5f, __fadd_rn(gmin[a], gmax[a]));
            ghalf[a] = __fmul_rn(0.5f, __fsub_rn(gmax[a], gmin[a]));
        }

        if (FILTER && cut)
            filter_group(w, me, gc, ghalf, rcut);
        // With a cutoff, leaves wholly inside it for every target ("sure": the farthest corners of
        // leaf and group) are listed from the far end of the leaf list and summed without the
        // per-lane filter; the margin covers the rounding of a pair's own distance test.
        const float sure2 = p.rcut2 * 0.9999f;
        const bool sort_leaves = SLICED && cut && o.pair_src == nullptr &&
                                 ghalf[0] * ghalf[0] + ghalf[1] * ghalf[1] + ghalf[2] * ghalf[2] < p.rcut2;
        if (lane == 0)
            w.stack[0] = static_cast<unsigned>(groot[g]);  // the group's system root, as one child
        __syncwarp();
        int top = 1, gtop = 0, nn = 0, nl = 0, ns = 0, lp = 0;
        unsigned cnt_pp = 0, cnt_pn = 0;  // (a group lists a particle or a node at most once)
        Acc acc;
        acc.zero();
        int npair = 0;
        unsigned evald = 0;  // pairs this lane's target took through the pair law
        // one traversal step (while nodes are left) and the flushes it makes due; the last turn
        // flushes what is still listed
        for (;;) {
            const bool done = top == 0 && gtop == 0;
            if (!done) {
                if (top == 0) {  // refill from the spill area (uniform branch)
                    const int m = min(gtop, kStack / 2);
                    for (int i = lane; i < m; i += 32)
                        w.stack[i] = static_cast<unsigned>(spill[gtop - m + i]);
                    gtop -= m;
                    top = m;
                    __syncwarp();
                }
                // the children of the four nodes opened last, eight lanes a node
                const int from = top - 1 - (lane >> 3);
                const unsigned ent = w.stack[max(from, 0)];
                const int child = lane & 7;
                const bool on = from >= 0 && child <= static_cast<int>(ent >> kIndexBits);
                const int k = on ? static_cast<int>(ent & kIndexMask) + child : -1;
                top = max(top - 4, 0);
                __syncwarp();
                bool accept = false, leaf = false, sure = false;
                int nch = 0, link = 0, info = 0, code = 0;
                if (k >= 0) {
                    const float4 b0 = t.box0[k];
                    const float4 b1 = t.box1[k];
                    // the centre of mass matters only to a node that may be accepted; with a node
                    // size cap (TreePM) most nodes are too large, and skip the load
                    const bool capped = SPLIT && p.max_node_size > 0.0f;  // the cap is a TreePM setting
                    float4 mo = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (!capped)
                        mo = t.mono[k];
                    link = __float_as_int(b0.w);
                    info = __float_as_int(b1.w);
                    const float bmin[3] = {b0.x, b0.y, b0.z}, bmax[3] = {b1.x, b1.y, b1.z};
                    float sh[3] = {0.0f, 0.0f, 0.0f};
                    bool amb = false;
                    if (PERIODIC) {
                        // Image-ambiguous node (its extent + the group's + the cutoff reaches half
                        // the box): always opened; a leaf is summed with per-pair minimum images.
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            const float nh = __fmul_rn(0.5f, __fsub_rn(bmax[a], bmin[a]));
                            if (__fadd_rn(__fadd_rn(ghalf[a], nh), rcut) > half_box)
                                amb = true;
                        }
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            const float cn = __fmul_rn(0.5f, __fadd_rn(bmin[a], bmax[a]));
                            const float r = rintf(__fmul_rn(__fsub_rn(cn, gc[a]), inv_box));
                            sh[a] = __fmul_rn(p.box, r);
                            code |= (static_cast<int>(r) + 1) << (2 * a);
                        }
                        if (amb)
                            code = kPerPairImage;
                    }
                    bool pruned = false;
                    if (PERIODIC && amb) {
                        if (info < 0)
                            leaf = true;
                        else
                            nch = info;
                    } else if (cut) {
                        float d2 = 0.0f;
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            const float lo = __fsub_rn(bmin[a], sh[a]), hi = __fsub_rn(bmax[a], sh[a]);
                            const float d = fmaxf(fmaxf(__fsub_rn(lo, gmax[a]), __fsub_rn(gmin[a], hi)), 0.0f);
                            d2 = __fadd_rn(d2, __fmul_rn(d, d));
                        }
                        pruned = d2 > p.rcut2;
                    }
                    if (!pruned && !(PERIODIC && amb)) {
                        float l = 0.0f;
#pragma unroll
                        for (int a = 0; a < 3; ++a)
                            l = fmaxf(l, __fsub_rn(bmax[a], bmin[a]));
                        // The split kernel varies on the scale r_s, so its expansion error depends on
                        // the node size itself, not only on l/d: nodes at least max_node_size large
                        // are never accepted.
                        const bool small = !capped || l < p.max_node_size;
                        if (small) {
                            if (capped)
                                mo = t.mono[k];
                            const float com[3] = {mo.x, mo.y, mo.z};
                            float e2 = 0.0f;
#pragma unroll
                            for (int a = 0; a < 3; ++a) {
                                const float c = __fsub_rn(com[a], sh[a]);
                                const float e = fmaxf(fmaxf(__fsub_rn(gmin[a], c), __fsub_rn(c, gmax[a])), 0.0f);
                                e2 = __fadd_rn(e2, __fmul_rn(e, e));
                            }
                            accept = __fmul_rn(l, l) < __fmul_rn(p.theta2, e2);
                        }
                        if (!accept) {
                            if (info < 0) {
                                leaf = true;
                                if (SLICED && sort_leaves) {
                                    float m2 = 0.0f;
#pragma unroll
                                    for (int a = 0; a < 3; ++a) {
                                        const float lo = bmin[a] - sh[a], hi = bmax[a] - sh[a];
                                        const float m = fmaxf(hi - gmin[a], gmax[a] - lo);
                                        m2 = fmaf(m, m, m2);
                                    }
                                    sure = m2 <= sure2;
                                }
                            } else {
                                nch = info;
                            }
                        }
                    }
                }
                const unsigned am = __ballot_sync(kFullMask, accept);
                const unsigned lm = __ballot_sync(kFullMask, leaf);
                if (accept)
                    w.nlist[nn + __popc(am & lt)] = k | (code << kIndexBits);
                unsigned lmf = lm;
                if (SLICED && sort_leaves)
                    lmf = lm & ~__ballot_sync(kFullMask, sure);
                if (leaf) {
                    const unsigned mine = sure ? lm & ~lmf : lmf;
                    const int at = __popc(mine & lt);
                    const int pos = sure ? kList - 1 - ns - at : nl + at;
                    w.lstart[pos] = link;
                    w.lnode[pos] = k;
                    w.lcount[pos] = -info;
                    w.lcode[pos] = code;
                }
                nn += __popc(am);
                cnt_pn += __popc(am);
                if (lm != 0u) {
                    const unsigned lsum = __reduce_add_sync(kFullMask, leaf ? static_cast<unsigned>(-info) : 0u);
                    nl += __popc(lmf);
                    ns += __popc(lm & ~lmf);
                    lp += static_cast<int>(lsum);
                    cnt_pp += lsum;
                }
                const unsigned om = __ballot_sync(kFullMask, nch > 0);
                const int opened = __popc(om);
                if (top + opened > kStack) {  // spill the oldest half (uniform branch)
                    const int half = kStack / 2;
                    if (gtop + half > kSpill) {
                        if (lane == 0)
                            raise_error(err, kErrWalkStack);
                        break;
                    }
                    for (int i = lane; i < half; i += 32)
                        spill[gtop + i] = static_cast<int>(w.stack[i]);
                    __syncwarp();
                    for (int i = lane; i < top - half; i += 32)
                        w.stack[i] = w.stack[i + half];
                    __syncwarp();
                    gtop += half;
                    top -= half;
                }
                if (nch > 0)
                    w.stack[top + __popc(om & lt)] =
                        static_cast<unsigned>(link) | static_cast<unsigned>(nch - 1) << kIndexBits;
                top += opened;
                __syncwarp();
            }
            if (nn >= (done ? 1 : kNodes)) {
                const int m = min(nn, kNodes);
                flush_nodes<PERIODIC, SPLIT, QUAD, POT>(w, m, t, p, inv2rs, lanes, acc);
                nn -= m;  // the entries past a whole batch (fewer than 32) stay listed
                const int e = w.nlist[kNodes + lane];
                __syncwarp();
                if (lane < nn)
                    w.nlist[lane] = e;
                __syncwarp();
            }
            if (nl + ns >= (done ? 1 : 32) || lp >= (FILTER ? kFilterFlush : kFlushParticles)) {
#pragma unroll 1
                for (int part = 0; part < (SLICED ? 2 : 1); ++part) {
                    const int cnt = part ? ns : nl;
                    if (cnt > 0)
                        flush_leaves<PERIODIC, SPLIT, POT, SLICED, FILTER>(
                            w, part ? kList - ns : 0, cnt, part != 0, pos4, t, p, inv2rs, cut, me.x, me.y,
                            me.z, ti, acc, phase, err, o, valid ? ti : -1, npair, evald, lanes);
                }
                nl = ns = lp = 0;
            }
            if (done && nn == 0)
                break;
        }
        if (valid) {
            // the walk's sum is clamped, and so is its sum with a mesh force already in the
            // output (treePmComputeAcceleration, TpmTreeForce.inl:9-25; OctGpu.inl:227); without one
            // the output is only written
            float fx = acc.total(0), fy = acc.total(1), fz = acc.total(2);
            clamp_acceleration(fx, fy, fz, p.max_acc);
            if (p.add_total) {
                fx += o.ax[ti];
                fy += o.ay[ti];
                fz += o.az[ti];
                clamp_acceleration(fx, fy, fz, p.max_acc);
            }
            o.ax[ti] = fx;
            o.ay[ti] = fy;
            o.az[ti] = fz;
            if (POT && o.pot)
                o.pot[ti] = acc.total(3);
            if (o.pair_cnt) {
                o.pair_cnt[ti] = min(npair, kPairSlots);
                if (npair > kPairSlots)
                    raise_error(err, kErrListCapacity);
            }
        }
        const unsigned ev = __reduce_add_sync(kFullMask, valid ? evald : 0u);
        if (lane == 0) {
            if (o.n_pp)
                o.n_pp[g] = cnt_pp;
            if (o.n_pn)
                o.n_pn[g] = cnt_pn;
            if (o.totals) {
                // (of the targets evaluated: in adaptive substeps not the whole group)
                const unsigned long long ng = static_cast<unsigned long long>(gn);
                atomicAdd(&o.totals[0], ng * cnt_pp);
                atomicAdd(&o.totals[1], ng * cnt_pn);
                atomicAdd(&o.totals[2], static_cast<unsigned long long>(ev));
            }
        }
        __syncwarp();
    }
}

struct WalkLaunch {
    int blocks = 0;
    int sms = 0;
    size_t smem = 0;
};

template <bool PERIODIC, bool SPLIT, bool QUAD, bool POT>
WalkLaunch walk_shape(int n, int blocks_per_sm)
{
    // function attributes and occupancy belong to the device: one cached shape per device
    static WalkLaunch cached[kMaxDevices];
    int dev = 0;
    cudaGetDevice(&dev);
    WalkLaunch local;
    WalkLaunch& c = (dev >= 0 && dev < kMaxDevices) ? cached[dev] : local;
    if (c.blocks == 0) {
        const size_t smem = sizeof(WarpSmem<QUAD, walk_filters<SPLIT, QUAD, POT>()>) * kWarps;
        cudaFuncSetAttribute(k_walk<PERIODIC, SPLIT, QUAD, POT>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        int sms = 148, per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk<PERIODIC, SPLIT, QUAD, POT>,
                                                      kWarps * 32, smem);
        c.smem = smem;
        c.sms = sms;
        c.blocks = sms * (per_sm > 0 ? per_sm : 1);
    }
    WalkLaunch l = c;
    if (blocks_per_sm > 0 && l.sms * blocks_per_sm < l.blocks)
        l.blocks = l.sms * blocks_per_sm;
    const int need = (n + kWarps - 1) / kWarps;  // groups <= n
    if (l.blocks > need)
        l.blocks = need < 1 ? 1 : need;
    return l;
}

template <bool PERIODIC, bool SPLIT, bool QUAD, bool POT>
void launch_variant(const float4* pos4, int n, const TreeArrays& t, const GroupTable& g,
                    const WalkParams& p, const WalkOutputs& o, unsigned* queue, int* spill,
                    int* err, cudaStream_t s)
{
    const WalkLaunch l = walk_shape<PERIODIC, SPLIT, QUAD, POT>(n, p.blocks_per_sm);
    const float inv_box = p.box > 0.0f ? 1.0f / p.box : 0.0f;
    count_launch();
    k_walk<PERIODIC, SPLIT, QUAD, POT><<<l.blocks, kWarps * 32, l.smem, s>>>(
        pos4, n, t, g.gstart, g.groot, g.ngroups, g.order, g.ordered, p, inv_box, o, queue, spill, err);
}

template <bool PERIODIC, bool SPLIT>
void dispatch_qp(const float4* pos4, int n, const TreeArrays& t, const GroupTable& g,
                 const WalkParams& p, const WalkOutputs& o, unsigned* queue, int* spill, int* err,
                 cudaStream_t s)
{
    if (p.quadrupole) {
        if (p.want_pot)
            launch_variant<PERIODIC, SPLIT, true, true>(pos4, n, t, g, p, o, queue, spill, err, s);
        else
            launch_variant<PERIODIC, SPLIT, true, false>(pos4, n, t, g, p, o, queue, spill, err, s);
    } else {
        if (p.want_pot)
            launch_variant<PERIODIC, SPLIT, false, true>(pos4, n, t, g, p, o, queue, spill, err, s);
        else
            launch_variant<PERIODIC, SPLIT, false, false>(pos4, n, t, g, p, o, queue, spill, err, s);
    }
}

// ---- reference formulation: the reference's walk on its one-leaf tree, i.e. a direct sum
// over the Morton-sorted order with the reference pair law (rsqrtf, erfcf, expf), FP32
// accumulation in leaf order, then the acceleration clamp (OctGpu.inl:138-227,
// CudForceKernels.inl:7-89).  One thread per particle in original order.
constexpr int kRefThreads = 256;
__global__ void __launch_bounds__(kRefThreads) k_reference_walk(
    const float4* __restrict__ orig, const float4* __restrict__ sorted,
    const uint32_t* __restrict__ sorted_index, int n, float softening, float min_distance2,
    float split_scale, float cutoff2, float max_acc, float* ax, float* ay, float* az)
{
    __shared__ float4 tile[kRefThreads];
    __shared__ int tile_id[kRefThreads];
    const int i = blockIdx.x * kRefThreads + threadIdx.x;
    const float4 self = i < n ? orig[i] : make_float4(0, 0, 0, 0);
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    const bool cutoff = cutoff2 > 0.0f;
    for (int base = 0; base < n; base += kRefThreads) {
        const int j = base + threadIdx.x;
        if (j < n) {
            tile[threadIdx.x] = sorted[j];
            tile_id[threadIdx.x] = static_cast<int>(sorted_index[j]);
        }
        __syncthreads();
        const int m = min(kRefThreads, n - base);
        if (i < n) {
            for (int q = 0; q < m; ++q) {
                if (tile_id[q] == i)
                    continue;
                const float4 s = tile[q];
                if (cutoff) {
                    const float ddx = self.x - s.x, ddy = self.y - s.y, ddz = self.z - s.z;
                    if (ddx * ddx + ddy * ddy + ddz * ddz > cutoff2)
                        continue;
                }
                const float dx = s.x - self.x, dy = s.y - self.y, dz = s.z - self.z;
                const float d2 = dx * dx + dy * dy + dz * dz + softening * softening;
                if (d2 <= min_distance2)
                    continue;
                const float inv = rsqrtf(d2);
                const float inv3 = inv * inv * inv;
                float wgt = 1.0f;
                if (split_scale > 0.0f) {
                    const float dist = 1.0f / inv;
                    const float arg = 0.5f * dist / split_scale;
                    wgt = erfcf(arg) + dist * 0.5641895835477563f / split_scale * expf(-arg * arg);
                }
                const float f = s.w * inv3 * wgt;
                fx += dx * f;
                fy += dy * f;
                fz += dz * f;
            }
        }
        __syncthreads();
    }
    if (i < n) {
        const float norm = sqrtf(fx * fx + fy * fy + fz * fz);
        if (norm > max_acc && norm > 1e-12f) {
            const float sc = max_acc / norm;
            fx *= sc;
            fy *= sc;
            fz *= sc;
        }
        ax[i] = fx;
        ay[i] = fy;
        az[i] = fz;
    }
}

} // namespace

int walk_spill_slots()
{
    // upper bound on concurrently resident warps of any walk variant
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms * (2048 / 32);
}
size_t walk_spill_entries() { return static_cast<size_t>(kSpill); }

void launch_walk(const float4* pos4, int n, const TreeArrays& t, const GroupTable& g,
                 const WalkParams& p, const WalkOutputs& o, unsigned* queue, int* spill, int* err,
                 cudaStream_t s)
{
    const bool periodic = p.box > 0.0f;
    const bool split = p.rsplit > 0.0f;
    if (periodic) {
        if (split)
            dispatch_qp<true, true>(pos4, n, t, g, p, o, queue, spill, err, s);
        else
            dispatch_qp<true, false>(pos4, n, t, g, p, o, queue, spill, err, s);
    } else {
        if (split)
            dispatch_qp<false, true>(pos4, n, t, g, p, o, queue, spill, err, s);
        else
            dispatch_qp<false, false>(pos4, n, t, g, p, o, queue, spill, err, s);
    }
}

void launch_reference_walk(const float4* pos_orig, const float4* pos_sorted,
                           const uint32_t* sorted_index, int n, float softening,
                           float min_distance2, float split_scale, float cutoff2,
                           float max_acceleration, float* ax, float* ay, float* az,
                           cudaStream_t s)
{
    const int blocks = (n + kRefThreads - 1) / kRefThreads;
    count_launch();
    k_reference_walk<<<blocks, kRefThreads, 0, s>>>(pos_orig, pos_sorted, sorted_index, n,
                                                    softening, min_distance2, split_scale,
                                                    cutoff2, max_acceleration, ax, ay, az);
}

} // namespace bz
