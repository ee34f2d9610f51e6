// errbound.cu -- sbr_error_bound: the error, per (angle, frequency) sample, of the
// mixed-precision sweep (FP32 traversal, FP64 path, FP32 phase pairs, fixed-point sums
// of the terms or of FP32 block partials) against the FP64 sweep of the same job.  No counterpart in the reference, which has no
// mixed-precision mode.
//
// A second pass re-traces every ray of the plan with the mixed sweep's own
// arithmetic (start_f and the step of ray.cuh, the watertight test of trace.cuh:
// the same hits bit for bit) while carrying bounds on how far the FP32 ray can be
// from the FP64 ray with the same hits:
//   e   position error across the ray (m): origin rounding, then per bounce the
//       lateral drift t * a, the induced change of t and the FP32 roundings;
//   a   direction error (rad): rounding of -dir, then per reflection twice the
//       error of the FP32 normal (8 u / sin of the triangle's corner angle) + 4 u;
//   dL  path-length error (m): per bounce (e + t a) / |cos i| + 4 u t.
// A ray is re-traced in FP64 when one of its decisions lies within that
// uncertainty of flipping -- a tested triangle whose edge lies within 2 (e + a D)
// of the ray (hit or miss; D = scene diagonal, 2 covers the oblique projection of
// the sheared test), |det| within a factor 2 of the 1e-6 threshold, t within
// dt = 4 m + 4 u (|o| + D) of tMin or of the current closest hit -- or when its
// phase uncertainty 2 k_max dL exceeds 0.05 rad.  Boxes are widened by the same
// margin during this pass, so a near miss inside a culled box is still tested
// (boxes only prune; the closest hit does not change).  For those rays the exact
// difference of the FP64 and mixed terms is summed per sample (Delta_k).  The other
// rays differ from FP64 only by rounding, |d term| <= scale_k (amp 2 k dL + amp eps
// + damp), damp = 2 R^n (dn_last + a).  Part of those errors is the same for every
// ray that sees the same geometry the same way (a face-on plate): the relative error
// of t from the approximate reciprocals of the triangle test (bounded by 8 u t per
// bounce, dLs) and the error of the sine / cosine approximation (eps).  That shared
// part adds coherently, so it is bounded by the field itself times its
// amp-weighted mean, |S_k| (2 k c1 + eps) with c1 = sum amp dLs / sum amp.  The rest
// (origin, hit-point and direction rounding) varies from ray to ray as independent,
// zero-mean errors, bounded with the probabilistic rounding-error bound of Higham
// and Mary (SIAM J. Sci. Comput. 41(5), 2019): |sum| <= lambda sqrt(sum of squares),
// exceeded with probability below 4 exp(-lambda^2 / 2) (lambda = 6: 6e-8).  Per
// sample
//   E_k = |Delta_k| + |S_k| (2 k c1 + eps) + lambda scale_k (2 k sqrt(Q1) + sqrt(Q0))
//         + fixed_k + lambda scale_k u sqrt(Q2),
// Q1 = sum (amp (dL - dLs))^2, Q0 = sum damp^2 over the rounding-only rays.  fixed_k
// covers the sweep's fixed-point sums: each of the N rays (or each group of them) is
// rounded once, within half a unit of the sample in the real and in the imaginary part,
// whatever items and launches it ran in.  Roundings of different terms count as
// independent: lambda sqrt(N / 2) units, and one for the final conversion.  fixed_k is
// the larger of that and 2^-60 of the field's bound per run of blocks, which covers it
// from about 1,150 rays on and is what a statement of the same run always held.  Equal
// terms round equally, by at most sqrt(1/2) N units in all; that part adds coherently, as
// the share sqrt(1/2) N units / (scale_k sum amp) of the field, and belongs to eps, which
// has 3.4e-7 over its other parts (a sweep of 10^6 rays of full amplitude needs 2e-13; it
// grows with max(1, R)^max_bounces).  The last term covers
// the FP32 partial sums of the lane-owned epilogue: each term of a 4x8 ray block is
// added to its channel's FP32 partial by one FMA, rounded within u |partial|, and
// every partial is within A_b = sum |amp| of the block, so Q2 = sum over blocks of
// n_b A_b^2 (n_b terms); the per-lane layouts round each term and the term only
// overstates their error.  The phase pair's 2^-45 |x| turns (ray.cuh, turns_frac)
// is added to dLs as 2^-45 L.
#include <algorithm>
#include <cmath>
#include <vector>

#include "plan.hpp"
#include "ray.cuh"

namespace sbr {
namespace {

constexpr float kU = 5.9604644775390625e-08f;  // 2^-24, unit roundoff of FP32
// Phase / amplitude error of one mixed term: the rounding of the FP32 remainder of
// 2 k L in turns (2 pi 2^-25 rad; the FP32 pair's 2^-45 |x| is carried in dLs),
// __sincosf (below 4e-7 absolute), FP32 amplitude (2^-24).
constexpr double kPhaseEps = 1.0e-6;
constexpr double kPhaseParts = 6.6e-7;  // the sum of these

constexpr double kPhaseExact = 0.05;  // rad: rays with more phase uncertainty are re-traced in FP64
constexpr double kLambda = 6.0;       // probabilistic bound multiplier (failure below 6e-8)

// A ray bound for the FP64 re-trace, and its mixed term.
struct Flagged {
    int32_t seg, i, j;
    float amp, Lh, Ll;
};
constexpr long long kFlaggedMax = 16ll << 20;  // rays of one launch: all of them may be flagged

struct ErrParams {
    SceneView S;
    const Segment* segs;
    const int64_t* seg_item_base;
    int32_t n_segs;
    const JobConst* jobs;
    const FreqConst* freqs;
    int64_t item_begin, n_items;   // items of this launch: [item_begin, n_items)
    unsigned long long* queue;
    Flagged* flagged;              // [rays of a launch]
    unsigned long long* n_flagged;
    double* acc;       // [n_segs][8]: sum amp, sum amp dLs, Q2, Q1, Q0, re-traced rays, rays, -
    double* dfield;    // [n_samples][2]: sum of (FP64 term - mixed term) of the re-traced rays
    float diag;        // scene bounding-box diagonal (m)
    uint32_t* err;
    const volatile int32_t* cancel;
};

__device__ __forceinline__ float norm1(F3 v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z); }

// The watertight test of trace.cuh (wt_tri, identical decisions), flagging in `amb`
// a decision within the margin m (edges) / dt (t) of flipping.
template <int KZ>
__device__ __forceinline__ bool wt_tri_flag(const GTri& T, F3 o, const WtRay& w, float tMin, float tMax, float m,
                                            float dt, float& t, bool& amb) {
    constexpr int KX = (KZ + 1) % 3, KY = (KZ + 2) % 3;
    const float ox = axis<KX>(o), oy = axis<KY>(o), oz = axis<KZ>(o);
    const float az = __fsub_rn(axis<KZ>(T.v0), oz), bz = __fsub_rn(axis<KZ>(T.v1), oz),
                cz = __fsub_rn(axis<KZ>(T.v2), oz);
    const float ax = __fmaf_rn(-w.sx, az, __fsub_rn(axis<KX>(T.v0), ox));
    const float ay = __fmaf_rn(-w.sy, az, __fsub_rn(axis<KY>(T.v0), oy));
    const float bx = __fmaf_rn(-w.sx, bz, __fsub_rn(axis<KX>(T.v1), ox));
    const float by = __fmaf_rn(-w.sy, bz, __fsub_rn(axis<KY>(T.v1), oy));
    const float cx = __fmaf_rn(-w.sx, cz, __fsub_rn(axis<KX>(T.v2), ox));
    const float cy = __fmaf_rn(-w.sy, cz, __fsub_rn(axis<KY>(T.v2), oy));
    float U = __fsub_rn(__fmul_rn(cx, by), __fmul_rn(cy, bx));
    float V = __fsub_rn(__fmul_rn(ax, cy), __fmul_rn(ay, cx));
    float W = __fsub_rn(__fmul_rn(bx, ay), __fmul_rn(by, ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = float(__dsub_rn(__dmul_rn(cx, by), __dmul_rn(cy, bx)));
        V = float(__dsub_rn(__dmul_rn(ax, cy), __dmul_rn(ay, cx)));
        W = float(__dsub_rn(__dmul_rn(bx, ay), __dmul_rn(by, ax)));
    }
    const bool inside = !((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f));
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    const float T3 = __fmaf_rn(U, az, __fmaf_rn(V, bz, __fmul_rn(W, cz)));
    const float tp = det != 0.0f ? T3 * w.sz / det : 0.0f;
    const bool inRange = tp >= tMin - dt && tp <= tMax + dt;
    if (inRange && !amb) {
        // margins: distance (sheared plane) from the ray to each edge line
        const float dU = fabsf(U) * rhypotf(cx - bx, cy - by), dV = fabsf(V) * rhypotf(ax - cx, ay - cy),
                    dW = fabsf(W) * rhypotf(bx - ax, by - ay);
        if (inside) {
            if (fminf(dU, fminf(dV, dW)) < m) amb = true;
        } else {
            // the ray is outside across the edges whose function disagrees with the
            // orientation; it would be inside if each of those moved by less than m
            const bool pos = det >= 0.0f;
            const bool vU = pos ? U < 0.0f : U > 0.0f, vV = pos ? V < 0.0f : V > 0.0f, vW = pos ? W < 0.0f : W > 0.0f;
            if ((!vU || dU < m) && (!vV || dV < m) && (!vW || dW < m)) amb = true;
        }
        const float adet = fabsf(det) * w.adz;
        if (adet >= 0.5e-6f && adet < 2.0e-6f) amb = true;
    }
    if (!inside) return false;
    if (!(fabsf(det) * w.adz >= 1.0e-6f)) return false;
    float rdet;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rdet) : "f"(det));
    const float tt = __fmul_rn(__fmul_rn(T3, w.sz), rdet);
    if (fabsf(tt - tMin) < dt || fabsf(tt - tMax) < dt) amb = true;
    if (!(tt >= tMin && tt <= tMax)) return false;
    t = tt;
    return true;
}

template <int KZ>
__device__ __forceinline__ void leaf_flag(const GTri* __restrict__ tris, const int32_t* tie, int first, int cnt, F3 o,
                                          const WtRay& w, float tMin, float m, float dt, float& tBest, int& best,
                                          bool& amb) {
    for (int k = 0; k < cnt; ++k) {
        float tt;
        if (wt_tri_flag<KZ>(tris[first + k], o, w, tMin, tBest, m, dt, tt, amb) &&
            replaces(tt, first + k, tBest, best, tie)) {
            tBest = tt;
            best = first + k;
        }
    }
}

// Closest hit as Walker<false> finds it (4-wide nodes, watertight test), with every
// box widened by m across the ray and dt along it, and decisions near flipping
// flagged in `amb`.
__device__ int closest_flag(const SceneView& S, F3 o, F3 d, float tMin, float& tBest, float m, float dt, bool& amb,
                            uint32_t& err) {
    const F3 inv{slab_inv(d.x), slab_inv(d.y), slab_inv(d.z)};
    const WtRay wr = wt_ray(d);
    const F3 oi{o.x * inv.x, o.y * inv.y, o.z * inv.z};
    const float px = m * fabsf(inv.x), py = m * fabsf(inv.y), pz = m * fabsf(inv.z);
    const unsigned onx = inv.x < 0.0f ? 16u : 0u, ony = inv.y < 0.0f ? 48u : 32u, onz = inv.z < 0.0f ? 80u : 64u;
    const unsigned ofx = onx ^ 16u, ofy = ony ^ 16u, ofz = onz ^ 16u;
    unsigned long long stack[kStackDepth];
    int sp = 0, ref = 0, best = -1;
    uint32_t iters = 0;
    auto plane = [](const GNode4* p, unsigned off) {
        return __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const char*>(p) + off));
    };
    auto slab = [&](float nx, float fx, float ny, float fy, float nz, float fz, bool& hit) {
        const float tn = max3f(fmaf(nx, inv.x, -oi.x) - px, fmaf(ny, inv.y, -oi.y) - py,
                               fmaxf(fmaf(nz, inv.z, -oi.z) - pz, tMin - dt));
        const float tf = min3f(fmaf(fx, inv.x, -oi.x) + px, fmaf(fy, inv.y, -oi.y) + py,
                               fminf(fmaf(fz, inv.z, -oi.z) + pz, tBest + dt));
        hit = tn <= tf * kSlabSlack;
        return tn;
    };
    auto pop = [&]() {
        while (sp > 0) {
            const unsigned long long e = stack[--sp];
            if (__uint_as_float((unsigned)(e >> 32)) <= tBest + dt) { ref = (int)(unsigned)e; return true; }
        }
        return false;
    };
    auto push = [&](int r, float t) {
        if (sp < kStackDepth) stack[sp++] = pack_entry(r, t);
        else err |= DEV_ERR_STACK;
    };
    // nodes until every lane of the warp has a leaf (or is done), then leaves: taking each
    // lane's leaf as it comes ran the triangle tests on a few lanes at a time (11.6 -> 8.5 ms)
    for (;;) {
        while (ref >= 0) {
            if (++iters > kIterBudget) { err |= DEV_ERR_BUDGET; return -1; }
            const GNode4* np = S.nodes + ref;
            const float4 nx = plane(np, onx), fx = plane(np, ofx), ny = plane(np, ony), fy = plane(np, ofy);
            const float4 nz = plane(np, onz), fz = plane(np, ofz);
            const int4 ch = __ldg(&np->child);
            bool h[4];
            float t[4] = {slab(nx.x, fx.x, ny.x, fy.x, nz.x, fz.x, h[0]), slab(nx.y, fx.y, ny.y, fy.y, nz.y, fz.y, h[1]),
                          slab(nx.z, fx.z, ny.z, fy.z, nz.z, fz.z, h[2]), slab(nx.w, fx.w, ny.w, fy.w, nz.w, fz.w, h[3])};
            int c[4] = {ch.x, ch.y, ch.z, ch.w};
            const int nh = int(h[0]) + int(h[1]) + int(h[2]) + int(h[3]);
            // the nearest accepted child next, the others pushed, farthest first; where
            // the nearest lies beyond the closest hit (by the slab's slack) they all do
            bool enter = false;
            if (nh == 1) {
                ref = h[0] ? c[0] : h[1] ? c[1] : h[2] ? c[2] : c[3];
                enter = (h[0] ? t[0] : h[1] ? t[1] : h[2] ? t[2] : t[3]) <= tBest + dt;
            } else if (nh > 1) {
                const float inf = __int_as_float(0x7f800000);
#pragma unroll
                for (int k = 0; k < 4; ++k) t[k] = h[k] ? t[k] : inf;
                sort4(t, c);
                enter = t[0] <= tBest + dt;
                if (enter) {
                    if (nh > 3) push(c[3], t[3]);
                    if (nh > 2) push(c[2], t[2]);
                    push(c[1], t[1]);
                    ref = c[0];
                }
            }
            if (!enter && !pop()) return best;
        }
        do {
            if (++iters > kIterBudget) { err |= DEV_ERR_BUDGET; return -1; }
            const int code = ~ref;
            const int first = code >> 4, cnt = code & 15;
            switch (wr.kz) {
                case 0: leaf_flag<0>(S.tris, S.tie, first, cnt, o, wr, tMin, m, dt, tBest, best, amb); break;
                case 1: leaf_flag<1>(S.tris, S.tie, first, cnt, o, wr, tMin, m, dt, tBest, best, amb); break;
                default: leaf_flag<2>(S.tris, S.tie, first, cnt, o, wr, tMin, m, dt, tBest, best, amb); break;
            }
            if (!pop()) return best;
        } while (ref < 0);
    }
}

// One ray: the mixed sweep's path (start_f, then step_f's arithmetic per bounce)
// with the uncertainty bounds carried along; rays near a decision or with a large
// phase uncertainty are listed for the FP64 re-trace, the others add to the lane's sums of
// squares.
// Returns the amplitude the sweep adds for the ray (0 when it adds nothing).
__device__ __forceinline__ float ray_bound(const ErrParams& P, int seg, const Segment& G, const JobConst& J,
                                         double kmax, int i, int j, bool valid, double& sa, double& s1, double& q1,
                                         double& s0, unsigned& nex, uint32_t& err) {
    RayF r;
    r.count = 0;
    r.o = f3(0, 0, 0);
    if (valid) start_f<SBR_PREC_MIXED>(r, G, J, i, j);
    float ue = 2.0f * kU * norm1(r.o);  // origin formed in FP64, rounded to FP32
    float ua = 2.0f * kU;                // FP32 direction
    double dL = double(kU * norm1(r.o));
    double dLs = 0.0;  // the part shared by rays seeing the same geometry the same way
    float dnl = 0.0f;
    bool amb = false;
    // one query per step for the whole warp: on their own the lanes drift apart, one in its
    // first query while another is in its second, and run nearly one at a time (61 looks at
    // a 200k-triangle ellipsoid, 8.5 -> 3.0 ms)
    bool walking = valid && J.max_bounces > 0;
    while (__any_sync(0xffffffffu, walking)) {
        if (!walking) continue;
        // a ray already bound for the FP64 re-trace needs no more margins: it walks
        // unpadded (its uncertainty can grow to metres after a grazing bounce, and
        // boxes widened that far would open most of the tree)
        const bool exact = amb || 2.0 * kmax * dL > kPhaseExact;
        const float m = exact ? 0.0f : 2.0f * (ue + ua * P.diag);
        const float dt = exact ? 0.0f : 4.0f * m + 4.0f * kU * (norm1(r.o) + P.diag);
        float tB = 1e20f;
        const int slot = closest_flag(P.S, r.o, r.d, 1.0e-3f, tB, m, dt, amb, err);
        walking = slot >= 0;
        if (!walking) continue;
        const GTri T = P.S.tris[slot];
        const F3 n = f3(T.v0.w, T.v1.w, T.v2.w);
        // the step of step_f (ray.cuh), operation for operation
        r.cosl = dot(n, f3(-r.d.x, -r.d.y, -r.d.z));
        r.nl = n;
        r.dl = r.d;
        ++r.count;
        r.L += double(tB);
        const F3 p = fma3(tB, r.d, r.o);
        r.d = reflect_dir(r.d, n);
        r.o = nudge(p, n);
        // uncertainty of this bounce
        const F3 e1 = f3(T.v1.x - T.v0.x, T.v1.y - T.v0.y, T.v1.z - T.v0.z);
        const F3 e2 = f3(T.v2.x - T.v0.x, T.v2.y - T.v0.y, T.v2.z - T.v0.z);
        const F3 N = cross(e1, e2);
        const float sinang = sqrtf(dot(N, N) / fmaxf(dot(e1, e1) * dot(e2, e2), 1e-30f));
        const float dnrm = 8.0f * kU / fmaxf(sinang, 1e-6f);
        const float ci = fmaxf(fabsf(r.cosl), 1e-6f);
        const float dtb = (ue + tB * ua) / ci + 8.0f * kU * tB;
        dL += double(dtb);
        dLs += double(8.0f * kU * tB);
        ue = ue + tB * ua + dtb + 2.0f * kU * norm1(p) + 1.0e-4f * dnrm;
        ua = ua + 2.0f * dnrm + 4.0f * kU;
        dnl = dnrm;
        walking = r.count < J.max_bounces;
    }
    if (!valid) return 0.0f;
    const RayOut om = finish_f<SBR_PREC_MIXED>(r, J);
    dLs += ldexp(om.L, -45);  // the FP32 phase pair (ray.cuh, turns_frac)
    dL += ldexp(om.L, -45);
    if (amb || (r.count > 0 && 2.0 * kmax * dL > kPhaseExact)) {
        // left to k_exact: the FP64 walk of a few lanes would hold up the other rays' warps
        P.flagged[atomicAdd(P.n_flagged, 1ull)] = Flagged{seg, i, j, om.amp, om.Lh, om.Ll};
        ++nex;
    } else if (r.count > 0) {
        const double amp = double(fabsf(om.amp));  // (negative with a negative R and an odd count)
        sa += amp;
        s1 += amp * dLs;
        const double e1 = amp * (dL - dLs), e0 = 2.0 * double(fabsf(om.Rn)) * double(dnl + ua);
        q1 += e1 * e1;
        s0 += e0 * e0;
    }
    return om.amp;
}

// One flagged ray per lane: the FP64 sweep's own ray (start_d / step_d), a query per step
// for the whole warp, and per frequency the difference of its term and the mixed one.  As
// a kernel of its own it runs on full warps: inside k_errbound the flagged rays of a block,
// a few of its 32, walked while the others waited (61 looks at a 200k-triangle ellipsoid
// 12.7 -> 11.6 ms; k_exact itself 0.3 ms of the 3.0 of the whole pass).
__global__ void __launch_bounds__(kCtaThreads, 8) k_exact(const ErrParams P) {
    constexpr unsigned FULL = 0xffffffffu;
    uint32_t err = 0;
    const unsigned long long n = *P.n_flagged;
    const int lane = threadIdx.x & 31;
    for (unsigned long long first = blockIdx.x * (unsigned long long)kCtaThreads + (threadIdx.x & ~31); first < n;
         first += (unsigned long long)gridDim.x * kCtaThreads) {
        const bool valid = first + lane < n;
        const Flagged f = P.flagged[valid ? first + lane : first];
        const Segment& G = P.segs[f.seg];
        const JobConst J = P.jobs[G.job];
        const FreqConst* F = P.freqs + J.freq_base;
        RayD rd;
        PolD ed;
        start_d(rd, G, J, f.i, f.j);
        bool walking = valid && J.max_bounces > 0;
        while (__any_sync(FULL, walking))
            if (walking) walking = !step_d<false, false>(rd, ed, P.S, J.max_bounces, err, nullptr);
        if (!valid) continue;
        const RayOut od = finish_d(rd, J);
        RayOut om;
        om.amp = f.amp;
        om.Lh = f.Lh;
        om.Ll = f.Ll;
        for (int q = 0; q < J.n_freqs; ++q) {
            double re = 0.0, im = 0.0, rm = 0.0, imm = 0.0;
            if (od.amp != 0.0f) po_term(SBR_PREC_FP64, F[q], od, re, im);
            if (om.amp != 0.0f) po_term(SBR_PREC_MIXED, F[q], om, rm, imm);
            re -= rm * F[q].scale;  // mixed terms are summed without k A / (4 pi)
            im -= imm * F[q].scale;
            if (re != 0.0 || im != 0.0) {
                atomicAdd(P.dfield + 2 * (G.sample_base + q), re);
                atomicAdd(P.dfield + 2 * (G.sample_base + q) + 1, im);
            }
        }
    }
    if (err) atomicOr(P.err, err);
}

__global__ void __launch_bounds__(kCtaThreads, 8) k_errbound(const ErrParams P) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint32_t err = 0;
    for (;;) {
        long long item = 0;
        if (lane == 0) {
            item = P.item_begin + (long long)atomicAdd(P.queue, 1ull);
            if (item < P.n_items && P.cancel && *P.cancel != 0) {
                atomicOr(P.err, DEV_ERR_CANCEL);
                item = P.n_items;
            }
        }
        item = __shfl_sync(FULL, item, 0);
        if (item >= P.n_items) break;
        const int seg = find_segment(P.seg_item_base, P.n_segs, item);
        const Segment& G = P.segs[seg];
        const JobConst J = P.jobs[G.job];
        const FreqConst* F = P.freqs + J.freq_base;
        double kmax = 0.0;
        for (int k = 0; k < J.n_freqs; ++k) kmax = fmax(kmax, F[k].k);
        const Run run = item_run(G, item, false);
        const int b0 = run.first, b1 = run.first + run.count;
        double sa = 0.0, s1 = 0.0, q1 = 0.0, s0 = 0.0, q2 = 0.0;
        unsigned nex = 0, nray = 0;
        for (int blk = b0; blk < b1; ++blk) {
            const int i = G.i0 + (blk % G.blocks_x) * kBlockW + (lane % kBlockW);
            const int j = G.j0 + (blk / G.blocks_x) * kBlockH + (lane / kBlockW);
            const bool valid = i < G.i0 + G.ni && j < G.j0 + G.nj;
            const float am = ray_bound(P, seg, G, J, kmax, i, j, valid, sa, s1, q1, s0, nex, err);
            nray += valid;
            // the block's FP32 partial sums: n_b terms, every partial within A_b
            double ab = double(fabsf(am));
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) ab += __shfl_xor_sync(FULL, ab, off);
            const int nb = __popc(__ballot_sync(FULL, am != 0.0f));
            if (lane == 0) q2 += double(nb) * ab * ab;
        }
        for (int off = 16; off > 0; off >>= 1) {
            sa += __shfl_xor_sync(FULL, sa, off);
            s1 += __shfl_xor_sync(FULL, s1, off);
            q1 += __shfl_xor_sync(FULL, q1, off);
            s0 += __shfl_xor_sync(FULL, s0, off);
            q2 += __shfl_xor_sync(FULL, q2, off);
        }
        nex = __reduce_add_sync(FULL, nex);
        nray = __reduce_add_sync(FULL, nray);
        if (lane == 0) {
            double* A = P.acc + 8 * seg;
            atomicAdd(A, sa);
            atomicAdd(A + 1, s1);
            atomicAdd(A + 2, q2);
            atomicAdd(A + 3, q1);  // sums of squares of independent per-ray bounds
            atomicAdd(A + 4, s0);
            atomicAdd(A + 5, double(nex));
            atomicAdd(A + 6, double(nray));
        }
    }
    if (err) atomicOr(P.err, err);
}

}  // namespace
}  // namespace sbr

extern "C" sbr_status sbr_error_bound(sbr_scene* s, const sbr_job* jobs, size_t n_jobs, const sbr_run_opts* opts,
                                      const double* field, double* err_field, double* err_db) {
    using namespace sbr;
    if (!s || (!jobs && n_jobs) || !field) return fail(SBR_ERR_INVALID_ARG, "scene, jobs and field are required");
    sbr_run_opts o{};
    if (opts) o = *opts;
    if (o.precision != SBR_PREC_MIXED)
        return fail(SBR_ERR_UNSUPPORTED, "the error bound is stated for SBR_PREC_MIXED results");
    if (o.polarization != SBR_POL_SCALAR) return fail(SBR_ERR_UNSUPPORTED, "the error bound covers the scalar field");
    o.mode = SBR_MODE_BATCHED;
    o.first_hit = SBR_FIRST_HIT_TRAVERSE;
    o.use_graph = 0;
    o.autotune = 0;
    DeviceGuard device_guard;
    SBR_CUDA(cudaSetDevice(s->device));
    sbr_status st = ensure_fp64(s);  // the re-traced rays walk the FP64 triangles
    if (st != SBR_OK) return st;
    sbr_plan* p = nullptr;
    st = sbr_plan_create(s, jobs, n_jobs, &o, &p);
    if (st != SBR_OK) return st;
    double* d_acc = nullptr;
    double* d_dfield = nullptr;
    unsigned long long* d_queue = nullptr;
    std::vector<int32_t> run_blocks;  // the most blocks an item of each segment has
    for (const Segment& g : p->segs) run_blocks.push_back(g.parts > 1 ? g.part_blocks : g.blocks_per_item);
    std::vector<double> acc(8 * (size_t)std::max<int64_t>(p->n_segs, 1), 0.0);
    std::vector<double> dfield(2 * (size_t)std::max<int64_t>(p->n_samples, 1), 0.0);
    Parts parts;
    const size_t acc_at = parts.add(acc.size() * sizeof(double)), df_at = parts.add(dfield.size() * sizeof(double)),
                 queue_at = parts.add(2 * sizeof(unsigned long long)), zero_b = parts.add(0);
    // a launch takes as many items as the list of flagged rays has room for, which is
    // halved until the device has the memory
    const long long run = std::max<int64_t>(1, p->n_items > 0 ? *std::max_element(run_blocks.begin(), run_blocks.end()) : 1);
    long long per_launch = std::max<long long>(1, std::min<long long>(p->n_items, kFlaggedMax / (32 * run)));
    const size_t flag_at = parts.add(0);
    char* block = nullptr;
    cudaError_t e;
    while ((e = pool_alloc(p->device, &block, flag_at + (size_t)(per_launch * run * 32) * sizeof(Flagged))) ==
               cudaErrorMemoryAllocation && per_launch > 1)
        per_launch = (per_launch + 1) / 2;
    if (e != cudaSuccess) st = fail(SBR_ERR_OOM, "error-bound accumulators");
    if (st == SBR_OK) {
        d_acc = reinterpret_cast<double*>(block + acc_at);
        d_dfield = reinterpret_cast<double*>(block + df_at);
        d_queue = reinterpret_cast<unsigned long long*>(block + queue_at);
        e = cudaMemsetAsync(block, 0, zero_b, p->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "error-bound clear");
    }
    if (st == SBR_OK && p->n_items > 0) {
        ErrParams P{};
        P.S = s->view();
        P.freqs = p->d_freqs;
        P.dfield = d_dfield;
        P.segs = p->d_segs;
        P.seg_item_base = p->d_seg_base;
        P.n_segs = (int32_t)p->n_segs;
        P.jobs = p->d_jobs;
        P.queue = d_queue;
        P.n_flagged = d_queue + 1;
        P.flagged = reinterpret_cast<Flagged*>(block + flag_at);
        P.acc = d_acc;
        const double dx = s->aabb_hi[0] - s->aabb_lo[0], dy = s->aabb_hi[1] - s->aabb_lo[1],
                     dz = s->aabb_hi[2] - s->aabb_lo[2];
        P.diag = float(std::sqrt(dx * dx + dy * dy + dz * dz));
        P.err = p->d_err;
        P.cancel = p->d_cancel;
        int occ = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_errbound, kCtaThreads, 0);
        if (e != cudaSuccess) st = cuda_fail(e, "occupancy");
        if (st == SBR_OK) {
            for (long long at = 0; at < p->n_items && e == cudaSuccess; at += per_launch) {
                P.item_begin = at;
                P.n_items = std::min<long long>(p->n_items, at + per_launch);
                if (at > 0) e = cudaMemsetAsync(d_queue, 0, 2 * sizeof(unsigned long long), p->stream);
                if (e != cudaSuccess) break;
                const long long grid = std::min<long long>((long long)std::max(occ, 1) * p->num_sms, (P.n_items - at + 3) / 4);
                k_errbound<<<(unsigned)std::max(grid, 1LL), kCtaThreads, 0, p->stream>>>(P);
                const long long most = (per_launch * run * 32 + kCtaThreads - 1) / kCtaThreads;
                k_exact<<<(unsigned)std::min<long long>(most, 8ll * p->num_sms), kCtaThreads, 0, p->stream>>>(P);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) e = cudaStreamSynchronize(p->stream);
            if (e != cudaSuccess) st = cuda_fail(e, "error-bound pass");
        }
        if (st == SBR_OK) {
            uint32_t de = 0;
            e = cudaMemcpy(&de, p->d_err, sizeof(de), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) st = cuda_fail(e, "error word");
            else if (de) {
                clear_device_word(p->d_err);
                st = (de & DEV_ERR_CANCEL) ? fail(SBR_ERR_CANCELLED, "run cancelled")
                     : (de & DEV_ERR_BUDGET) ? fail(SBR_ERR_TIMEOUT, "traversal iteration budget exceeded")
                                             : fail(SBR_ERR_STACK, "traversal stack overflow");
            }
        }
    }
    if (st == SBR_OK) {
        e = cudaMemcpy(acc.data(), d_acc, acc.size() * sizeof(double), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(dfield.data(), d_dfield, dfield.size() * sizeof(double),
                                             cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) st = cuda_fail(e, "error-bound copy");
    }
    if (st == SBR_OK) {
        for (int64_t g = 0; g < p->n_segs; ++g) {
            const Segment& G = p->segs[(size_t)g];
            const JobConst& J = p->jobs[(size_t)G.job];
            // the fixed-point term in units of the job
            const int run = o.blocks_per_item > 0 ? G.blocks_per_item : auto_run(G.blocks);
            const int64_t runs = (G.blocks + run - 1) / run;
            const double rays = double((int64_t)G.ni * G.nj);
            const double fixed = std::max(4.0 * double(runs + 1), (kLambda * std::sqrt(0.5 * rays) + 1.0) / double(G.finer));
            for (int k = 0; k < J.n_freqs; ++k) {
                const FreqConst& F = p->freqs[(size_t)(J.freq_base + k)];
                const int64_t smp = G.sample_base + k;
                const double* A = acc.data() + 8 * g;
                const double a = std::hypot(field[2 * smp], field[2 * smp + 1]);
                const double equal = std::sqrt(0.5) * rays * (F.quantum / double(G.finer)) / F.scale;  // of equal terms, times sum amp
                const double shared = a * (A[0] > 0.0 ? 2.0 * F.k * A[1] / A[0] + std::max(kPhaseEps, kPhaseParts + equal / A[0])
                                                      : kPhaseEps);
                const double E = std::hypot(dfield[2 * smp], dfield[2 * smp + 1]) + shared +
                                 kLambda * F.scale * (2.0 * F.k * std::sqrt(A[3]) + std::sqrt(A[4])) +
                                 fixed * F.quantum + kLambda * F.scale * double(kU) * std::sqrt(A[2]);
                if (err_field) err_field[smp] = E;
                if (err_db) {
                    const double db = 10.0 * std::log10(std::max(4.0 * M_PI * a * a, 1e-10));
                    const double hi = 10.0 * std::log10(std::max(4.0 * M_PI * (a + E) * (a + E), 1e-10));
                    const double lo_a = std::max(a - E, 0.0);
                    const double lo = 10.0 * std::log10(std::max(4.0 * M_PI * lo_a * lo_a, 1e-10));
                    err_db[smp] = std::max(hi - db, db - lo);
                }
            }
        }
    }
    if (cudaStreamSynchronize(p->stream) != cudaSuccess) cudaDeviceSynchronize();
    pool_free(p->device, block);
    sbr_plan_destroy(p);
    return st;
}
