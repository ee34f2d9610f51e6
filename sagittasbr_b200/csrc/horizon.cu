// horizon.cu -- per-triangle horizons: above which elevation a ray that leaves a
// triangle's front side meets nothing any more.  No counterpart in the reference,
// which walks its tree for every reflected ray.
//
// Most rays that a body reflects escape (on the 2.15 M-triangle aircraft 93 % of the
// second queries miss), and such a miss is the dearest query there is: the ray starts
// inside every box around its hit point and no hit ever prunes its walk (78 of the
// 202 ms of a 61-azimuth, 64-frequency sweep were second queries).  For every leaf
// slot and every octant of directions (the signs of d) this pass bounds
//     H = sup d.n   over the directions d of that octant in which a ray from the
//                   triangle can meet any triangle of the scene at t >= tMin,
// and stores it as a byte, rounded up.  A reflected ray with d.n above its triangle's
// byte is known to miss without a walk; every other ray walks as before.  The bound
// is conservative, so hits, counters and fields stay the same bit for bit.
//
// A ray leaves from o = p + 1e-4 n + e, p on the triangle T, and meets q at o + t d
// with t >= 1e-3.  With h = (q - p).n that gives d.n = (h - 1e-4 - e.n) / t, so a
// triangle X bounds d.n by
//   A  max over X of (h - c) / max(1e-3, dist(T, X) - |o - p|),  c = 1e-4 - |e.n|;
//   B  r / sqrt(1 + r^2), r = max over the vertices of X of (h - c) / (f - |e|), where
//      f is the distance from T along an in-plane direction w that has X beyond T
//      (h - c and f - |e| are affine on X, so their ratio is largest at a vertex, and
//      vertices shared with T, where f = 0 and h < c, only lower it).  B is what makes
//      the neighbours' bound their slope instead of 1.
// |e| covers what the sweep's FP32 hit points can be off: t of the watertight test and
// the hit point's rounding, 12 u t across the plane and 18 u t along it for d.n >= 0.1
// (t is at most the scene's diagonal: the launch plane stands just outside the scene).
// Triangles whose FP32 normal is uncertain by more than 4e-3, whose vertices are not
// flat to the tolerance, or scenes so large that |e| reaches the 1e-4 nudge get no
// horizon.  The FP32 mode's Moller-Trumbore test can report hits well outside a
// triangle near grazing incidence, so that mode does not use horizons.
//
// A scene starts without horizons (all bytes 255: every ray walks) and gets them, in the
// stream of the sweep that needs them, once its sweeps have launched kHorizonRays rays per
// triangle.  They cost 5 to 15 ns a triangle and save 2 to 130 ps a launched ray (break-even
// at 60 rays per triangle on a smooth ellipsoid, 120 on a small sphere, 650 on a coarse
// aircraft, 3,900 on a fine jittered one seen from the nose), and a ray costs 30 to 100 ps:
// by then a scene's sweeps have taken 45 to 150 ns a triangle, so the build is 3 to 33 % of
// them once.  It falls on the sweep that reaches the count, however short that one is (a
// single look at the full-size aircraft can take 21 ms longer).  A first look at a new
// model, or a step that moves the vertices again, does not pay for what it cannot use (at
// 200 a first sweep took up to 36 % longer).
// The bytes change in place: a plan or graph made before reads them too, and a kernel that
// runs meanwhile sees 255 or the final byte.
//
// The search walks the 4-wide tree once per triangle, children with the largest bound
// first, and drops a box when its bound A is below the octants' current H or below
// kFloor; a box seen under less than kAccept is taken by its bound instead of being
// opened.  One thread per slot: neighbouring slots are neighbouring triangles, so a
// warp's walks stay together (mean visits 126, mean of a warp's longest 198 on the
// aircraft).  Bound by the bounds' arithmetic, 9.8 ns a triangle there (21 ms;
// 0.3 ms for a 20k-triangle sphere).  Measured on the aircraft's
// 10 azimuths from the nose, floor / accept: 0.1 / 0.12 35.9 ms and 52.6 M of the 80.6 M
// second queries still walked, 0.1 / 0.25 22.2 ms and 53.2 M, 0.15 / 0.25 21.0 ms and
// 54.1 M, 0.2 / 0.25 19.7 ms and 55.5 M; broadside 30 % still walk.
//
// Measured on B200, second and later queries of a sweep (360 sphere looks: 0.26 -> 0.05
// ms; narrow 181-azimuth aircraft, 133k triangles: 6.5 -> 3.5 ms; ellipsoid, 121 looks:
// 1.17 -> 0.36 ms).
#include <cmath>

#include "plan.hpp"
#include "ray.cuh"

namespace sbr {
namespace {

constexpr float kFloor = 0.15f;      // smallest horizon told apart
constexpr unsigned kTop = 229;       // byte (0.9) from which a direction counts as blocked
constexpr float kAccept = 0.25f;     // diagonal / (2 distance) below which a box is not opened
constexpr int64_t kHorizonRays = 1500; // launched rays per triangle from which a scene has them
constexpr int kVisits = 4096;        // node visits per triangle before it is given up (blocked)
constexpr float kU32 = 5.9604644775390625e-08f;  // 2^-24

// Horizons of the eight octants as bytes, octant k (bit 0: d.x < 0, bit 1: d.y < 0,
// bit 2: d.z < 0) in byte k & 3 of word k >> 2.
struct Oct {
    unsigned a, b;
};

struct HorizonTri {
    F3 a, n;           // first vertex, unit normal
    F3 lo, hi;         // bounds
    F3 g;              // centroid
    float rad;         // radius about it
    float off;         // added to (q - a).n: flatness - c
    float el;          // |e| along the plane
    float eo;          // |o - p|
    F3 w[6];           // in-plane unit directions: outward of the edges and of the corners
    float sup[6];      // T's largest w.(p - a)
};

__device__ __forceinline__ float fast_sqrt(float x) { return x * rsqrtf(x); }  // NaN at 0

// A bound as a byte, rounded up; from kTop on 255.
__device__ __forceinline__ unsigned bound_byte(float s) {
    const unsigned q = __float2uint_ru(s * kHorizonUnit);
    return q >= kTop ? 255u : q;
}

// Octants in which something can lie whose bounds are ax = lo.x - T.hi.x above and
// bx = T.lo.x - hi.x below T's (and so on), as byte masks.
__device__ __forceinline__ Oct octants(float ax, float bx, float ay, float by, float az, float bz, float eo) {
    unsigned m = 0xffffffffu;
    if (bx > eo) m &= 0xff00ff00u;  // nothing at larger x: only d.x < 0
    if (ax > eo) m &= 0x00ff00ffu;
    if (by > eo) m &= 0xffff0000u;
    if (ay > eo) m &= 0x0000ffffu;
    return {bz > eo ? 0u : m, az > eo ? 0u : m};
}

// Bounds A and B of one triangle of the scene raise the horizons H.
__device__ __forceinline__ void add_tri(const HorizonTri& T, const GTri& X, Oct& H) {
    const F3 x[3] = {f3(X.v0.x, X.v0.y, X.v0.z), f3(X.v1.x, X.v1.y, X.v1.z), f3(X.v2.x, X.v2.y, X.v2.z)};
    F3 r[3];
    float h[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        r[i] = x[i] - T.a;
        h[i] = dot(r[i], T.n) + T.off;
    }
    const float hm = fmaxf(h[0], fmaxf(h[1], h[2]));
    if (hm <= 0.0f) return;
    const F3 lo = f3(min3f(x[0].x, x[1].x, x[2].x), min3f(x[0].y, x[1].y, x[2].y), min3f(x[0].z, x[1].z, x[2].z));
    const F3 hi = f3(max3f(x[0].x, x[1].x, x[2].x), max3f(x[0].y, x[1].y, x[2].y), max3f(x[0].z, x[1].z, x[2].z));
    const Oct m = octants(lo.x - T.hi.x, T.lo.x - hi.x, lo.y - T.hi.y, T.lo.y - hi.y, lo.z - T.hi.z, T.lo.z - hi.z, T.eo);
    const F3 c = 0.333333343f * (x[0] + x[1] + x[2]);
    float rx = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const F3 v = x[i] - c;
        rx = fmaxf(rx, dot(v, v));
    }
    const F3 cg = c - T.g;
    const float dist = 0.99999f * fast_sqrt(dot(cg, cg)) - 1.00001f * fast_sqrt(rx) - T.rad - T.eo;
    float s = fminf(1.0f, __fdividef(hm, fmaxf(0.999e-3f, dist)));
    unsigned q = bound_byte(s) * 0x01010101u;
    if (((__vcmpltu4(H.a, q) & m.a) | (__vcmpltu4(H.b, q) & m.b)) == 0u) return;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        float slope = 0.0f, near = 1.0f, fm = 1.0f;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float f = dot(r[i], T.w[k]) - T.sup[k];
            fm = fminf(fm, f);
            if (f <= 2.0e-4f) near = fminf(near, -h[i]);
            else slope = fmaxf(slope, __fdividef(h[i], f - T.el));
        }
        if (fm >= -1.0e-6f && slope * (T.el + 1.0e-6f) < near) s = fminf(s, 1.00001f * slope * rsqrtf(1.0f + slope * slope));
    }
    q = bound_byte(s) * 0x01010101u;
    H.a = __vmaxu4(H.a, q & m.a);
    H.b = __vmaxu4(H.b, q & m.b);
}

__global__ void __launch_bounds__(128) k_horizon(const GNode4* __restrict__ nodes, const GTri* __restrict__ tris,
                                                 int64_t ntris, unsigned long long* out) {
    const int64_t slot = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (slot >= ntris) return;
    // the scene's bounds from the root's children
    float far2 = 0.0f, diag2 = 0.0f;
    {
        const GNode4& R = nodes[0];
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int c = 0; c < 4; ++c) {
            if ((&R.child.x)[c] == -1) continue;
            lo[0] = fminf(lo[0], (&R.lox.x)[c]); hi[0] = fmaxf(hi[0], (&R.hix.x)[c]);
            lo[1] = fminf(lo[1], (&R.loy.x)[c]); hi[1] = fmaxf(hi[1], (&R.hiy.x)[c]);
            lo[2] = fminf(lo[2], (&R.loz.x)[c]); hi[2] = fmaxf(hi[2], (&R.hiz.x)[c]);
        }
        for (int a = 0; a < 3; ++a) {
            const float f = fmaxf(fabsf(lo[a]), fabsf(hi[a])), d = hi[a] - lo[a];
            far2 += f * f;
            diag2 += d * d;
        }
    }
    const float far = sqrtf(far2), diag = 1.01f * sqrtf(diag2) + 0.02f;
    const float en = kU32 * (12.0f * diag + 12.0f * far);  // |e.n|, and the rounding of (q - a).n
    const GTri V = tris[slot];
    HorizonTri T;
    T.a = f3(V.v0.x, V.v0.y, V.v0.z);
    T.n = f3(V.v0.w, V.v1.w, V.v2.w);
    T.el = kU32 * (18.0f * diag + 3.0f * far);
    T.eo = 1.01e-4f + en + T.el;
    const F3 b = f3(V.v1.x, V.v1.y, V.v1.z), c = f3(V.v2.x, V.v2.y, V.v2.z);
    const F3 ab = b - T.a, ac = c - T.a, bc = c - b;
    const float lmax = sqrtf(fmaxf(dot(ab, ab), fmaxf(dot(ac, ac), dot(bc, bc))));
    const F3 N = cross(ab, ac);
    const float alt = sqrtf(dot(N, N)) / fmaxf(lmax, 1e-30f);
    const float flat = fmaxf(fabsf(dot(ab, T.n)), fabsf(dot(ac, T.n)));
    T.off = flat - (1.0e-4f - en);
    if (!(dot(T.n, T.n) > 0.9f) || !(4.0f * kU32 * (far + lmax) <= 4.0e-3f * alt) || !(T.off <= -2.0e-5f)) {
        store_horizon(out + slot, ~0ull);
        return;
    }
    T.lo = f3(min3f(T.a.x, b.x, c.x), min3f(T.a.y, b.y, c.y), min3f(T.a.z, b.z, c.z));
    T.hi = f3(max3f(T.a.x, b.x, c.x), max3f(T.a.y, b.y, c.y), max3f(T.a.z, b.z, c.z));
    T.g = 0.333333343f * (T.a + b + c);
    const F3 ga = T.a - T.g, gb = b - T.g, gc = c - T.g;
    T.rad = 1.00001f * sqrtf(fmaxf(dot(ga, ga), fmaxf(dot(gb, gb), dot(gc, gc))));
    const F3 dir[6] = {cross(ab, T.n), cross(bc, T.n), cross(f3(-ac.x, -ac.y, -ac.z), T.n), ga, gb, gc};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const F3 w = fma3(-dot(dir[k], T.n), T.n, dir[k]);
        T.w[k] = unit(w);
        T.sup[k] = fmaxf(0.0f, fmaxf(dot(ab, T.w[k]), dot(ac, T.w[k])));
    }
    // octants that no ray of the front side leaves in above the floor start out blocked
    Oct H{0u, 0u};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float px = fmaxf(0.0f, (k & 1) ? -T.n.x : T.n.x), py = fmaxf(0.0f, (k & 2) ? -T.n.y : T.n.y),
                    pz = fmaxf(0.0f, (k & 4) ? -T.n.z : T.n.z);
        const unsigned q = px * px + py * py + pz * pz > kFloor * kFloor ? bound_byte(kFloor) : 255u;
        if (k < 4) H.a |= q << (8 * k);
        else H.b |= q << (8 * (k - 4));
    }
    const float offn = T.off - dot(T.a, T.n);

    int stack[kStackDepth];
    int sp = 0, ref = 0, visits = 0;
    bool over = false;
    for (;;) {
        if (++visits > kVisits) { over = true; break; }
        if (ref >= 0) {
            const GNode4 nd = load_node(nodes + ref);
            float top = 0.0f;
            int next = -1;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int ch = (&nd.child.x)[k];
                const F3 lo = f3((&nd.lox.x)[k], (&nd.loy.x)[k], (&nd.loz.x)[k]);
                const F3 hi = f3((&nd.hix.x)[k], (&nd.hiy.x)[k], (&nd.hiz.x)[k]);
                // the box's corner farthest along n
                const float hm = fmaf(T.n.x > 0.0f ? hi.x : lo.x, T.n.x, fmaf(T.n.y > 0.0f ? hi.y : lo.y, T.n.y,
                                 fmaf(T.n.z > 0.0f ? hi.z : lo.z, T.n.z, offn)));
                if (ch == -1 || hm <= 0.0f) continue;
                const float ax = lo.x - T.hi.x, bx = T.lo.x - hi.x, ay = lo.y - T.hi.y, by = T.lo.y - hi.y,
                            az = lo.z - T.hi.z, bz = T.lo.z - hi.z;
                const float gx = max3f(ax, bx, 0.0f), gy = max3f(ay, by, 0.0f), gz = max3f(az, bz, 0.0f);
                const float dist = 0.99999f * fast_sqrt(gx * gx + gy * gy + gz * gz) - T.eo;
                const float s = fminf(1.0f, __fdividef(hm, fmaxf(0.999e-3f, dist)));
                const Oct m = octants(ax, bx, ay, by, az, bz, T.eo);
                const unsigned q = bound_byte(s) * 0x01010101u;
                if (((__vcmpltu4(H.a, q) & m.a) | (__vcmpltu4(H.b, q) & m.b)) == 0u) continue;
                const F3 e = hi - lo;
                if (dist > 0.0f && dot(e, e) < 4.0f * kAccept * kAccept * dist * dist) {
                    H.a = __vmaxu4(H.a, q & m.a);
                    H.b = __vmaxu4(H.b, q & m.b);
                    continue;
                }
                // the child with the largest bound next, the others later
                int later = ch;
                if (s > top) {
                    top = s;
                    later = next;
                    next = ch;
                }
                if (later != -1) {
                    if (sp < kStackDepth) stack[sp++] = later;
                    else over = true;
                }
            }
            if (next != -1) {
                ref = next;
                continue;
            }
        } else {
            const int code = ~ref, first = code >> 4, cnt = code & 15;
            for (int k = 0; k < cnt; ++k) add_tri(T, tris[first + k], H);
        }
        if (sp == 0 || over) break;
        ref = stack[--sp];
    }
    // 0.01 above the bound: the roundings of this pass and of the ray's own d.n
    unsigned long long v = (unsigned long long)__vaddus4(H.b, 0x03030303u) << 32 | __vaddus4(H.a, 0x03030303u);
    store_horizon(out + slot, over ? ~0ull : v);
}

}  // namespace

sbr_status use_horizons(sbr_scene* s, int64_t rays, cudaStream_t stream) {
    std::lock_guard<std::mutex> lock(s->horizon_mu);
    if (s->horizon_built) return SBR_OK;
    s->horizon_rays += rays;
    if (s->horizon_rays < kHorizonRays * s->ntris) return SBR_OK;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    SBR_CUDA(cudaStreamIsCapturing(stream, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return SBR_OK;  // not into somebody's graph
    if (!s->horizon_done) SBR_CUDA(cudaEventCreateWithFlags(&s->horizon_done, cudaEventDisableTiming));
    k_horizon<<<(unsigned)((s->ntris + 127) / 128), 128, 0, stream>>>(s->d_nodes, s->d_tris, s->ntris, s->d_horizon);
    SBR_CUDA(cudaGetLastError());
    SBR_CUDA(cudaEventRecord(s->horizon_done, stream));
    s->horizon_built = true;
    return SBR_OK;
}

sbr_status clear_horizons(sbr_scene* s) {
    std::lock_guard<std::mutex> lock(s->horizon_mu);
    if (s->horizon_done) SBR_CUDA(cudaStreamWaitEvent(s->stream, s->horizon_done, 0));
    SBR_CUDA(cudaMemsetAsync(s->d_horizon, 0xff, sizeof(unsigned long long) * (size_t)s->ntris, s->stream));
    s->horizon_built = false;
    s->horizon_rays = 0;
    return SBR_OK;
}

}  // namespace sbr
