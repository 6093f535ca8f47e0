// Device code shared by the forward and backward trace kernels: the k-nearest hierarchy walk that
// replaces optixTrace + __anyhit__ot (optix_tracer/forward.cu:117-132, 481-525), the ray/ray-grid
// mapping, and spherical-harmonics colour.
#pragma once
#include "dst_common.cuh"

#define DST_STACK 96                 // >= depth bound of a Karras tree over 63-bit keys + 32-bit index tie-breaks
#define DST_MAX_CHUNKS 4096          // bound on enumerations per ray segment (the reference loops without one)
#define DST_MAX_INTERSECTION 256     // optix_tracer/config.h:23
#define DST_PAD_FACTOR 4e-6f         // box padding per unit of coordinate magnitude, see knearest()

struct TraceCounters { unsigned long long segs, enums, nodes, quads, evals, contribs; };

__device__ __forceinline__ unsigned long long make_key(float t, unsigned int pidx) {
    return ((unsigned long long)__float_as_uint(t) << 32) | pidx;
}
__device__ __forceinline__ float hitkey_t(unsigned long long k) { return __uint_as_float((unsigned int)(k >> 32)); }

// 256-bit read-only loads (one instruction per 32-byte record: what bounds the walk is the number of cache lines its load
// instructions touch, and a record fetched in pieces touches its line once per piece)
__device__ __forceinline__ void ldg256(const void* p, float4& lo, float4& hi) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w) : "l"(p));
}
__device__ __forceinline__ BvhChild load_child(const BvhChild* p) {
    float4 a, b;
    ldg256(p, a, b);
    BvhChild c;
    c.lox = a.x; c.loy = a.y; c.hix = a.z; c.hiy = a.w; c.loz = b.x; c.hiz = b.y; c.c = __float_as_int(b.z); c.pad = 0;
    return c;
}
struct Quad { float4 a, b, c; unsigned int gid; };
__device__ __forceinline__ Quad load_quad(const BvhView& bvh, int pos) {
    Quad q;
    float4 d;
    const float4* p = bvh.quads + 4 * (size_t)pos;
    ldg256(p, q.a, q.b); ldg256(p + 2, q.c, d);
    q.gid = (unsigned int)__float_as_int(d.x);
    return q;
}

// The DST_CHUNK smallest (t, primitive id) hits with 0 <= t < 1e16 from origin o, ascending, in
// kb[0], kb[KS], kb[2 KS], ... (a column of a shared-memory array). Returns min(#hits, DST_CHUNK).
//
// Differences from the reference's scheme (every hit on the whole ray goes through an any-hit
// program that insertion-sorts into a 16-slot buffer): nodes and quads whose nearest possible t
// lies beyond the current 16th hit are culled, so the cost is that of a k-nearest query instead
// of growing with the number of hits behind the chunk.
//
// Conservativeness: a hit accepted by ray_quad() lies on the ray within ~20 ulp(M) of the quad,
// M = |o|_inf + largest |coordinate| of the scene. Child boxes are therefore padded by
// DST_PAD_FACTOR * M through the per-ray plane offsets (no extra work per node), which also
// covers the rounding of the slab arithmetic itself.
template <bool BRUTE, bool COUNT, int KS>
__device__ __forceinline__ int knearest(const BvhView& bvh, float ox, float oy, float oz, float dx, float dy, float dz,
                                        unsigned long long* kb, unsigned int* status, TraceCounters& tc,
                                        float kmax0 = DST_T_MAX) {
    int n = 0;
    float kmax = kmax0;          // hits beyond kmax0 are of no interest to the caller
    if (bvh.P <= 0) return 0;

    auto offer = [&](int pos) {
        const Quad q = load_quad(bvh, pos);
        if (COUNT) tc.quads++;
        float t; int tri;
        if (!ray_quad(q.a, q.b, q.c, ox, oy, oz, dx, dy, dz, kmax, t, tri)) return;
        const unsigned int gid = q.gid;
        const unsigned long long key = make_key(t, 2u * gid + (unsigned int)tri);
        if (n == DST_CHUNK && key >= kb[(DST_CHUNK - 1) * KS]) return;
        int j = n;
        while (j > 0 && kb[(j - 1) * KS] > key) j--;
        if (n == DST_CHUNK) n = DST_CHUNK - 1;
        for (int i = n; i > j; i--) kb[i * KS] = kb[(i - 1) * KS];
        kb[j * KS] = key;
        n++;
        if (n == DST_CHUNK) kmax = hitkey_t(kb[(DST_CHUNK - 1) * KS]);
    };

    if (BRUTE) {
        for (int pos = 0; pos < bvh.P; pos++) offer(pos);
        return n;
    }

    const float omax = fmaxf(fabsf(ox), fmaxf(fabsf(oy), fabsf(oz)));
    if (!(omax < INFINITY)) return 0;
    const float pad = DST_PAD_FACTOR * (omax + __ldg(bvh.header + 6)) + 1e-30f;
    const float sdx = fabsf(dx) < 1e-20f ? copysignf(1e-20f, dx) : dx;
    const float sdy = fabsf(dy) < 1e-20f ? copysignf(1e-20f, dy) : dy;
    const float sdz = fabsf(dz) < 1e-20f ? copysignf(1e-20f, dz) : dz;
    const float ix = 1.0f / sdx, iy = 1.0f / sdy, iz = 1.0f / sdz;
    const bool px = !(sdx < 0.0f), py = !(sdy < 0.0f), pz = !(sdz < 0.0f);
    // entry plane t = near * i - on, exit plane t = far * i - of, with the padding folded in
    const float onx = fmaf(ox, ix, pad * fabsf(ix)), ofx = fmaf(ox, ix, -pad * fabsf(ix));
    const float ony = fmaf(oy, iy, pad * fabsf(iy)), ofy = fmaf(oy, iy, -pad * fabsf(iy));
    const float onz = fmaf(oz, iz, pad * fabsf(iz)), ofz = fmaf(oz, iz, -pad * fabsf(iz));

    unsigned long long stack[DST_STACK];
    int sp = 0;
    constexpr int DONE = 0x7fffffff;
    // pops the next subtree that can still hold a hit nearer than the 16th
    auto pop = [&]() -> int {
        while (sp > 0) {
            const unsigned long long e = stack[--sp];
            if (__uint_as_float((unsigned int)(e >> 32)) <= kmax) return (int)(unsigned int)e;
        }
        return DONE;
    };
    int cur = 0;
    for (;;) {
        // "while-while": lanes walk internal nodes until each holds a leaf (or is done), then test leaves together
        while ((unsigned int)cur < (unsigned int)DONE) {
            const BvhChild k0 = load_child(bvh.nodes[cur].child), k1 = load_child(bvh.nodes[cur].child + 1);
            if (COUNT) tc.nodes++;
            const float n0x = px ? k0.lox : k0.hix, f0x = px ? k0.hix : k0.lox;
            const float n0y = py ? k0.loy : k0.hiy, f0y = py ? k0.hiy : k0.loy;
            const float n0z = pz ? k0.loz : k0.hiz, f0z = pz ? k0.hiz : k0.loz;
            const float n1x = px ? k1.lox : k1.hix, f1x = px ? k1.hix : k1.lox;
            const float n1y = py ? k1.loy : k1.hiy, f1y = py ? k1.hiy : k1.loy;
            const float n1z = pz ? k1.loz : k1.hiz, f1z = pz ? k1.hiz : k1.loz;
            const float tn0 = fmaxf(fmaxf(fmaf(n0x, ix, -onx), fmaf(n0y, iy, -ony)), fmaxf(fmaf(n0z, iz, -onz), 0.0f));
            const float tf0 = fminf(fminf(fmaf(f0x, ix, -ofx), fmaf(f0y, iy, -ofy)), fmaf(f0z, iz, -ofz));
            const float tn1 = fmaxf(fmaxf(fmaf(n1x, ix, -onx), fmaf(n1y, iy, -ony)), fmaxf(fmaf(n1z, iz, -onz), 0.0f));
            const float tf1 = fminf(fminf(fmaf(f1x, ix, -ofx), fmaf(f1y, iy, -ofy)), fmaf(f1z, iz, -ofz));
            const bool h0 = (tn0 <= tf0) && (tn0 <= kmax);
            const bool h1 = (tn1 <= tf1) && (tn1 <= kmax);
            if (h0 && h1) {
                const bool swap = tn1 < tn0 || (tn1 == tn0 && tf1 < tf0);      // entered first; on a tie (inside both boxes) left first
                const int cf = swap ? k0.c : k1.c;
                const float tfar = swap ? tn0 : tn1;
                if (sp < DST_STACK) stack[sp++] = ((unsigned long long)__float_as_uint(tfar) << 32) | (unsigned int)cf;
                else atomicOr(status, DST_STATUS_STACK_OVERFLOW);
                cur = swap ? k1.c : k0.c;
            } else if (h0) cur = k0.c;
            else if (h1) cur = k1.c;
            else cur = pop();
        }
        if (cur == DONE) break;
        offer(~cur);
        cur = pop();
    }
    return n;
}

// SH constants, optix_tracer/auxiliary.h:26-43
#define SHC0 0.28209479177387814f
#define SHC1 0.4886025119029199f
#define SHC2_0 1.0925484305920792f
#define SHC2_1 -1.0925484305920792f
#define SHC2_2 0.31539156525252005f
#define SHC2_3 -1.0925484305920792f
#define SHC2_4 0.5462742152960396f
#define SHC3_0 -0.5900435899266435f
#define SHC3_1 2.890611442640554f
#define SHC3_2 -0.4570457994644658f
#define SHC3_3 0.3731763325901154f
#define SHC3_4 -0.4570457994644658f
#define SHC3_5 1.445305721320277f
#define SHC3_6 -0.5900435899266435f

// loads the first 3*ncoef floats of a row of SH coefficients; vectorised when the row is 16-byte aligned
__device__ __forceinline__ void load_sh_row(const float* __restrict__ row, int nfloat, bool aligned, float* c) {
    if (aligned) {
        const float4* r4 = reinterpret_cast<const float4*>(row);
        const int nv = nfloat >> 2;
        if (nv == 12 && (reinterpret_cast<uintptr_t>(row) & 31) == 0) {       // degree 3, the usual layout: six 256-bit loads
#pragma unroll
            for (int i = 0; i < 6; i++) {
                float4 q, r;
                ldg256(r4 + 2 * i, q, r);
                c[8 * i] = q.x; c[8 * i + 1] = q.y; c[8 * i + 2] = q.z; c[8 * i + 3] = q.w;
                c[8 * i + 4] = r.x; c[8 * i + 5] = r.y; c[8 * i + 6] = r.z; c[8 * i + 7] = r.w;
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < 12; i++) {
            if (i < nv) { const float4 q = __ldg(r4 + i); c[4 * i] = q.x; c[4 * i + 1] = q.y; c[4 * i + 2] = q.z; c[4 * i + 3] = q.w; }
        }
#pragma unroll
        for (int i = 0; i < 48; i++) if (i >= (nv << 2) && i < nfloat) c[i] = __ldg(row + i);
    } else {
#pragma unroll
        for (int i = 0; i < 48; i++) if (i < nfloat) c[i] = __ldg(row + i);
    }
}

// Signed basis factors b[j] such that the reference's expression tree for the SH colour
// (optix_tracer/forward.cu:18-58) is r = b0*sh0; r = r + b[j]*sh[j] (j = 1..); r + 0.5; max(r, 0),
// one rounding per operation, in that order.
__device__ __forceinline__ void sh_basis(int deg, float x, float y, float z, float* b) {
    b[0] = SHC0;
    if (deg > 0) {
        b[1] = -xmul(SHC1, y); b[2] = xmul(SHC1, z); b[3] = -xmul(SHC1, x);
        if (deg > 1) {
            const float xx = xmul(x, x), yy = xmul(y, y), zz = xmul(z, z), xy = xmul(x, y), yz = xmul(y, z), xz = xmul(x, z);
            b[4] = xmul(SHC2_0, xy); b[5] = xmul(SHC2_1, yz);
            b[6] = xmul(SHC2_2, xsub(xsub(xmul(2.0f, zz), xx), yy));
            b[7] = xmul(SHC2_3, xz); b[8] = xmul(SHC2_4, xsub(xx, yy));
            if (deg > 2) {
                b[9] = xmul(xmul(SHC3_0, y), xsub(xmul(3.0f, xx), yy));
                b[10] = xmul(xmul(SHC3_1, xy), z);
                b[11] = xmul(xmul(SHC3_2, y), xsub(xsub(xmul(4.0f, zz), xx), yy));
                b[12] = xmul(xmul(SHC3_3, z), xsub(xsub(xmul(2.0f, zz), xmul(3.0f, xx)), xmul(3.0f, yy)));
                b[13] = xmul(xmul(SHC3_4, x), xsub(xsub(xmul(4.0f, zz), xx), yy));
                b[14] = xmul(xmul(SHC3_5, z), xsub(xx, yy));
                b[15] = xmul(xmul(SHC3_6, x), xsub(xx, xmul(3.0f, yy)));
            }
        }
    }
}

// unclamped colour channel ch (0..2) from the loaded coefficient row
__device__ __forceinline__ float sh_channel(int ncoef, const float* b, const float* c, int ch) {
    float r = xmul(b[0], c[ch]);
#pragma unroll
    for (int j = 1; j < 16; j++) if (j < ncoef) r = xadd(r, xmul(b[j], c[3 * j + ch]));
    return xadd(r, 0.5f);
}

// The three unclamped colour channels of one surfel, summed as its row arrives: the same operations as sh_channel, without the 48
// registers that hold a row whole (k_fwd_shade fits 96 registers with it; with the row held it spilled 144 bytes there).
__device__ __forceinline__ void sh_rgb(const float* __restrict__ row, int ncoef, bool aligned, const float* b, float& R, float& G, float& B) {
    if (ncoef == 16 && aligned && (reinterpret_cast<uintptr_t>(row) & 31) == 0) {
        float r[3];
#pragma unroll
        for (int i = 0; i < 6; i++) {
            float4 q[2];
            ldg256(reinterpret_cast<const float4*>(row) + 2 * i, q[0], q[1]);
            const float* c = reinterpret_cast<const float*>(q);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int v = 8 * i + k, j = v / 3, ch = v % 3;
                r[ch] = j == 0 ? xmul(b[0], c[k]) : xadd(r[ch], xmul(b[j], c[k]));
            }
        }
        R = xadd(r[0], 0.5f); G = xadd(r[1], 0.5f); B = xadd(r[2], 0.5f);
        return;
    }
    if (aligned) {
        float r[3];
#pragma unroll
        for (int i = 0; i < 12; i++) {
            if (4 * i < 3 * ncoef) {       // (an aligned row holds a multiple of four floats)
                const float4 q = __ldg(reinterpret_cast<const float4*>(row) + i);
                const float c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int v = 4 * i + k, j = v / 3, ch = v % 3;
                    if (j < ncoef) r[ch] = j == 0 ? xmul(b[0], c[k]) : xadd(r[ch], xmul(b[j], c[k]));
                }
            }
        }
        R = xadd(r[0], 0.5f); G = xadd(r[1], 0.5f); B = xadd(r[2], 0.5f);
        return;
    }
    R = xmul(b[0], __ldg(row)); G = xmul(b[0], __ldg(row + 1)); B = xmul(b[0], __ldg(row + 2));
#pragma unroll
    for (int j = 1; j < 16; j++)
        if (j < ncoef) { R = xadd(R, xmul(b[j], __ldg(row + 3 * j))); G = xadd(G, xmul(b[j], __ldg(row + 3 * j + 1))); B = xadd(B, xmul(b[j], __ldg(row + 3 * j + 2))); }
    R = xadd(R, 0.5f); G = xadd(G, 0.5f); B = xadd(B, 0.5f);
}

// exp for x <= 0 as a fixed sequence of rounded operations (Cody-Waite reduction, degree-7 Taylor
// polynomial, exact power-of-two scaling): reproducible bit for bit on a CPU, about 1 ulp from a
// correctly rounded exp. The falloff G = exp(-rho/2) decides which hits contribute
// (optix_tracer/forward.cu:247-252), so it belongs to the exactly specified part.
__device__ __forceinline__ float pexp(float x) {
    if (!(x >= -87.0f)) return (x != x) ? x : 0.0f;
    if (x > 88.0f) x = 88.0f;
    const float kf = xsub(xadd(xmul(x, 1.44269504088896341f), 12582912.0f), 12582912.0f);
    float r = xfma(kf, -0.693145751953125f, x);
    r = xfma(kf, -1.42860682030941723212e-6f, r);
    float p = 0.0001984126984126984f;
    p = xfma(p, r, 0.001388888888888889f);
    p = xfma(p, r, 0.008333333333333333f);
    p = xfma(p, r, 0.041666666666666664f);
    p = xfma(p, r, 0.16666666666666666f);
    p = xfma(p, r, 0.5f);
    p = xfma(p, r, 1.0f);
    p = xfma(p, r, 1.0f);
    return xmul(p, __int_as_float(((int)kf + 127) << 23));
}

// Everything the compositing loop needs to know about one gathered hit.
struct SlotEval {
    float dpt, X, Y, Z;       // depth along the segment and world position
    float u, v;               // tangent-plane coordinates in units of the scales
    float nsign;              // +1 / -1: the normal is flipped toward the ray (DUAL_VISIABLE)
    float G, alpha;
    float4 r0, r1, r2, r3;    // the surfel's shading record
};

// Steps of optix_tracer/forward.cu:211-249 for one k-buffer entry, in the reference's operation
// order with one rounding per operation: depth, position, compute_transmat_uv (63-90), the
// visibility / near-depth / support tests and alpha. Returns false where the reference `continue`s.
// Shared by the forward and backward kernels so that the retrace takes identical decisions.
__device__ __forceinline__ bool eval_slot(unsigned long long key, float offset, float sox, float soy, float soz,
                                          float sdx, float sdy, float sdz, float min_depth, const float4* __restrict__ cache,
                                          int gidx, SlotEval& e) {
    e.dpt = xadd(hitkey_t(key), offset);
    e.X = xadd(sox, xmul(e.dpt, sdx)); e.Y = xadd(soy, xmul(e.dpt, sdy)); e.Z = xadd(soz, xmul(e.dpt, sdz));
    const float4* rec = cache + 4 * (size_t)gidx;
    ldg256(rec, e.r0, e.r1); ldg256(rec + 2, e.r2, e.r3);
    const float u1 = xadd(rdot3(e.r0.x, e.r0.y, e.r0.z, e.X, e.Y, e.Z), -e.r0.w);
    const float v1 = xadd(rdot3(e.r1.x, e.r1.y, e.r1.z, e.X, e.Y, e.Z), -e.r1.w);
    e.u = xdiv(u1, e.r3.x); e.v = xdiv(v1, e.r3.y);
    const float rho3d = xadd(xmul(e.u, e.u), xmul(e.v, e.v));
    const float cosv = -rdot3(sdx, sdy, sdz, e.r2.x, e.r2.y, e.r2.z);
    if (cosv == 0.0f) return false;
    e.nsign = cosv > 0.0f ? 1.0f : -1.0f;
    if (e.dpt < min_depth) return false;
    const float power = -0.5f * rho3d;
    if (power > 0.0f) return false;
    e.G = pexp(power);
    e.alpha = fminf(0.99f, xmul(e.r2.w, e.G));
    if (e.alpha < 1.0f / 255.0f) return false;
    return true;
}

// ---------------------------------------------------------------------------------------------
// Wavefront plumbing. A trace call runs as rounds of kernels over the list of rays that are
// still alive: the gather (k_enum, k_enum_group, k_enum_ray) finds the 16 nearest hits of each ray's
// current enumeration, a shade kernel composites them and decides what the ray does next. Ray state, hit buffers and the lists live in scratch memory owned by the handle.
// counts[r] is the length of list[r & 1] in round r; a round whose list is shorter than
// `min_count` is skipped by all of them and left to the tail kernel, which runs the remaining rays to
// completion: a warp per ray, in the backward a warp per few rays, and a thread per ray where a forward
// leaves more than 32,768.
// ---------------------------------------------------------------------------------------------
// A request: origin and direction of the ray's segment, how far along it the enumeration starts (0 in the segment's first), and the largest distance from
// there that is of interest. off < 0: starts at -off, and the ray's last request was answered by a later gather step than k_enum.
struct __align__(16) EnumReq {
    float ox, oy, oz, dx, dy, dz, kmax0, off;
    // Origin the enumeration starts from: the segment's, moved along the ray past the last evaluated hit (forward.cu:303-306).
    __device__ __forceinline__ void start(float& x, float& y, float& z) const {
        const float t = fabsf(off);
        x = ox; y = oy; z = oz;
        if (t != 0.0f) { x = xadd(ox, xmul(t, dx)); y = xadd(oy, xmul(t, dy)); z = xadd(oz, xmul(t, dz)); }
    }
};

// Everything a ray keeps between kernels is indexed by its list slot (its place in the tile-ordered list of round 0, see slot_ray()), in blocks of
// 32 slots with the words of a record one after the other and the 32 slots of a block side by side. The rays of a warp are (survivors of)
// neighbouring slots, so a warp's access to one word of its rays' records touches a few cache lines; as one record per ray it touched
// 32, and the composite kernel, whose loads those mostly were, was bound by them.
__device__ __forceinline__ size_t soa(int slot, int word, int words) { return ((size_t)(slot >> 5) * words + word) * 32 + (slot & 31); }
__device__ __forceinline__ EnumReq load_req(const float4* req, int slot) {
    const float4 a = req[soa(slot, 0, 2)], b = req[soa(slot, 1, 2)];
    EnumReq q;
    q.ox = a.x; q.oy = a.y; q.oz = a.z; q.dx = a.w; q.dy = b.x; q.dz = b.y; q.kmax0 = b.z; q.off = b.w;
    return q;
}
__device__ __forceinline__ void store_req(float4* req, int slot, const EnumReq& q) {
    req[soa(slot, 0, 2)] = make_float4(q.ox, q.oy, q.oz, q.dx);
    req[soa(slot, 1, 2)] = make_float4(q.dy, q.dz, q.kmax0, q.off);
}
__device__ __forceinline__ float& req_bound(float4* req, int slot) { return req[soa(slot, 1, 2)].z; }

constexpr int ENUM_THREADS = 128;
#ifndef DST_ENUM_MIN_BLOCKS
#define DST_ENUM_MIN_BLOCKS 8         // resident blocks per SM the gather kernel is compiled for
#endif
#define DST_TAIL_CURSOR (DST_COUNTS_STRIDE - 1)          // word of a set of round counters no round uses: next list entry of the tail kernel

// ---------------------------------------------------------------------------------------------
// Gather: per live ray, the 16 nearest hits from the requested origin (same result as knearest()).
//
// Large overlapping quads put hundreds of boxes around any origin: a walk for 16 hits opens 300 nodes in the dense scenes, and
// neighbouring rays open the same ones. So a warp walks the hierarchy for the HULL of a set of rays (origins and
// directions, component by component), and its lanes are 32 child boxes, then 32 quads, of one step, instead of 32
// copies of nearly the same ray. Everything the hull test lets through is tested exactly, with each ray's own 16th-nearest distance;
// the hull tests are conservative, so the hit set is that of an independent walk per ray. What a hull costs depends on how alike its rays are
// (the hull of rays that fan out reaches quads none of them comes near), so a gather has three steps, each taking what the one before gave up:
//   k_enum        32 consecutive live rays per warp (a pixel tile, or the survivors of neighbouring ones: the lists keep tile order, see
//                 k_compact). Quads that pass the hull test are tested by every lane against its own ray. Given up past DST_BEAM_STEPS
//                 steps or DST_BEAM_CANDS such quads.
//   k_enum_group  8 rays per warp (a 4x2 patch of the tile); every lane holds one quad and tests the 8 rays in turn. Given up past DST_GROUP_STEPS.
//   k_enum_ray    one ray per warp (the hull is the ray), one quad per lane.
// Forward (3M-surfel 1080p one-bounce scene / 6M-surfel two-bounce scene at 4 x 540 x 960) against a walk in which every lane tested its own
// ray against each node's two boxes: 43 -> 18.4 ms and 230 -> 88.7 ms (composite included). Groups of 4 or 16: 10-15 % slower on the two-bounce
// scene. Runs of 2 or 4 quads as leaves of the walk: 2-9 % slower than single quads.
// Blocks are persistent and take batches from a cursor; no block waits for another.
// ---------------------------------------------------------------------------------------------
// What a walk may take before it is given up: steps, and quads that pass the hull test. A launch with a few times more work than it has
// warps (with what the call's other slices launch) takes the larger limits, because giving up costs work; with less, the time is that of its longest walk,
// and the smaller ones are the faster. Measured, one set of limits (160 / 300 / 192) against two: two-bounce scene 93.3 -> 88.7 ms, 400 x 400
// object views 4.40 -> 3.63 ms, four LiDAR sweeps 2.44 -> 2.26 ms.
// Steps of a group in a launch without a load: 150 -> 100 object views 4.13 -> 3.99 ms, LiDAR sweeps 2.46 -> 2.36. 200 instead of 260 steps in all loaded launches cost two
// bounces 1 %, 400 or 600 the object view 9-23 %. Fewer quads without a load (70) suit scenes where a quad is hit by few of a batch's rays (object views 3.43 ms
// instead of 3.92), but a 200 x 200 patch of a dense scene takes 4.15 ms instead of 3.52, and with the rays' hits as the criterion a 170 x 150 view
// of a ball 200 us instead of 180.
#define DST_LOADED_BEAMS 2                 // times as many batches as warps of the launch
#define DST_LOADED_GROUPS 3
// A group launch counts the work of at most this many slices, itself included: with more, the others are at other stages when it runs. All slices
// counted | four, forwards in five and six slices: 560 x 900 and 720 x 1280 views of an object (0.3M surfels) 3.08 | 2.86 and 3.51 | 3.55 ms, secondary rays from its
// surface 3.20 | 3.01 and 4.70 | 4.41, views of a scene (0.6M) with a reflection 8.41 | 8.34 and 11.12 | 11.04, with two 36.9 | 36.8 and 60.1 | 60.2.
#define DST_GROUP_LOAD_SLICES 4
#define DST_BEAM_STEPS 160
#define DST_BEAM_STEPS_LOADED 240
#define DST_BEAM_CANDS 200
#define DST_BEAM_CANDS_LOADED 400
#define DST_GROUP_STEPS 100
#define DST_GROUP_STEPS_LOADED 260
#define DST_GROUP 8
#define DST_GROUP_MIN_BLOCKS 10
// Stack entries: one step adds at most 24. The stacks are most of a warp's shared memory, and what the walks wait for is memory latency, so they are
// as small as they can be: 32 instead of 24 warps an SM in k_enum and 40 in the other steps take 8 % off the two-bounce scene. A walk that may be
// given up is when its stack is full; one that has to end needs room for a depth-first descent.
#define DST_BEAM_STACK 192
#define DST_WALK_STACK 288
#define DST_WALK_QUADS 64
#define DST_WALK_STEP_LIMIT (1 << 20)      // bound on the steps of a walk that cannot be given up (status flag instead of a hang)
// Hull of a set of rays, component by component: origins oc +- orad, directions dc +- drad.
struct BeamQ { float oc[3], orad[3], dc[3], drad[3], dsum, dmax; };      // dsum: sum of the largest |d| per axis, dmax: largest of them

// Conservative test of one quad against the hull, in interval arithmetic (centre and radius): can ANY ray of the set pass ray_quad() with a hit no
// farther than kmaxb? The steps are those of ray_quad(): t = n.(p0 - o) / n.d, h = t d - (p0 - o), u = wu.h, v = wv.h,
// accepted iff 0 <= t <= kmax and u, v in [0, 1]. Every interval is widened by more than the rounding of either computation, so a quad some ray hits is
// never rejected: by an order of magnitude more in what grows with the quad's distance from the hull's origin, the distance to the hit and the
// direction, by 1.6 times as much in what grows with how far the rays have been moved (in orad, see make_beam()). For neighbouring rays (close origins, directions a
// degree apart) the intervals are narrow, and nearly every quad that no ray hits is rejected here by ONE lane. tl: nearest possible hit.
__device__ __forceinline__ bool hull_quad(const BeamQ& bm, const float4 qa, const float4 qb, const float4 qc, float kmaxb, float& tl) {
    const float p0[3] = { qa.x, qa.y, qa.z }, nn[3] = { qa.w, qb.x, qb.y }, wu[3] = { qb.z, qb.w, qc.x }, wv[3] = { qc.y, qc.z, qc.w };
    float rc[3], bc = 0.f, br = 0.f, ac = 0.f, ar = 0.f, scale = 0.f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        rc[a] = p0[a] - bm.oc[a];
        bc = fmaf(nn[a], bm.dc[a], bc); br = fmaf(fabsf(nn[a]), bm.drad[a], br);
        ac = fmaf(nn[a], rc[a], ac); ar = fmaf(fabsf(nn[a]), bm.orad[a], ar);
        scale = fmaxf(scale, fabsf(rc[a]) + bm.orad[a]);
    }
    const float nmag = fabsf(nn[0]) + fabsf(nn[1]) + fabsf(nn[2]);
    br = fmaf(4e-6f * nmag, bm.dsum, br); ar = fmaf(12e-6f * nmag, scale, ar);
    const float bs = fabsf(bc), as = bc < 0.f ? -ac : ac;
    tl = 0.f;
    if (!(bs - br > 1e-30f)) return true;        // some direction of the hull is (all but) parallel to the plane: no bound
    // quotients by approximate reciprocals (two units in the last place; the interval is widened by 1e-5 relative below)
    const float al = as - ar, ah = as + ar;
    tl = __fdividef(al, al >= 0.f ? bs + br : bs - br);
    float th = __fdividef(ah, ah >= 0.f ? bs - br : bs + br);
    tl -= 1e-5f * fabsf(tl) + 1e-30f; th += 1e-5f * fabsf(th) + 1e-30f;
    if (!(th >= 0.f && tl <= kmaxb)) return false;
    tl = fmaxf(tl, 0.f); th = fminf(th, kmaxb);
    const float tc = 0.5f * (tl + th), tr = 0.5f * (th - tl) + 1e-6f * th;
    float uc = -0.5f, ur = 0.5f + 1e-5f, vc = -0.5f, vr = 0.5f + 1e-5f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float hc = fmaf(tc, bm.dc[a], -rc[a]), hr = fmaf(tr, fabsf(bm.dc[a]) + bm.drad[a], fmaf(tc, bm.drad[a], bm.orad[a]));
        uc = fmaf(wu[a], hc, uc); ur = fmaf(fabsf(wu[a]), hr, ur);
        vc = fmaf(wv[a], hc, vc); vr = fmaf(fabsf(wv[a]), hr, vr);
    }
    // u and v are of order 1; their rounding error is that of h (cancellation of t d against p0 - o) times |w|
    const float eh = 16e-6f * fmaf(th, bm.dmax, scale);
    ur = fmaf(eh, fabsf(wu[0]) + fabsf(wu[1]) + fabsf(wu[2]), ur);
    vr = fmaf(eh, fabsf(wv[0]) + fabsf(wv[1]) + fabsf(wv[2]), vr);
    return !(fabsf(uc) > ur || fabsf(vc) > vr);
}

// Three-operand minimum / maximum and packed multiply-add, instructions sm_100 has and the compiler does not form here.
__device__ __forceinline__ float min3(float a, float b, float c) { float r; asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float2 fma2(float ax, float ay, float4 fo) {      // (ax, ay) * (fo.x, fo.y) + (fo.z, fo.w)
    float2 r;
    asm("{ .reg .b64 a, b, c, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7}; fma.rn.f32x2 d, a, b, c; mov.b64 {%0, %1}, d; }"
        : "=f"(r.x), "=f"(r.y) : "f"(ax), "f"(ay), "f"(fo.x), "f"(fo.y), "f"(fo.z), "f"(fo.w));
    return r;
}

// Slab constants of the hull for the child-box test of the walk. For every ray of the hull, with origin in [omin, omax] and direction
// in [dmin, dmax] along an axis:
//   entry  t >= (lo - omax) / dmax if the box lies ahead in +, t >= (omin - hi) / -dmin if it lies ahead in -, else t >= 0
//   exit   t <= (hi - omin) / dmin if every ray travels in +, t <= (omax - lo) / -dmax if every ray travels in -, else unbounded
// Each is one multiply-add of a box coordinate, taken two at a time (factors x, y and offsets z, w); an impossible direction has a huge factor.
struct BeamSlab { float4 in_lo, in_hi, out_lo, out_hi, in_z, out_z; };       // x and y of lo, x and y of hi, z of lo and hi
#define DST_KCNT_WIDE 0x100                // flag in a ray's hit count: answered by a later step than k_enum
struct WalkMemBase {
    unsigned long long place[DST_CHUNK];             // see take_hits()
    BeamSlab slab;
    BeamQ beam;
    int quads[DST_WALK_QUADS];                       // leaf positions of quads whose box the hull reaches
};
template <int STACK>
struct WalkStack : WalkMemBase {
    int stack[STACK];                                // subtrees, nearest on top
    unsigned short stack_t[STACK];                   // their nearest possible t, upper half (rounded towards 0: still a lower bound)
};
typedef WalkStack<DST_WALK_STACK> WalkMem;           // walks of one ray, which have to end
typedef WalkStack<DST_BEAM_STACK> BeamMem;           // walks of a hull, which may be given up

// Walks the hierarchy for the hull in m.beam / m.slab: a step takes up to 8 nodes from the top of the stack and tests their 32
// child boxes, one per lane. Single quads whose box passes go to a queue; whenever it holds 32 of them (or no node is
// left) leaf_step(valid, position) gets one quad per lane. krun (uniform) is the largest distance any ray still searches;
// leaf_step lowers it, and returns false to give the walk up. Returns false when given up or after max_steps steps.
template <bool COUNT, int STACK, class LeafStep>
__device__ __forceinline__ bool beam_walk(const BvhView& bvh, WalkStack<STACK>& m, float& krun, int max_steps, unsigned int* status, TraceCounters& tc, LeafStep leaf_step) {
    constexpr unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u, quad_below = (1u << (lane & 28)) - 1u;
    int sp = 1, nq = 0;
    if (lane == 0) { m.stack[0] = 0; m.stack_t[0] = 0; }
    __syncwarp();
    for (int step = 0; step < max_steps; step++) {
        if (nq >= 32 || sp == 0) {
            if (nq == 0) return true;
            const int take = nq < 32 ? nq : 32;
            nq -= take;
            const int pos = lane < take ? m.quads[nq + lane] : 0;
            __syncwarp();
            if (!leaf_step(lane < take, pos)) return false;
            continue;
        }
        // lanes 28..31 take the top entry, lanes 24..27 the next, ...: lane order is then the order in which surviving children
        // go back onto the stack (farthest first). A walk that may be given up is when its stack is full; a nearly full one of a walk
        // that has to end is walked one node at a time (it then grows by at most three entries per two levels of the tree).
        int width = 8;
        if (max_steps < DST_WALK_STEP_LIMIT) { if (sp > STACK - 24) return false; }
        else if (sp > STACK - 176) {
            width = 1;
            if (sp > STACK - 4) { if (lane == 0) atomicOr(status, DST_STATUS_STACK_OVERFLOW); return true; }
        }
        const int take = sp < width ? sp : width;
        const bool valid = 7 - (lane >> 2) < take;
        const int node = valid ? m.stack[sp - 8 + (lane >> 2)] : 0;
        const float node_t = valid ? __uint_as_float((unsigned int)m.stack_t[sp - 8 + (lane >> 2)] << 16) : INFINITY;
        sp -= take;
        __syncwarp();
        const BvhChild b = load_child(bvh.wide + 4 * (size_t)node + (lane & 3));          // (lanes without an entry read the root)
        if (COUNT && valid && (lane & 3) == 0) tc.nodes++;
        const float2 il = fma2(b.lox, b.loy, m.slab.in_lo), ih = fma2(b.hix, b.hiy, m.slab.in_hi), iz = fma2(b.loz, b.hiz, m.slab.in_z);
        const float2 ol = fma2(b.lox, b.loy, m.slab.out_lo), oh = fma2(b.hix, b.hiy, m.slab.out_hi), oz = fma2(b.loz, b.hiz, m.slab.out_z);
        const float tn = max3(max3(il.x, il.y, ih.x), max3(ih.y, iz.x, iz.y), 0.0f);
        const float tf = min3(min3(ol.x, ol.y, oh.x), oh.y, fminf(oz.x, oz.y));
        const bool h = node_t <= krun && tn <= fminf(tf, krun);
        const bool inside = h && b.c >= 0;
        const unsigned int inner = __ballot_sync(FULL, inside), leaves = __ballot_sync(FULL, h && b.c < 0);
        // Of the four children the nearest goes on top: entered first, or left first among those the rays start inside of. The key orders
        // them so (its two low bits are the lane's, so that no two are equal; 0: does not go on the stack).
        const unsigned int key = inside ? (((tn > 0.0f ? 0x80000000u | __float_as_uint(tn) : __float_as_uint(fmaxf(tf, 0.0f))) & ~3u) | (lane & 3)) : 0u;
        const int farther = (__shfl_xor_sync(FULL, key, 1) > key) + (__shfl_xor_sync(FULL, key, 2) > key) + (__shfl_xor_sync(FULL, key, 3) > key);
        if (inside) {
            const int at = sp + __popc(inner & quad_below) + farther;
            m.stack[at] = b.c;
            m.stack_t[at] = (unsigned short)(__float_as_uint(tn) >> 16);
        } else if (h) m.quads[nq + __popc(leaves & below)] = ~b.c;
        sp += __popc(inner);
        nq += __popc(leaves);
        __syncwarp();
    }
    return false;
}

__device__ __forceinline__ float redux_min(float v) { float r; asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }
__device__ __forceinline__ float redux_max(float v) { float r; asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }

// Where a hull of rays starts. The rays of a batch are at different distances along their segments, and where they come from one place a hull of the points
// they have reached is that much longer than it is wide, in a box with sides along the axes wide too. So such rays are taken back to the distance the least
// advanced of them has reached, and each searches `rel` further than from where its enumeration starts (rounded up). Where the box of the points reached
// is the narrower one (rays that started at distances of their own towards the same surface, directions of different length) the hull starts at those.
// Hulls of the points reached -> of the lines, by themselves: 0.93M rays of a reflective scene 15.1 -> 10.7 ms (reflective-render of perf/cases.py, seed 5;
// k_enum_group 8.2 -> 3.7, now 3.2 with the limits above: rays k_enum and k_enum_group gave up before), four LiDAR sweeps 2.91 -> 2.46, two 400 x 400
// object views 4.50 -> 4.13; 2M rays with one or two bounces, whose hulls are as wide as their directions fan out either way, 30.8 -> 30.5 and 114.4 -> 114.5. Hulls of whole segments (back to distance 0) lose 2 % there.
// 560 x 900 views of 0.3M surfels on an object, lines for all | the narrower: starts jittered along the rays 12.0 | 8.2 ms, directions of 0.8 to 1 units
// 7.7 | 5.6 (of 0.6M surfels and a reflection 17.4 | 12.5); views from one place with directions of one length as they were (within 0.3 %).
// Asking for 0.7 or 0.4 of the lines' extent gains nothing anywhere and costs a reflective scene with such directions 2 and 12 %; lines of normalised directions
// walked by length make them as fast as others and all others 1 to 2 % slower.
struct HullStart { float lo[3], hi[3], rel, moved; };      // box of the origins; moved: largest distance an origin has been moved along its ray
__device__ __forceinline__ HullStart hull_start(bool active, const EnumReq& q) {
    const float off = fabsf(q.off), first = redux_min(active ? off : INFINITY);
    HullStart s;
    auto box = [&](float x, float y, float z, float* lo, float* hi) {
        lo[0] = redux_min(active ? x : INFINITY); lo[1] = redux_min(active ? y : INFINITY); lo[2] = redux_min(active ? z : INFINITY);
        hi[0] = redux_max(active ? x : -INFINITY); hi[1] = redux_max(active ? y : -INFINITY); hi[2] = redux_max(active ? z : -INFINITY);
        return (hi[0] - lo[0]) + (hi[1] - lo[1]) + (hi[2] - lo[2]);
    };
    const float extent = box(fmaf(first, q.dx, q.ox), fmaf(first, q.dy, q.oy), fmaf(first, q.dz, q.oz), s.lo, s.hi);
    s.moved = redux_max(active ? off : 0.0f);
    s.rel = (off - first) + 1e-6f * off;
    if (s.moved > first) {
        float x, y, z, lo[3], hi[3];
        q.start(x, y, z);
        if (box(x, y, z, lo, hi) < extent) {
#pragma unroll
            for (int a = 0; a < 3; a++) { s.lo[a] = lo[a]; s.hi[a] = hi[a]; }
            s.rel = s.moved = 0.0f;
        }
    }
    return s;
}

// distance k from the start of a ray's enumeration, from the start of the hull (k < 0: none)
__device__ __forceinline__ float from_hull(float rel, float k) { return k < 0.0f ? k : (1.0f + 1e-6f) * (rel + k); }

// Slab constants of one axis for origins in [ol, oh] and directions in [dl, dh]; pad: padding of the boxes.
__device__ __forceinline__ void make_slab(BeamSlab& slab, int a, float ol, float oh, float dl, float dh, float pad) {
    const float lo = ol - pad, hi = oh + pad;
    const float ip = 1.0f / fmaxf(dh, 1e-30f), in = 1.0f / fmaxf(-dl, 1e-30f);
    const float xp = dl > 1e-20f ? 1.0f / dl : 0.0f, xn = dh < -1e-20f ? 1.0f / dh : 0.0f;
    const float f_in_lo = ip, o_in_lo = -hi * ip, f_in_hi = -in, o_in_hi = lo * in;
    const float f_out_lo = xn, o_out_lo = xn != 0.0f ? -hi * xn : 3e38f, f_out_hi = xp, o_out_hi = xp != 0.0f ? -lo * xp : 3e38f;
    if (a < 2) {
        (&slab.in_lo.x)[a] = f_in_lo; (&slab.in_lo.z)[a] = o_in_lo; (&slab.in_hi.x)[a] = f_in_hi; (&slab.in_hi.z)[a] = o_in_hi;
        (&slab.out_lo.x)[a] = f_out_lo; (&slab.out_lo.z)[a] = o_out_lo; (&slab.out_hi.x)[a] = f_out_hi; (&slab.out_hi.z)[a] = o_out_hi;
    } else {
        slab.in_z = make_float4(f_in_lo, f_in_hi, o_in_lo, o_in_hi);
        slab.out_z = make_float4(f_out_lo, f_out_hi, o_out_lo, o_out_hi);
    }
}

// The slabs of a single ray, the same in all lanes: its quads are tested exactly, no hull test sees them.
__device__ __forceinline__ void make_ray(WalkMemBase& m, float ox, float oy, float oz, float dx, float dy, float dz, float absmax) {
    const int a = threadIdx.x & 31;
    const float om = fmaxf(fabsf(ox), fmaxf(fabsf(oy), fabsf(oz)));
    if (a < 3) {
        const float o = a == 0 ? ox : a == 1 ? oy : oz, d = a == 0 ? dx : a == 1 ? dy : dz;
        make_slab(m.slab, a, o, o, d, d, DST_PAD_FACTOR * (om + absmax) + 1e-30f);
    }
    __syncwarp();
}

// Hull of the rays of the lanes with `active` (at least one), into m.beam and m.slab.
// The origins the exact tests use and the box's corners are off the rays by the rounding of moving them along. With u = 2^-24, per axis, D = off |d| and
// S = |corner| of a ray, D + S <= om: the exact origin is off by u (D + |D + S|) at most, the corner by u S; the steps of ray_quad() see the distance
// between the two once more, in p0 - o (u D) and in n.(p0 - o) (3 u D). Together 6 u D + 2 u S <= 6 u om = 3.6e-7 om, and the radius takes 6e-7 om.
__device__ __forceinline__ void make_beam(WalkMemBase& m, bool active, const HullStart& hs, float dx, float dy, float dz, float absmax) {
    const int lane = threadIdx.x & 31;
    const float d3[3] = { dx, dy, dz };
    float dlo[3], dhi[3], om = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        dlo[a] = redux_min(active ? d3[a] : INFINITY); dhi[a] = redux_max(active ? d3[a] : -INFINITY);
        om = fmaxf(om, fmaf(hs.moved, fmaxf(fabsf(dlo[a]), fabsf(dhi[a])), fmaxf(fabsf(hs.lo[a]), fabsf(hs.hi[a]))));
    }
    if (lane < 3) {
        const int a = lane;
        const float ol = a == 0 ? hs.lo[0] : a == 1 ? hs.lo[1] : hs.lo[2], oh = a == 0 ? hs.hi[0] : a == 1 ? hs.hi[1] : hs.hi[2];
        const float dl = a == 0 ? dlo[0] : a == 1 ? dlo[1] : dlo[2], dh = a == 0 ? dhi[0] : a == 1 ? dhi[1] : dhi[2];
        m.beam.oc[a] = 0.5f * (ol + oh); m.beam.orad[a] = 0.5f * (oh - ol) + 2e-7f * fmaxf(fabsf(ol), fabsf(oh)) + (hs.moved > 0.0f ? 6e-7f * om : 0.0f);      // (the centre is rounded)
        m.beam.dc[a] = 0.5f * (dl + dh); m.beam.drad[a] = 0.5f * (dh - dl) + 2e-7f * fmaxf(fabsf(dl), fabsf(dh));
        make_slab(m.slab, a, ol, oh, dl, dh, DST_PAD_FACTOR * (om + absmax) + 1e-30f);      // padding as in knearest(), for the ray with the largest coordinates
    }
    if (lane == 0) {
        const float a0 = fmaxf(fabsf(dlo[0]), fabsf(dhi[0])), a1 = fmaxf(fabsf(dlo[1]), fabsf(dhi[1])), a2 = fmaxf(fabsf(dlo[2]), fabsf(dhi[2]));
        m.beam.dsum = a0 + a1 + a2; m.beam.dmax = fmaxf(a0, fmaxf(a1, a2));
    }
    __syncwarp();
}

// First step of a gather: 32 consecutive entries of the live list per warp. A batch that is given up goes to `heavy` with its 32 slots, each ray
// with the search bound it has found.
template <bool COUNT>
__global__ void __launch_bounds__(ENUM_THREADS, DST_ENUM_MIN_BLOCKS) k_enum(BvhView bvh, float4* req, const int* __restrict__ list,
                                                       const int* __restrict__ count_ptr, int* cursor, int min_count,
                                                       unsigned long long* __restrict__ kbuf, int* __restrict__ kcnt,
                                                       unsigned int* status, unsigned long long* counters, int* heavy, int* heavy_count, int slices) {
    __shared__ unsigned long long kshared[DST_CHUNK * ENUM_THREADS];
    __shared__ BeamMem walk_mem[ENUM_THREADS / 32];
    const int total = *count_ptr;
    if (total < min_count || bvh.P <= 0) return;
    constexpr int KS = ENUM_THREADS;
    constexpr unsigned int FULL = 0xffffffffu;
    unsigned long long* kb = kshared + threadIdx.x;
    const int lane = threadIdx.x & 31;
    BeamMem& m = walk_mem[threadIdx.x >> 5];
    const float absmax = __ldg(bvh.header + 6);
    const bool loaded = (long long)total * slices > DST_LOADED_BEAMS * (long long)(gridDim.x * ENUM_THREADS);
    const int max_steps = loaded ? DST_BEAM_STEPS_LOADED : DST_BEAM_STEPS, max_cands = loaded ? DST_BEAM_CANDS_LOADED : DST_BEAM_CANDS;
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(cursor, 32);
        base = __shfl_sync(FULL, base, 0);
        if (base >= total) break;
        // The list is taken from its end: rays on a reflected segment come last in it (k_compact) and their batches are
        // the slow ones, so they start first and the cheap batches of primary rays fill the end of the round.
        const int idx = (((total + 31) >> 5) - 1 - (base >> 5)) * 32 + lane;
        const int slot = idx < total ? list[idx] : -1;
        bool active = false, wide = false;
        int n = 0;
        float kmax = -1.0f, ox = 0.f, oy = 0.f, oz = 0.f, dx = 0.f, dy = 0.f, dz = 0.f;
        EnumReq q = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
        if (slot >= 0) {
            q = load_req(req, slot);
            q.start(ox, oy, oz);
            dx = q.dx; dy = q.dy; dz = q.dz;
            active = fabsf(ox) < INFINITY && fabsf(oy) < INFINITY && fabsf(oz) < INFINITY && fabsf(dx) < INFINITY && fabsf(dy) < INFINITY && fabsf(dz) < INFINITY;
            if (active) { kmax = q.kmax0; wide = q.off < 0.0f; }
            if (COUNT) tc.enums++;
        }
        const unsigned int am = __ballot_sync(FULL, active);
        if (am != 0u) {
            // most of these rays' last requests were not answered here: their hull is still as wide, and trying it first is wasted
            bool done = 2 * __popc(__ballot_sync(FULL, wide)) <= __popc(am);
            if (done) {
            const HullStart hs = hull_start(active, q);
            make_beam(m, active, hs, dx, dy, dz, absmax);
            const float rel = hs.rel;
            float krun = redux_max(from_hull(rel, kmax));
            int cands = 0;
            done = beam_walk<COUNT>(bvh, m, krun, max_steps, status, tc, [&](bool valid, int pos) {
                // the quads that pass, nearest first: hits then come almost in order, and nothing is left to do at the first quad
                // that begins beyond every ray's 16th hit
                float tl = 0.0f;
                bool pass = false;
                if (valid) { const Quad q = load_quad(bvh, pos); pass = hull_quad(m.beam, q.a, q.b, q.c, krun, tl); }
                cands += __popc(__ballot_sync(FULL, pass));
                if (cands > max_cands) return false;
                unsigned int order = pass ? (__float_as_uint(tl) & ~31u) | lane : ~0u;
                unsigned int first = __reduce_min_sync(FULL, order);
                auto take = [&](const Quad& q, float t, int tri) {
                    const unsigned long long key = make_key(t, 2u * q.gid + (unsigned int)tri);
                    if (n == DST_CHUNK && key >= kb[(DST_CHUNK - 1) * KS]) return;
                    int j = n < DST_CHUNK ? n : DST_CHUNK - 1;
                    while (j > 0) {
                        const unsigned long long prev = kb[(j - 1) * KS];
                        if (prev < key) break;
                        kb[j * KS] = prev;
                        j--;
                    }
                    kb[j * KS] = key;
                    if (n < DST_CHUNK) n++;
                    if (n == DST_CHUNK) kmax = hitkey_t(kb[(DST_CHUNK - 1) * KS]);
                };
                // Two at a time, whose loads and tests do not wait for each other: a launch is as long as its slowest walks, and those are chains of such
                // tests. k_enum of 2M reflective rays 9.66 -> 9.21 ms, of an 800 x 800 object view 1.13 -> 1.04 (one quad ahead, loaded and not yet
                // tested, before); whole passes 1 to 3 %.
                while (first != ~0u) {
                    if (!__any_sync(FULL, __uint_as_float(first & ~31u) <= from_hull(rel, kmax))) break;
                    const Quad qa = load_quad(bvh, __shfl_sync(FULL, pos, first & 31));
                    if (lane == (first & 31)) order = ~0u;
                    const unsigned int second = __reduce_min_sync(FULL, order);
                    const Quad qb = load_quad(bvh, __shfl_sync(FULL, pos, second & 31));
                    if (lane == (second & 31)) order = ~0u;
                    first = __reduce_min_sync(FULL, order);
                    if (COUNT && lane == 0) tc.quads += second != ~0u ? 2 : 1;
                    float ta, tb; int tria, trib;
                    const bool ha = ray_quad(qa.a, qa.b, qa.c, ox, oy, oz, dx, dy, dz, kmax, ta, tria);
                    const bool hb = second != ~0u && ray_quad(qb.a, qb.b, qb.c, ox, oy, oz, dx, dy, dz, kmax, tb, trib);
                    if (ha) take(qa, ta, tria);
                    if (hb) take(qb, tb, trib);
                }
                krun = redux_max(from_hull(rel, kmax));
                return true;
            });
            }
            if (!done) {
                // (a bound below the request's can only have come from a full k-buffer: the repeated search finds 16 hits again)
                int at = 0;
                if (lane == 0) at = atomicAdd(heavy_count, 32);
                heavy[__shfl_sync(FULL, at, 0) + lane] = active ? slot : -1;
                if (active) { req_bound(req, slot) = kmax; continue; }
                n = 0;
            }
        }
        if (slot >= 0) {
            kcnt[slot] = n;
#pragma unroll
            for (int i = 0; i < DST_CHUNK; i++) if (i < n) kbuf[soa(slot, i, DST_CHUNK)] = kb[i * KS];
        }
    }
    if (COUNT && counters) { atomicAdd(counters + 1, tc.enums); atomicAdd(counters + 2, tc.nodes); atomicAdd(counters + 3, tc.quads); }
}

// Takes the hits found by one quad step (lanes with `hit`, in `key`) into the sorted k-buffer held by lanes 0..15 (`mine`, ~0 where empty). Every
// hit is handed round once: a lane counts the hits below its own hit and below its buffer entry, and a ballot the entries below
// each hit. The counts are the new places; nothing waits for the hit before (one insertion after the other was a chain of seven
// cross-lane operations per hit, a fifth of the latency of a walk). place: DST_CHUNK words of shared memory of the warp.
__device__ __forceinline__ void take_hits(bool hit, unsigned long long key, unsigned long long& mine, unsigned long long* place) {
    constexpr unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned long long last = __shfl_sync(FULL, mine, DST_CHUNK - 1);
    unsigned int hits = __ballot_sync(FULL, hit && key < last);      // (nearer than the 16th)
    if (hits == 0u) return;
    hit = (hits >> lane) & 1u;
    const bool held = lane < DST_CHUNK && mine != ~0ull;
    int at = 0, old_at = lane;
    while (hits) {
        const int hl = __ffs(hits) - 1;
        hits &= hits - 1u;
        const unsigned long long k = __shfl_sync(FULL, key, hl);
        const int below = __popc(__ballot_sync(FULL, held && mine < k));
        at += lane == hl ? below : (k < key ? 1 : 0);
        old_at += k < mine ? 1 : 0;
    }
    const int n = __popc(__ballot_sync(FULL, held)) + __popc(__ballot_sync(FULL, hit));
    __syncwarp();
    if (held && old_at < DST_CHUNK) place[old_at] = mine;
    if (hit && at < DST_CHUNK) place[at] = key;
    __syncwarp();
    mine = lane < n && lane < DST_CHUNK ? place[lane] : ~0ull;
}

// The 16 nearest hits of ONE ray, found by a whole warp (same result as knearest()): the walk of a hull that is a single
// ray, its quads tested exactly, one per lane. The k-buffer lives in registers, one key per lane (lanes 0..15, ascending).
// All arguments are warp-uniform.
template <bool COUNT>
__device__ __forceinline__ int knearest_warp(const BvhView& bvh, float ox, float oy, float oz, float dx, float dy, float dz, float kmax0, float absmax,
                                             WalkMem& m, unsigned long long& mykey, unsigned int* status, TraceCounters& tc) {
    constexpr unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    mykey = ~0ull;
    if (bvh.P <= 0) return 0;
    if (!(fabsf(ox) < INFINITY && fabsf(oy) < INFINITY && fabsf(oz) < INFINITY && fabsf(dx) < INFINITY && fabsf(dy) < INFINITY && fabsf(dz) < INFINITY)) return 0;
    make_ray(m, ox, oy, oz, dx, dy, dz, absmax);
    float krun = kmax0;
    const bool done = beam_walk<COUNT>(bvh, m, krun, DST_WALK_STEP_LIMIT, status, tc, [&](bool valid, int pos) {
        bool hit = false;
        unsigned long long key = 0ull;
        if (valid) {
            const Quad q = load_quad(bvh, pos);
            float t; int tri;
            if (COUNT) tc.quads++;
            if (ray_quad(q.a, q.b, q.c, ox, oy, oz, dx, dy, dz, krun, t, tri)) {
                key = make_key(t, 2u * q.gid + (unsigned int)tri);
                hit = true;
            }
        }
        take_hits(hit, key, mykey, m.place);
        const unsigned long long last = __shfl_sync(FULL, mykey, DST_CHUNK - 1);
        if (last != ~0ull) krun = hitkey_t(last);
        return true;
    });
    if (!done && lane == 0) atomicOr(status, DST_STATUS_STACK_OVERFLOW);
    return __popc(__ballot_sync(FULL, lane < DST_CHUNK && mykey != ~0ull));
}

// Second step of a gather: the batches k_enum gave up, in groups of DST_GROUP rays, one warp per group. The walk is again
// that of the group's hull; a quad step tests its 32 quads (one per lane) exactly against one ray of the group after the
// other. The k-buffers are in shared memory; lanes 0..15 hold one of them at a time.
template <bool COUNT>
__global__ void __launch_bounds__(ENUM_THREADS, DST_GROUP_MIN_BLOCKS) k_enum_group(BvhView bvh, float4* req, const int* __restrict__ list,
                                                       const int* __restrict__ count_ptr, int* cursor,
                                                       unsigned long long* __restrict__ kbuf, int* __restrict__ kcnt,
                                                       unsigned int* status, unsigned long long* counters, int* heavy, int* heavy_count, int direct_max, int slices) {
    constexpr unsigned int FULL = 0xffffffffu;
    __shared__ BeamMem walk_mem[ENUM_THREADS / 32];
    __shared__ unsigned long long skeys[ENUM_THREADS / 32][DST_GROUP][DST_CHUNK];
    __shared__ float4 srays[ENUM_THREADS / 32][DST_GROUP][2];
    const int total = *count_ptr / DST_GROUP;
    if (total * DST_GROUP <= direct_max) return;        // none, or few enough for a warp per ray (k_enum_ray takes them)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    BeamMem& m = walk_mem[w];
    const int max_steps = (long long)total * slices > DST_LOADED_GROUPS * (long long)(gridDim.x * (ENUM_THREADS / 32)) ? DST_GROUP_STEPS_LOADED : DST_GROUP_STEPS;
    const float absmax = __ldg(bvh.header + 6);
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(cursor, 1);
        i = __shfl_sync(FULL, i, 0);
        if (i >= total) break;
        const int slot = lane < DST_GROUP ? list[i * DST_GROUP + lane] : -1;
        const unsigned int members = __ballot_sync(FULL, slot >= 0);
        if (members == 0u) continue;
        EnumReq q = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1.0f, 0.f };
        if (slot >= 0) q = load_req(req, slot);
        const HullStart hs = hull_start(slot >= 0, q);
        if (lane < DST_GROUP) {
            float x, y, z;
            q.start(x, y, z);
            srays[w][lane][0] = make_float4(x, y, z, q.dx); srays[w][lane][1] = make_float4(q.dy, q.dz, q.kmax0, hs.rel);
        }
        for (int k = lane; k < DST_GROUP * DST_CHUNK; k += 32) (&skeys[w][0][0])[k] = ~0ull;
        make_beam(m, slot >= 0, hs, q.dx, q.dy, q.dz, absmax);
        float krun = redux_max(from_hull(hs.rel, q.kmax0));
        const bool done = beam_walk<COUNT>(bvh, m, krun, max_steps, status, tc, [&](bool valid, int pos) {
            Quad q;
            q.a = q.b = q.c = make_float4(0.f, 0.f, 0.f, 0.f); q.gid = 0u;
            if (valid) { q = load_quad(bvh, pos); if (COUNT) tc.quads++; }
            float kall = -1.0f;
#pragma unroll 1
            for (int r = 0; r < DST_GROUP; r++) {
                const float4 ra = srays[w][r][0], rb = srays[w][r][1];
                float t; int tri;
                const bool hit = valid && ray_quad(q.a, q.b, q.c, ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, t, tri);
                float kr = rb.z;
                if (__any_sync(FULL, hit)) {
                    const unsigned long long key = make_key(t, 2u * q.gid + (unsigned int)tri);
                    unsigned long long mine = lane < DST_CHUNK ? skeys[w][r][lane] : ~0ull;
                    take_hits(hit, key, mine, m.place);
                    const unsigned long long last = __shfl_sync(FULL, mine, DST_CHUNK - 1);
                    if (lane < DST_CHUNK) skeys[w][r][lane] = mine;
                    if (last != ~0ull) { kr = hitkey_t(last); if (lane == 0) srays[w][r][1].z = kr; }
                }
                kall = fmaxf(kall, from_hull(rb.w, kr));
            }
            krun = kall;
            __syncwarp();
            return true;
        });
        __syncwarp();
        if (done) {
#pragma unroll 1
            for (int r = 0; r < DST_GROUP; r++) {
                if (!((members >> r) & 1u)) continue;
                const int to = __shfl_sync(FULL, slot, r);
                const unsigned long long mine = skeys[w][r][lane & (DST_CHUNK - 1)];
                const int n = __popc(__ballot_sync(FULL, lane < DST_CHUNK && mine != ~0ull));
                if (lane < n) kbuf[soa(to, lane, DST_CHUNK)] = mine;
                if (lane == 0) kcnt[to] = n | DST_KCNT_WIDE;
            }
        } else {
            int at = 0;
            if (lane == 0) at = atomicAdd(heavy_count, __popc(members));
            at = __shfl_sync(FULL, at, 0) + __popc(members & ((1u << lane) - 1u));
            if (slot >= 0) { heavy[at] = slot; req_bound(req, slot) = srays[w][lane][1].z; }
        }
        __syncwarp();
    }
    if (COUNT && counters) { atomicAdd(counters + 2, tc.nodes); atomicAdd(counters + 3, tc.quads); }
}

// Last step of a gather: the rays whose group was given up, one warp per ray. When k_enum gave up no more rays than the GPU has room for
// warps (direct_max) these are all of its rays: a group's walk tests eight rays one after the other, and a few of them made every
// round of a small call or of its end half as long again.
template <bool COUNT>
__global__ void __launch_bounds__(ENUM_THREADS, DST_GROUP_MIN_BLOCKS) k_enum_ray(BvhView bvh, const float4* __restrict__ req, const int* __restrict__ heavy,
                                                       const int* __restrict__ heavy_count, const int* __restrict__ heavy2, const int* __restrict__ heavy2_count,
                                                       int* cursor, int direct_max,
                                                       unsigned long long* __restrict__ kbuf, int* __restrict__ kcnt,
                                                       unsigned int* status, unsigned long long* counters) {
    __shared__ WalkMem walk_mem[ENUM_THREADS / 32];
    const int given_up = *heavy_count;
    const int* list = given_up <= direct_max ? heavy : heavy2;
    const int total = given_up <= direct_max ? given_up : *heavy2_count;
    if (total <= 0) return;
    const int lane = threadIdx.x & 31;
    WalkMem& m = walk_mem[threadIdx.x >> 5];
    const float absmax = __ldg(bvh.header + 6);
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(cursor, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= total) break;
        const int slot = list[i];
        if (slot < 0) continue;
        const EnumReq q = load_req(req, slot);
        float x, y, z;
        q.start(x, y, z);
        unsigned long long key;
        const int n = knearest_warp<COUNT>(bvh, x, y, z, q.dx, q.dy, q.dz, q.kmax0, absmax, m, key, status, tc);
        if (lane < n) kbuf[soa(slot, lane, DST_CHUNK)] = key;
        if (lane == 0) kcnt[slot] = n | DST_KCNT_WIDE;
        __syncwarp();
    }
    if (COUNT && counters) { atomicAdd(counters + 2, tc.nodes); atomicAdd(counters + 3, tc.quads); }
}

// the gather launches of a wavefront round (diag: with traversal counters). cnt: the round's entry in the set of round counters;
// heavy, heavy2: lists of as many rays as the round has slots; slices: slices of the call, this one included
static inline void launch_gather(bool diag, int grid, int sm_count, int slices, cudaStream_t st, const BvhView& bvh, float4* req, const int* list,
                                 const int* count_ptr, int* cnt, int min_count, unsigned long long* kbuf, int* kcnt, unsigned int* status,
                                 unsigned long long* counters, int* heavy, int* heavy2) {
    constexpr int R = DST_WF_ROUNDS + 2;
    const int direct_max = sm_count * DST_GROUP_MIN_BLOCKS * (ENUM_THREADS / 32), ray_grid = sm_count * DST_GROUP_MIN_BLOCKS;
    const int group_slices = slices < DST_GROUP_LOAD_SLICES ? slices : DST_GROUP_LOAD_SLICES;
    if (diag) {
        k_enum<true><<<grid, ENUM_THREADS, 0, st>>>(bvh, req, list, count_ptr, cnt + R, min_count, kbuf, kcnt, status, counters, heavy, cnt + 2 * R, slices);
        k_enum_group<true><<<grid, ENUM_THREADS, 0, st>>>(bvh, req, heavy, cnt + 2 * R, cnt + 3 * R, kbuf, kcnt, status, counters, heavy2, cnt + 4 * R, direct_max, group_slices);
        k_enum_ray<true><<<ray_grid, ENUM_THREADS, 0, st>>>(bvh, req, heavy, cnt + 2 * R, heavy2, cnt + 4 * R, cnt + 5 * R, direct_max, kbuf, kcnt, status, counters);
    } else {
        k_enum<false><<<grid, ENUM_THREADS, 0, st>>>(bvh, req, list, count_ptr, cnt + R, min_count, kbuf, kcnt, status, nullptr, heavy, cnt + 2 * R, slices);
        k_enum_group<false><<<grid, ENUM_THREADS, 0, st>>>(bvh, req, heavy, cnt + 2 * R, cnt + 3 * R, kbuf, kcnt, status, nullptr, heavy2, cnt + 4 * R, direct_max, group_slices);
        k_enum_ray<false><<<ray_grid, ENUM_THREADS, 0, st>>>(bvh, req, heavy, cnt + 2 * R, heavy2, cnt + 4 * R, cnt + 5 * R, direct_max, kbuf, kcnt, status, nullptr);
    }
}

// List slot i -> ray index (or -1). Image-like grids are walked in 8x4 pixel tiles (one tile = the 32
// rays a warp of the gather kernel takes), and the tiles in Z order inside blocks of 8x8 tiles (64x32 pixels): any
// aligned run of 2 or 4 consecutive tiles is a compact 16x4 or 16x8 pixel patch. That matters once rays have
// dropped out: the lists keep this order, so a warp of a later round holds the survivors of a few consecutive
// tiles, and the tighter the patch they come from, the tighter the hull of their rays. Batched ray lists (few rows)
// are walked linearly.
#ifndef DST_TILE_BLOCK
#define DST_TILE_BLOCK 8              // tiles per side of a Z-ordered block (1: row-major tile order)
#endif
__device__ __forceinline__ int slot_ray(long long i, int H, int W, bool tiled) {
    if (!tiled) return i < (long long)H * W ? (int)i : -1;
    const int tiles_x = (W + 7) >> 3;
    long long tile = i >> 5;
    const int lane = (int)(i & 31);
    int tx, ty;
    if (DST_TILE_BLOCK > 1) {
        constexpr int BB = DST_TILE_BLOCK * DST_TILE_BLOCK;
        const int blocks_x = (tiles_x + DST_TILE_BLOCK - 1) / DST_TILE_BLOCK;
        const long long blk = tile / BB;
        const unsigned int in = (unsigned int)(tile - blk * BB);
        // Z order inside the block: even bits -> x, odd bits -> y
        const unsigned int zx = (in & 1u) | ((in >> 1) & 2u) | ((in >> 2) & 4u), zy = ((in >> 1) & 1u) | ((in >> 2) & 2u) | ((in >> 3) & 4u);
        tx = (int)(blk % blocks_x) * DST_TILE_BLOCK + (int)zx;
        ty = (int)(blk / blocks_x) * DST_TILE_BLOCK + (int)zy;
    } else { tx = (int)(tile % tiles_x); ty = (int)(tile / tiles_x); }
    const int x = tx * 8 + ((lane & 1) | ((lane >> 1) & 2) | ((lane >> 2) & 4));      // Z order inside the tile too: 8 consecutive lanes are a 4x2 patch
    const int y = ty * 4 + (((lane >> 1) & 1) | ((lane >> 2) & 2));
    if (x >= W || y >= H) return -1;
    return y * W + x;
}
__host__ __device__ __forceinline__ long long slots_of_grid(int H, int W, bool tiled) {
    if (!tiled) return (long long)H * W;
    const long long tiles_x = (W + 7) >> 3, tiles_y = (H + 3) >> 2;
    if (DST_TILE_BLOCK > 1) {
        const long long bx = (tiles_x + DST_TILE_BLOCK - 1) / DST_TILE_BLOCK, by = (tiles_y + DST_TILE_BLOCK - 1) / DST_TILE_BLOCK;
        return bx * by * DST_TILE_BLOCK * DST_TILE_BLOCK * 32;
    }
    return tiles_x * tiles_y * 32;
}

// appends `ray` to the next round's list when `alive`; one atomic per warp, order kept within a warp
__device__ __forceinline__ void append_alive(bool alive, int ray, int* __restrict__ next_list, int* next_count) {
    __syncwarp();
    const unsigned int m = __ballot_sync(__activemask(), alive);
    if (!alive) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(next_count, __popc(m));
    base = __shfl_sync(m, base, leader);
    next_list[base + __popc(m & ((1u << lane) - 1u))] = ray;
}

// ---------------------------------------------------------------------------------------------
// Order-preserving hand-over of the live list from one round to the next.
//
// append_alive() above packs the survivors of every warp behind one atomic counter: cheap, but the
// warps arrive in whatever order the scheduler ran them, so after a few rounds neighbouring list
// entries are unrelated rays and the gather kernel's shared walk (one hierarchy walk for 32
// neighbouring rays) falls apart. The stable form keeps the list in its original order (8x4 pixel
// tiles, tile after tile) and, within that, puts rays on their primary segment before rays on a
// reflected one, so that a warp of the next round again holds rays that start close together and
// are in the same stage:
//   shade kernel   live_out(): survivor (or -1) of list position i into tmp[i]; survivors per warp
//                  and class into wcnt[i / 32]; the same added to the counter of the 4096-entry
//                  block the position lies in (bcnt, two classes packed 16 + 16 bits).
//   k_compact      one block per 4096 positions: sums the block counters before its own (and all of
//                  them, for the start of the second class), scans its 128 warp counts and copies
//                  every survivor to its final position. Block 0 publishes the new list length.
// The block counters come in two sets used by alternate rounds; k_compact of round r clears the set
// round r + 1 accumulates into (nothing waits on anything: all of this is ordinary stream order).
// ---------------------------------------------------------------------------------------------
#define DST_LIVE_BLOCK 4096
#define DST_LIVE_CLASS_BIT 30            // slot numbers stay below 2^30 (dst_slot_grid)
struct LiveLists {
    int* tmp;            // per list position of the current round: slot | class << 30, or -1
    int* wcnt;           // per 32 positions: survivors of class 0 | survivors of class 1 << 16
    int* bcnt[2];        // per DST_LIVE_BLOCK positions, same packing; set (round & 1) belongs to the current round
    int stable;          // 0: append_alive() order (atomic per warp)
};
static inline long long dst_live_blocks(long long slots) { return slots / DST_LIVE_BLOCK + 2; }
int dst_live_lists(dst_handle* h, LiveLists* lv, cudaStream_t st);

// called by all 32 lanes of a warp for 32 consecutive list positions (i of lane 0 is a multiple of 32)
__device__ __forceinline__ void live_out(const LiveLists& lv, int round, int i, bool alive, int ray, int cls) {
    __syncwarp();
    const unsigned int m0 = __ballot_sync(0xffffffffu, alive && cls == 0), m1 = __ballot_sync(0xffffffffu, alive && cls != 0);
    lv.tmp[i] = alive ? (ray | (cls != 0 ? (1 << DST_LIVE_CLASS_BIT) : 0)) : -1;
    if ((threadIdx.x & 31) == 0) {
        const int packed = __popc(m0) | (__popc(m1) << 16);
        lv.wcnt[i >> 5] = packed;
        if (packed) atomicAdd(lv.bcnt[round & 1] + i / DST_LIVE_BLOCK, packed);
    }
}

static __global__ void __launch_bounds__(256) k_compact(LiveLists lv, const int* __restrict__ count_ptr, int* next_count, int min_count,
                                                        int* __restrict__ next_list, int round) {
    __shared__ int red[4][8];
    __shared__ int woff[DST_LIVE_BLOCK / 32];
    const int n = *count_ptr;
    if (n < min_count) return;
    const int nb = (n + DST_LIVE_BLOCK - 1) / DST_LIVE_BLOCK;
    const int b = blockIdx.x;
    if (b >= nb) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int* bc = lv.bcnt[round & 1];
    // survivors per class in the blocks before this one, and in all blocks
    int before0 = 0, before1 = 0, all0 = 0, all1 = 0;
    for (int j = threadIdx.x; j < nb; j += 256) {
        const int c = bc[j], c0 = c & 0xffff, c1 = c >> 16;
        all0 += c0; all1 += c1;
        if (j < b) { before0 += c0; before1 += c1; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        before0 += __shfl_xor_sync(0xffffffffu, before0, o); before1 += __shfl_xor_sync(0xffffffffu, before1, o);
        all0 += __shfl_xor_sync(0xffffffffu, all0, o); all1 += __shfl_xor_sync(0xffffffffu, all1, o);
    }
    if (lane == 0) { red[0][w] = before0; red[1][w] = before1; red[2][w] = all0; red[3][w] = all1; }
    // exclusive scan of this block's 128 warp counts (both classes in one packed add: sums stay below 2^16)
    const int wpos = b * (DST_LIVE_BLOCK / 32) + threadIdx.x;
    int x = 0;
    if (threadIdx.x < DST_LIVE_BLOCK / 32 && wpos * 32 < n) x = lv.wcnt[wpos];
    int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    __shared__ int wsum[8];
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    before0 = before1 = all0 = all1 = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) { before0 += red[0][k]; before1 += red[1][k]; all0 += red[2][k]; all1 += red[3][k]; }
    if (threadIdx.x < DST_LIVE_BLOCK / 32) {
        int carry = 0;
        for (int k = 0; k < w; k++) carry += wsum[k];
        woff[threadIdx.x] = carry + incl - x;
    }
    __syncthreads();
    if (b == 0 && threadIdx.x == 0) *next_count = all0 + all1;
    if (threadIdx.x == 0) lv.bcnt[(round + 1) & 1][b] = 0;          // the set the next round accumulates into
    // every warp copies 16 groups of 32 positions
    for (int g = w; g < DST_LIVE_BLOCK / 32; g += 8) {
        const int i = (b * (DST_LIVE_BLOCK / 32) + g) * 32 + lane;
        const int v = i < n ? lv.tmp[i] : -1;          // positions up to the next multiple of 32 were written, the rest is dead
        const bool alive = v >= 0;
        const bool second = alive && ((v >> DST_LIVE_CLASS_BIT) & 1);
        const unsigned int m0 = __ballot_sync(0xffffffffu, alive && !second), m1 = __ballot_sync(0xffffffffu, second);
        if (!alive) continue;
        const int off = woff[g], below = (1u << lane) - 1u;
        const int pos = second ? all0 + before1 + (off >> 16) + __popc(m1 & below) : before0 + (off & 0xffff) + __popc(m0 & below);
        next_list[pos] = v & ((1 << DST_LIVE_CLASS_BIT) - 1);
    }
}

// first round the wavefront kernels left alone (list shorter than min_count)
__device__ __forceinline__ int first_skipped_round(const int* __restrict__ counts, int rounds, int min_count) {
    for (int r = 0; r < rounds; r++) if (counts[r] < min_count) return r;
    return rounds;
}
