// Backward trace: replaces optix_tracer/backward.cu (__raygen__ot 857-928, tracePath 658-853,
// traceRay 332-655 and its helpers) and the host launcher TraceSurfelsBackwardCUDA
// (trace_surfels.cpp:307-464).
//
// Bounces are visited last to first, each segment front to back with the forward kernel's exact evaluation (eval_slot), and every
// contributing hit adds its gradients. Where the forward left a contribution log, k_bwd_logged composites it again; rays without one are
// traced again as wavefront rounds (the gather kernels, k_bwd_shade) with a tail of one warp per few rays. Per-surfel gradients go to
// a packed arena of 16-byte aligned rows: rows are staged in shared memory, those of lanes with the same surfel added up there, and
// leave as one bulk reduction each (see send_rows); a streaming kernel unpacks the arena into the caller's tensors afterwards.
#include "dst_trace.cuh"

namespace {

#ifndef DST_BWD_THREADS
#define DST_BWD_THREADS 128
#endif
constexpr int BWD_THREADS = DST_BWD_THREADS;
#ifndef DST_BWD_BLOCKS
#define DST_BWD_BLOCKS 4               // resident blocks per SM the backward kernels are compiled for
#endif

struct BwdParams {
    dst_bwd_args a;
    BvhView bvh;
    const float4* cache;
    float* arena;
    unsigned int* status;
    int tiled, grid_h, grid_w;      // ray order, as in the forward
    int dist_on;                    // depth-distortion extension
    // wavefront scratch
    float4* state;
    float4* req;
    unsigned long long* kbuf;
    int* kcnt;
    int* list[2];
    int* counts;
    int min_count;
    int rounds;
    LiveLists lv;
    // contribution log of the matching forward call, see dst_begin_log()
    const unsigned long long* log_keys; const int* log_next; const int* log_head; const int* log_num; const unsigned char* log_ok;
    long long log_slots;
};

struct __align__(16) BwdState {
    float sox, soy, soz, sdx;
    float sdy, sdz, offset, dpt;
    float T_prev, rem, s_prod, Cp0;       // rem: what lies behind the hits composited so far, weighted with the upstream gradients (see bwd_chunk)
    float Cp1, Cp2, cp0, cp1;
    float cp2, t_rgb0, t_rgb1, t_rgb2;
    float t_dpt, t_acc, t_aux0, t_aux1;
    float t_nx, t_ny, t_nz, dir_g0;
    float dir_g1, dir_g2, dro_x, dro_y;
    float dro_z, drd_x, drd_y, drd_z;
    int last_gidx, contributor, chunk, seg;
    int dir_gidx;
    float dm0, dvs, dws;        // distortion term on the primary segment: mapped depth of the first contribution, running sums of w c^2 and w
};
static_assert(sizeof(BwdState) == 176, "ray state is eleven 16-byte words");

// ---------------------------------------------------------------------------------------------
// Gradient rows leave the SM as bulk reductions. A contribution adds an 80-byte row to the packed arena and (with
// SH colours) a row of coefficient gradients. As vector reductions those are 5 + 12 red.global.add.v4.f32 per contribution
// and lane, and the L2's reduction path is what the kernel then waits for. Instead a row is staged in shared memory and handed
// to the bulk copy engine as ONE cp.reduce.async.bulk (shared -> global, add.f32). Bulk operations want 16-byte aligned
// addresses and sizes that are multiples of 16 bytes: arena rows always qualify, SH rows when the gradient tensor is 16-byte
// aligned and 12 * (degree + 1)^2 is a multiple of 16 (degrees 1 and 3); other SH rows are added with scalar reductions.
//
// The lanes of a warp are neighbouring pixels that composite their chunks in step, so at one point of the hit loop most of
// them hold one of a handful of surfels. Their rows are summed in shared memory and leave as one. An SH row is the product of the 16
// basis values of the ray's direction, which stay the same for a whole segment, and three colour gradients: a lane stages the three,
// and the sum over the lanes of a group is formed from them and the basis values in shared memory.
// ---------------------------------------------------------------------------------------------
struct BwdWarp {
    float rows[32][DST_ARENA_FLOATS];   // lane's arena row
    float sh[32][48];                   // SH row of the lanes that send one
    float4 colour[32];                  // colour gradients of the lane's contribution (clamped channels 0)
    float basis[16][33];                // SH basis of the lane's segment direction, one column per lane
};
constexpr size_t BWD_STAGE_BYTES = sizeof(BwdWarp) * (BWD_THREADS / 32);   // dynamic shared memory of every backward kernel

// adds `bytes` bytes of floats at shared-memory `src` to global `dst` (both 16-byte aligned, bytes a multiple of 16)
__device__ __forceinline__ void bulk_add(float* dst, const float* src, int bytes) {
    const unsigned int s = (unsigned int)__cvta_generic_to_shared(src);
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" :: "l"(dst), "r"(s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }      // the engine has read this lane's rows
__device__ __forceinline__ void bulk_drain() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }               // ... and added them: before the kernel ends
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }            // staged values become visible to the engine

struct RowTarget { float* arena; float* dsh; int coeffs, ncoef; bool bulk; };       // dsh null: no SH colours

// Sends the contributions staged by the lanes with gidx >= 0 (the others pass -1); called by all 32 lanes. `group`: sum the rows of
// lanes with the same surfel where neighbours do hold the same ones: when fewer than three quarters of the rows have the surfel of
// the lane next door, every lane sends its own (grouping costs more than it saves where surfels are small against the pixel spacing).
__device__ __forceinline__ void send_rows(const RowTarget& t, BwdWarp& ws, int gidx, bool group) {
    constexpr unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int staged = __ballot_sync(FULL, gidx >= 0);
    if (staged == 0u) return;
    unsigned int peers = 1u << lane;
    if (group) {
        const int next_door = __shfl_xor_sync(FULL, gidx, 1);
        const unsigned int paired = __ballot_sync(FULL, gidx >= 0 && next_door == gidx);
        if (4 * __popc(paired) >= 3 * __popc(staged)) peers = __match_any_sync(FULL, gidx);
    }
    const bool alone = gidx >= 0 && (peers & (peers - 1u)) == 0u;
    if (t.dsh && alone) {       // a row of its own
        const float4 m = ws.colour[lane];
        if (t.bulk) {
            float4* o = reinterpret_cast<float4*>(ws.sh[lane]);
#pragma unroll
            for (int q = 0; q < 4; q++) {       // four basis values are three float4 of the row
                if (4 * q < t.ncoef) {
                    const float b0 = ws.basis[4 * q][lane], b1 = ws.basis[4 * q + 1][lane], b2 = ws.basis[4 * q + 2][lane], b3 = ws.basis[4 * q + 3][lane];
                    o[3 * q] = make_float4(b0 * m.x, b0 * m.y, b0 * m.z, b1 * m.x);
                    o[3 * q + 1] = make_float4(b1 * m.y, b1 * m.z, b2 * m.x, b2 * m.y);
                    o[3 * q + 2] = make_float4(b2 * m.z, b3 * m.x, b3 * m.y, b3 * m.z);
                }
            }
        } else {
            float* d = t.dsh + 3 * (size_t)gidx * t.coeffs;
            for (int j = 0; j < t.ncoef; j++) {
                const float b = ws.basis[j][lane];
                atomicAdd(d + 3 * j, b * m.x); atomicAdd(d + 3 * j + 1, b * m.y); atomicAdd(d + 3 * j + 2, b * m.z);
            }
        }
    }
    __syncwarp();                                                        // every lane's row is staged
    // Groups, one after the other. The lanes share the sums of a row out: floats 0..15 to lanes 16..31, 16..19 to lanes 0..3; SH
    // coefficient j, channels 0 and 1 to lane j, channel 2 to lane 16 + j.
    const int j = lane & 15, upper = lane >> 4;
    const float* col = &ws.rows[0][upper ? j : 16 + (lane & 3)];
    const float* bas = &ws.basis[j][0];
    const float2* clr = reinterpret_cast<const float2*>(ws.colour) + upper;
    const bool leads = gidx >= 0 && lane == __ffs(peers) - 1;            // (so does every lane with a row of its own)
    for (unsigned int todo = __ballot_sync(FULL, leads && !alone); todo; todo &= todo - 1u) {
        const int lead = __ffs(todo) - 1;
        unsigned int q = __shfl_sync(FULL, peers, lead);
        const int g = __shfl_sync(FULL, gidx, lead);
        float a = 0.0f, c0 = 0.0f, c1 = 0.0f;
        do {                                                             // two rows per pass (the second with weight 0 where there is none)
            const int r0 = __ffs(q) - 1;
            q &= q - 1u;
            const int r1 = q ? __ffs(q) - 1 : r0;
            const float w1 = q ? 1.0f : 0.0f;
            q &= q - 1u;
            a += fmaf(w1, col[r1 * DST_ARENA_FLOATS], col[r0 * DST_ARENA_FLOATS]);
            if (t.dsh) {
                const float2 m0 = clr[2 * r0], m1 = clr[2 * r1];
                const float b0 = bas[r0], b1 = w1 * bas[r1];
                c0 = fmaf(b0, m0.x, c0); c1 = fmaf(b0, m0.y, c1);
                c0 = fmaf(b1, m1.x, c0); c1 = fmaf(b1, m1.y, c1);
            }
        } while (q);
        __syncwarp();
        if (upper) ws.rows[lead][j] = a; else if (lane < 4) ws.rows[lead][16 + lane] = a;
        if (t.dsh && j < t.ncoef) {
            if (t.bulk) {
                if (upper) ws.sh[lead][3 * j + 2] = c0; else { ws.sh[lead][3 * j] = c0; ws.sh[lead][3 * j + 1] = c1; }
            } else {
                float* d = t.dsh + 3 * ((size_t)g * t.coeffs + j);
                if (upper) atomicAdd(d + 2, c0); else { atomicAdd(d, c0); atomicAdd(d + 1, c1); }
            }
        }
    }
    // All rows leave together. What this kernel takes is instructions and their latency; a fence, a wait for the warp and a send by one lane after every
    // group's sum cost 2.6 % of it (logged backward of 2M reflective rays 13.64 -> 13.28 ms, of 2M with two bounces 26.1 -> 25.5). Tried beside it: four rows
    // per pass of the sum (14.6 ms), SH rows staged 14 at a time for more L1 (13.4, but 27.5 with two bounces and 7 % slower where rows are not grouped).
    bulk_fence();
    __syncwarp();
    if (leads) {
        bulk_add(t.arena + (size_t)gidx * DST_ARENA_FLOATS, ws.rows[lane], DST_ARENA_FLOATS * 4);
        if (t.bulk) bulk_add(t.dsh + 3 * (size_t)gidx * t.coeffs, ws.sh[lane], 12 * t.ncoef);
        bulk_commit();
    }
}

struct V3 { float x, y, z; };
__device__ __forceinline__ V3 v3(float x, float y, float z) { V3 r; r.x = x; r.y = y; r.z = z; return r; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 operator*(float s, V3 a) { return v3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) { return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x); }

// optix_tracer/auxiliary.h:111-121
__device__ __forceinline__ V3 dnormvdv(V3 v, V3 dv) {
    const float sum2 = v.x * v.x + v.y * v.y + v.z * v.z;
    const float inv = 1.0f / sqrtf(sum2 * sum2 * sum2);
    return v3(((sum2 - v.x * v.x) * dv.x - v.y * v.x * dv.y - v.z * v.x * dv.z) * inv,
              (-v.x * v.y * dv.x + (sum2 - v.y * v.y) * dv.y - v.z * v.y * dv.z) * inv,
              (-v.x * v.z * dv.x - v.y * v.z * dv.y + (sum2 - v.z * v.z) * dv.z) * inv);
}
// optix_tracer/auxiliary.h:234-243
__device__ __forceinline__ V3 ddotndndn(V3 n, V3 d, V3 g) {
    const float nd = dot(n, d);
    return v3(g.x * (nd + d.x * n.x) + g.y * d.x * n.y + g.z * d.x * n.z,
              g.x * d.y * n.x + g.y * (nd + d.y * n.y) + g.z * d.y * n.z,
              g.x * d.z * n.x + g.y * d.z * n.y + g.z * (nd + d.z * n.z));
}
// optix_tracer/auxiliary.h:245-252
__device__ __forceinline__ V3 ddotndndd(V3 n, V3 g) {
    const float s = g.x * n.x + g.y * n.y + g.z * n.z;
    return v3(s * n.x, s * n.y, s * n.z);
}

// direction gradient of the SH colour (optix_tracer/backward.cu:96-165), s[j] = sh[j] . dL_dRGB
__device__ __forceinline__ V3 sh_dir_grad(int deg, const float* s, float x, float y, float z) {
    float gx = 0.f, gy = 0.f, gz = 0.f;
    if (deg > 0) {
        gx = -SHC1 * s[3]; gy = -SHC1 * s[1]; gz = SHC1 * s[2];
        if (deg > 1) {
            const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
            gx += SHC2_0 * y * s[4] + SHC2_2 * 2.f * -x * s[6] + SHC2_3 * z * s[7] + SHC2_4 * 2.f * x * s[8];
            gy += SHC2_0 * x * s[4] + SHC2_1 * z * s[5] + SHC2_2 * 2.f * -y * s[6] + SHC2_4 * 2.f * -y * s[8];
            gz += SHC2_1 * y * s[5] + SHC2_2 * 4.f * z * s[6] + SHC2_3 * x * s[7];
            if (deg > 2) {
                gx += SHC3_0 * s[9] * 6.f * xy + SHC3_1 * s[10] * yz + SHC3_2 * s[11] * -2.f * xy + SHC3_3 * s[12] * -6.f * xz +
                      SHC3_4 * s[13] * (-3.f * xx + 4.f * zz - yy) + SHC3_5 * s[14] * 2.f * xz + SHC3_6 * s[15] * 3.f * (xx - yy);
                gy += SHC3_0 * s[9] * 3.f * (xx - yy) + SHC3_1 * s[10] * xz + SHC3_2 * s[11] * (-3.f * yy + 4.f * zz - xx) +
                      SHC3_3 * s[12] * -6.f * yz + SHC3_4 * s[13] * -2.f * xy + SHC3_5 * s[14] * -2.f * yz + SHC3_6 * s[15] * -6.f * xy;
                gz += SHC3_1 * s[10] * xy + SHC3_2 * s[11] * 8.f * yz + SHC3_3 * s[12] * 3.f * (2.f * zz - xx - yy) +
                      SHC3_4 * s[13] * 8.f * xz + SHC3_5 * s[14] * (xx - yy);
            }
        }
    }
    return v3(gx, gy, gz);
}


__device__ __forceinline__ void bwd_load_state(const float4* base, int slot, BwdState& s) {
    float4* dst = reinterpret_cast<float4*>(&s);
#pragma unroll
    for (int i = 0; i < 11; i++) dst[i] = base[soa(slot, i, 11)];
}
__device__ __forceinline__ void bwd_store_state(float4* base, int slot, const BwdState& s) {
    const float4* src = reinterpret_cast<const float4*>(&s);
#pragma unroll
    for (int i = 0; i < 11; i++) base[soa(slot, i, 11)] = src[i];
}

__device__ __forceinline__ void bwd_request(const BwdState& s, EnumReq& q) {
    q.ox = s.sox; q.oy = s.soy; q.oz = s.soz; q.dx = s.sdx; q.dy = s.sdy; q.dz = s.sdz; q.kmax0 = DST_T_MAX; q.off = s.chunk == 0 ? 0.0f : s.offset;
}

// Finds the next segment to differentiate, from segment `start` downwards (backward.cu:706-802):
// skips the ones the reference skips, derives the segment's upstream gradients and the reflection
// chain, and resets the running sums. Writes the ray gradients and returns false when none is left.
__device__ __forceinline__ bool bwd_next_segment(const BwdParams& p, int ray, BwdState& s, int start) {
    const dst_trace_inputs& in = p.a.in;
    const int depth = in.max_trace_depth;
    const float* mid = p.a.mid_val + (size_t)ray * in.mid_stride;
    for (int i = start; i >= 0; i--) {
        const float4* mp = reinterpret_cast<const float4*>(mid + i * DST_MID_CHANNELS);
        const float4 m0 = __ldg(mp), m1 = __ldg(mp + 1), m2 = __ldg(mp + 2), m3 = __ldg(mp + 3);
        const float sdx = m0.w, sdy = m1.x, sdz = m1.y;
        const float tot_dpt = m1.z;
        const V3 tot_n = v3(m2.x, m2.y, m2.z);
        const float tot_o0 = m2.w, tot_c0 = m3.y, tot_c1 = m3.z, tot_c2 = m3.w;
        const float s_prev = i > 0 ? __ldg(mid + (i - 1) * DST_MID_CHANNELS + 11) : 1.0f;
        if (sqrtf(sdx * sdx + sdy * sdy + sdz * sdz) == 0.0f || s_prev <= in.specular_threshold) continue;    // :724

        // (an upstream gradient that is not given is zero)
        const float* up_rgb = p.a.dL_drgb ? p.a.dL_drgb + 3 * (size_t)ray : nullptr;
        const float g_rgb0 = up_rgb ? __ldg(up_rgb) : 0.f, g_rgb1 = up_rgb ? __ldg(up_rgb + 1) : 0.f, g_rgb2 = up_rgb ? __ldg(up_rgb + 2) : 0.f;
        const float f_this = (i == depth) ? 1.0f : 1.0f - tot_o0;
        s.t_rgb0 = g_rgb0 * f_this * s.s_prod; s.t_rgb1 = g_rgb1 * f_this * s.s_prod; s.t_rgb2 = g_rgb2 * f_this * s.s_prod;   // :760
        s.s_prod /= s_prev;                                                                                   // :762
        s.t_dpt = 0.f; s.t_acc = 0.f; s.t_aux0 = 0.f; s.t_aux1 = 0.f;
        V3 t_norm = v3(0.f, 0.f, 0.f);
        V3 dro = v3(s.dro_x, s.dro_y, s.dro_z), drd = v3(s.drd_x, s.drd_y, s.drd_z);
        if (i != depth) {
            // :769-774
            s.t_aux0 += g_rgb0 * (s.Cp0 / tot_o0) + g_rgb1 * (s.Cp1 / tot_o0) + g_rgb2 * (s.Cp2 / tot_o0);
            if (i > 0) {
                const float4 pm3 = __ldg(reinterpret_cast<const float4*>(mid + (i - 1) * DST_MID_CHANNELS) + 3);
                s.cp0 = pm3.y; s.cp1 = pm3.z; s.cp2 = pm3.w;
            } else { s.cp0 = s.cp1 = s.cp2 = 0.f; }
            s.Cp0 -= s.s_prod * (s.cp0 - tot_c0); s.Cp1 -= s.s_prod * (s.cp1 - tot_c1); s.Cp2 -= s.s_prod * (s.cp2 - tot_c2);
            const float nl = sqrtf(dot(tot_n, tot_n));
            if (nl != 0.0f) {                                                                                 // :778-790
                const V3 d = v3(sdx, sdy, sdz);
                drd = drd + 0.00001f * dro;
                const V3 n = (1.0f / nl) * tot_n;
                s.t_dpt += dro.x * sdx + dro.y * sdy + dro.z * sdz;
                const V3 gm2 = -2.0f * drd;
                t_norm = t_norm + dnormvdv(tot_n, ddotndndn(n, d, gm2));
                drd = tot_dpt * dro + drd + ddotndndd(n, gm2);
            }
        }
        if (i == 0) {                                                                                         // :793-802
            if (p.a.dL_ddpt) s.t_dpt += __ldg(p.a.dL_ddpt + ray);
            if (p.a.dL_dacc) s.t_acc += __ldg(p.a.dL_dacc + ray);
            if (p.a.dL_dnorm) t_norm = t_norm + v3(__ldg(p.a.dL_dnorm + 3 * (size_t)ray), __ldg(p.a.dL_dnorm + 3 * (size_t)ray + 1), __ldg(p.a.dL_dnorm + 3 * (size_t)ray + 2));
            if (p.a.dL_daux) { s.t_aux0 += __ldg(p.a.dL_daux + 2 * (size_t)ray); s.t_aux1 += __ldg(p.a.dL_daux + 2 * (size_t)ray + 1); }
        }
        s.t_nx = t_norm.x; s.t_ny = t_norm.y; s.t_nz = t_norm.z;
        s.drd_x = drd.x; s.drd_y = drd.y; s.drd_z = drd.z;
        s.sox = m0.x; s.soy = m0.y; s.soz = m0.z; s.sdx = sdx; s.sdy = sdy; s.sdz = sdz;
        s.offset = 0.f; s.dpt = 0.f; s.T_prev = 1.f;
        // everything the segment composited, and the background seen through it (counted a second time, as the reference does, :545-548)
        s.rem = s.t_rgb0 * tot_c0 + s.t_rgb1 * tot_c1 + s.t_rgb2 * tot_c2;
        if (in.others_precomp) s.rem += s.t_aux0 * tot_o0 + s.t_aux1 * m3.x;       // (without auxiliaries tot_o0 is zero and t_aux0 a quotient by it)
        s.rem += s.t_dpt * tot_dpt + (t_norm.x * tot_n.x + t_norm.y * tot_n.y + t_norm.z * tot_n.z) + s.t_acc * m1.w +
                (1.0f - m1.w) * (s.t_rgb0 * __ldg(in.background) + s.t_rgb1 * __ldg(in.background + 1) + s.t_rgb2 * __ldg(in.background + 2));
        s.last_gidx = -1; s.contributor = 0; s.chunk = 0; s.seg = i; s.dir_gidx = -1;
        s.dm0 = s.dvs = s.dws = 0.f;
        return true;
    }
    p.a.dL_dray_o[3 * (size_t)ray] = s.dro_x; p.a.dL_dray_o[3 * (size_t)ray + 1] = s.dro_y; p.a.dL_dray_o[3 * (size_t)ray + 2] = s.dro_z;
    p.a.dL_dray_d[3 * (size_t)ray] = s.drd_x; p.a.dL_dray_d[3 * (size_t)ray + 1] = s.drd_y; p.a.dL_dray_d[3 * (size_t)ray + 2] = s.drd_z;
    return false;
}

// backward.cu:683-703 (specular product over all bounces and the colour "behind" each one), then the first segment
__device__ __forceinline__ bool bwd_init_state(const BwdParams& p, int ray, BwdState& s) {
    const dst_trace_inputs& in = p.a.in;
    const float* mid = p.a.mid_val + (size_t)ray * in.mid_stride;
    s.Cp0 = __ldg(p.a.out_rgb + 3 * (size_t)ray); s.Cp1 = __ldg(p.a.out_rgb + 3 * (size_t)ray + 1); s.Cp2 = __ldg(p.a.out_rgb + 3 * (size_t)ray + 2);
    s.cp0 = s.cp1 = s.cp2 = 0.f;
    s.s_prod = 1.0f;
    for (int i = 0; i < in.max_trace_depth; i++) {
        const float4 m3 = __ldg(reinterpret_cast<const float4*>(mid + i * DST_MID_CHANNELS) + 3);
        const float4 m2 = __ldg(reinterpret_cast<const float4*>(mid + i * DST_MID_CHANNELS) + 2);
        s.Cp0 += s.s_prod * (s.cp0 - m3.y); s.Cp1 += s.s_prod * (s.cp1 - m3.z); s.Cp2 += s.s_prod * (s.cp2 - m3.w);
        s.cp0 = m3.y; s.cp1 = m3.z; s.cp2 = m3.w;
        s.s_prod *= m2.w;
    }
    s.dro_x = s.dro_y = s.dro_z = 0.f; s.drd_x = s.drd_y = s.drd_z = 0.f;
    s.dir_g0 = s.dir_g1 = s.dir_g2 = 0.f; s.dm0 = s.dvs = s.dws = 0.f;
    return bwd_next_segment(p, ray, s, in.max_trace_depth);
}

// what the hits of one ray segment have in common
struct BwdSegment { bool use_sh, has_aux, sh_aligned, sh_wide, dist_on; int ncoef; float tot_acc, t_dist, dist_mu, dist_V; };

// Called by the lanes with `in` at the start of a chunk / segment; writes the lane's SH basis.
template <bool DIST>
__device__ __forceinline__ BwdSegment bwd_segment(const BwdParams& p, bool in_seg, int ray, const BwdState& s, BwdWarp& ws) {
    const dst_trace_inputs& in = p.a.in;
    BwdSegment x;
    x.use_sh = in.colors_precomp == nullptr;
    x.has_aux = in.others_precomp != nullptr;
    x.ncoef = (in.sh_degree + 1) * (in.sh_degree + 1);
    x.sh_aligned = (in.sh_coeffs & 3) == 0 && ((reinterpret_cast<uintptr_t>(in.shs) & 15) == 0);
    x.sh_wide = x.ncoef == 16 && in.sh_coeffs == 16 && ((reinterpret_cast<uintptr_t>(in.shs) & 31) == 0);
    x.dist_on = false; x.tot_acc = x.t_dist = x.dist_mu = x.dist_V = 0.f;
    if (x.use_sh && in_seg) {
        float sb[16];
        sh_basis(in.sh_degree, s.sdx, s.sdy, s.sdz, sb);
#pragma unroll
        for (int j = 0; j < 16; j++) if (j < x.ncoef) ws.basis[j][threadIdx.x & 31] = sb[j];
    }
    // Distortion extension (primary segment only; see fwd_shade): upstream gradient, the totals the forward saved, the
    // running sums. With W = sum w (the accumulated opacity), mu = M1 / W, c_k = m_k - mu, V = M2 - M1^2 / W = sum w c^2:
    // d dist / d m_k = 2 w_k W c_k, d dist / d w_k = W c_k^2 + V, and what lies behind hit k enters through the
    // transmittance: sum_{i>k} (d dist / d w_i) w_i = W (V - V_k) + V (W - W_k) with the running sums through k.
    if (DIST && in_seg && s.seg == 0 && p.a.dL_ddist && p.a.out_dist) {
        x.tot_acc = __ldg(p.a.mid_val + (size_t)ray * in.mid_stride + 7);
        if (x.tot_acc > 0.0f) {
            x.dist_on = true;
            x.t_dist = __ldg(p.a.dL_ddist + ray);
            x.dist_mu = __ldg(p.a.out_dist + 3 * (size_t)ray + 1) / x.tot_acc;
            x.dist_V = __ldg(p.a.out_dist + 3 * (size_t)ray + 2) - __ldg(p.a.out_dist + 3 * (size_t)ray + 1) * x.dist_mu;
        }
    }
    return x;
}
__device__ __forceinline__ RowTarget row_target(const BwdParams& p) {
    const dst_trace_inputs& in = p.a.in;
    RowTarget t;
    t.arena = p.arena; t.dsh = in.colors_precomp == nullptr ? p.a.dL_dshs : nullptr; t.coeffs = in.sh_coeffs;
    t.ncoef = (in.sh_degree + 1) * (in.sh_degree + 1);
    t.bulk = t.dsh && (in.sh_coeffs & 3) == 0 && (t.ncoef & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.a.dL_dshs) & 15) == 0);
    return t;
}

// Gradients of one contributing hit (backward.cu:529-632), staged in ws for send_rows(). e: the evaluated hit.
//
// The reference differentiates each composited quantity on its own. All of them are sums of w f over the hits, so the gradient of a hit's alpha
// needs only F = (upstream gradients) . (what the hit contributes) and the one running value s.rem = (upstream gradients) . (totals of the
// segment, background and opacity included) - sum of w F so far: dL/dalpha = T (F + t_acc) - rem / (1 - alpha). The vertex terms are
// written in two edges of the triangle: the gradients of the three corners add up to E n, and their
// moments with the corner signs (the gradients of the scaled tangents) to 6 E e x h -+ 3 E n. Both are the reference's
// sums in exact arithmetic with a fraction of the operations.
template <bool DIST>
__device__ __forceinline__ void bwd_hit(const BwdParams& p, BwdState& s, const BwdSegment& x, const SlotEval& e, int pidx, bool first, BwdWarp& ws) {
    const dst_trace_inputs& in = p.a.in;
    const int lane = threadIdx.x & 31, gidx = pidx >> 1;
    const float alpha = e.alpha, T_prev = s.T_prev, dpt = e.dpt;
    const float w = xmul(alpha, T_prev);
    float F = s.t_dpt * dpt + e.nsign * (s.t_nx * e.r2.x + s.t_ny * e.r2.y + s.t_nz * e.r2.z);
    float m0 = s.t_rgb0 * w, m1 = s.t_rgb1 * w, m2 = s.t_rgb2 * w;
    float4* row = reinterpret_cast<float4*>(ws.rows[lane]);
    bulk_wait_read();                                          // the engine has read what this lane's row held
    row[4] = make_float4(m0, m1, m2, 0.f);
    if (x.use_sh) {
        float c0 = 0.5f, c1 = 0.5f, c2 = 0.5f;
        const float* sh = in.shs + 3 * (size_t)gidx * in.sh_coeffs;
        if (x.sh_wide) {       // degree 3, the usual layout: six 256-bit loads
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float c[24];
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    float4 q, r;
                    ldg256(reinterpret_cast<const float4*>(sh) + 6 * i + 2 * l, q, r);
                    c[8 * l] = q.x; c[8 * l + 1] = q.y; c[8 * l + 2] = q.z; c[8 * l + 3] = q.w;
                    c[8 * l + 4] = r.x; c[8 * l + 5] = r.y; c[8 * l + 6] = r.z; c[8 * l + 7] = r.w;
                }
#pragma unroll
                for (int l = 0; l < 8; l++) {
                    const float b = ws.basis[8 * i + l][lane];
                    c0 = fmaf(b, c[3 * l], c0); c1 = fmaf(b, c[3 * l + 1], c1); c2 = fmaf(b, c[3 * l + 2], c2);
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (4 * q < x.ncoef) {
                    float c[12];
                    if (x.sh_aligned) {
#pragma unroll
                        for (int l = 0; l < 3; l++) {
                            const float4 v = __ldg(reinterpret_cast<const float4*>(sh) + 3 * q + l);
                            c[4 * l] = v.x; c[4 * l + 1] = v.y; c[4 * l + 2] = v.z; c[4 * l + 3] = v.w;
                        }
                    } else {
#pragma unroll
                        for (int l = 0; l < 12; l++) c[l] = 12 * q + l < 3 * x.ncoef ? __ldg(sh + 12 * q + l) : 0.0f;
                    }
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        if (4 * q + l < x.ncoef) {
                            const float b = ws.basis[4 * q + l][lane];
                            c0 = fmaf(b, c[3 * l], c0); c1 = fmaf(b, c[3 * l + 1], c1); c2 = fmaf(b, c[3 * l + 2], c2);
                        }
                    }
                }
            }
        }
        if (c0 < 0.f) { c0 = 0.f; m0 = 0.f; }                 // clamped channels take no gradient
        if (c1 < 0.f) { c1 = 0.f; m1 = 0.f; }
        if (c2 < 0.f) { c2 = 0.f; m2 = 0.f; }
        F += s.t_rgb0 * c0 + s.t_rgb1 * c1 + s.t_rgb2 * c2;
        ws.colour[lane] = make_float4(m0, m1, m2, 0.f);
        s.dir_gidx = gidx; s.dir_g0 = m0; s.dir_g1 = m1; s.dir_g2 = m2;
    } else {
        const float* cp = in.colors_precomp + 3 * (size_t)gidx;
        F += s.t_rgb0 * __ldg(cp) + s.t_rgb1 * __ldg(cp + 1) + s.t_rgb2 * __ldg(cp + 2);
    }
    if (x.has_aux) {
        const float2 ax = __ldg(reinterpret_cast<const float2*>(in.others_precomp) + gidx);
        F += s.t_aux0 * ax.x + s.t_aux1 * ax.y;
    }
    const float inv = __frcp_rn(1.0f - alpha);
    s.rem = fmaf(-w, F, s.rem);
    float dL_dalpha = T_prev * (F + s.t_acc) - s.rem * inv;
    float dist_dd = 0.f;       // gradient of the distortion with respect to this hit's depth
    if (DIST && x.dist_on) {
        const float m_abs = DST_DIST_K * (1.0f - DST_DIST_NEAR / dpt);
        if (first) s.dm0 = m_abs;
        const float cm = (m_abs - s.dm0) - x.dist_mu;
        s.dws += w; s.dvs += w * cm * cm;
        const float d_dw = x.tot_acc * cm * cm + x.dist_V;
        const float behind = x.tot_acc * (x.dist_V - s.dvs) + x.dist_V * (x.tot_acc - s.dws);
        dL_dalpha += x.t_dist * (d_dw * T_prev - behind * inv);
        dist_dd = x.t_dist * 2.0f * w * x.tot_acc * cm * DST_DIST_K * DST_DIST_NEAR / (dpt * dpt);
    }
    // geometry (backward.cu:201-287, 581-607)
    const float opac = e.r2.w;
    const float gG = (opac * e.G) > 0.99f ? 0.0f : dL_dalpha * e.G;         // no gradient through a clamped alpha
    const float kG = gG * opac;
    const float sx = e.r3.x, sy = e.r3.y, u = e.u, v = e.v;
    const float au = -kG * u * e.r3.z, av = -kG * v * e.r3.w;               // dL/du / sx, dL/dv / sy
    const V3 R0 = v3(e.r0.x, e.r0.y, e.r0.z), R1 = v3(e.r1.x, e.r1.y, e.r1.z);
    const V3 rd = v3(s.sdx, s.sdy, s.sdz);
    const V3 dxyz = au * R0 + av * R1;
    const float dL_dd = s.t_dpt * w + dist_dd + dot(dxyz, rd);
    const float4* vq = reinterpret_cast<const float4*>(in.vertices + 12 * (size_t)gidx);
    const float4 va = __ldg(vq), vb = __ldg(vq + 1), vc = __ldg(vq + 2);
    const bool t0 = (pidx & 1) == 0;
    // corners p1, p2, p3 of the triangle, its normal as the reference forms it (at a grazing angle the quotients by n . d magnify the rounding of n)
    const V3 v1 = v3(va.w, vb.x, vb.y), v2 = v3(vb.z, vb.w, vc.x);
    const V3 p1 = t0 ? v3(va.x, va.y, va.z) : v1, p2 = t0 ? v1 : v2, p3 = t0 ? v2 : v3(vc.y, vc.z, vc.w);
    const V3 f1 = p2 - p1, f2 = p3 - p1;
    const V3 nn = cross(f1, f2);
    const V3 cvec = p1 - v3(s.sox, s.soy, s.soz);
    const float iq = __frcp_rn(dot(nn, rd)), depth = dot(nn, cvec) * iq;
    const V3 h = cvec - depth * rd;
    const float E = dL_dd * iq;
    const V3 En = E * nn;
    const float E6 = 6.0f * E, E6s = t0 ? -E6 : E6, En3 = t0 ? 3.0f : -3.0f;
    const V3 ex = t0 ? f1 : p3 - p2;
    const V3 shx = E6s * cross(ex, h) - 3.0f * En, shy = E6s * cross(f2, h) + En3 * En;
    const V3 dmean = En - dxyz;
    s.dro_x -= dmean.x; s.dro_y -= dmean.y; s.dro_z -= dmean.z;
    if (!x.use_sh) {   // with SH the value is replaced below
        s.drd_x += dpt * dxyz.x - depth * En.x; s.drd_y += dpt * dxyz.y - depth * En.y; s.drd_z += dpt * dxyz.z - depth * En.z;
    }
    const float hd = 0.5f * dpt;
    row[1] = make_float4(dmean.x, dmean.y, dmean.z, gG);
    row[2] = make_float4(dmean.x * hd, dmean.y * hd, dmean.z * hd, 0.f);
    row[3] = make_float4(dot(R0, shx) - au * u, dot(R1, shy) - av * v, x.has_aux ? s.t_aux0 * w : 0.f, x.has_aux ? s.t_aux1 * w : 0.f);
    // quaternion (auxiliary.h:433-477; no gradient through the normalisation)
    const V3 rel = v3(e.X - __ldg(in.means3D + 3 * (size_t)gidx), e.Y - __ldg(in.means3D + 3 * (size_t)gidx + 1), e.Z - __ldg(in.means3D + 3 * (size_t)gidx + 2));
    const V3 dR0 = au * rel + sx * shx, dR1 = av * rel + sy * shy;
    const float wn = w * e.nsign;
    const V3 dR2 = v3(s.t_nx * wn, s.t_ny * wn, s.t_nz * wn);
    const float4 q = __ldg(reinterpret_cast<const float4*>(in.rotations) + gidx);
    const float qs = 2.0f * rsqrtf(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    const float qw = q.x * qs, qx = q.y * qs, qy = q.z * qs, qz = q.w * qs;          // twice the unit quaternion
    const float a = dR1.z - dR2.y, b = dR2.x - dR0.z, c = dR0.y - dR1.x;
    const float d = dR0.y + dR1.x, f = dR0.z + dR2.x, g = dR1.z + dR2.y;
    row[0] = make_float4(qx * a + qy * b + qz * c, qw * a + qy * d + qz * f - 2.f * qx * (dR1.y + dR2.z),
                         qw * b + qx * d + qz * g - 2.f * qy * (dR0.x + dR2.z), qw * c + qx * f + qy * g - 2.f * qz * (dR0.x + dR1.y));
    s.T_prev = xmul(T_prev, xsub(1.0f, alpha));
}

// After the last contribution of a segment: true if an earlier one is left to differentiate.
__device__ __forceinline__ bool bwd_end_segment(const BwdParams& p, int ray, BwdState& s, const BwdSegment& x) {
    const dst_trace_inputs& in = p.a.in;
    // With SH colours the reference ASSIGNS the SH direction gradient to the ray-direction
    // accumulator at every contribution (backward.cu:165, 631-632), so what survives a segment
    // is the value of its last contribution.
    if (x.use_sh && s.dir_gidx >= 0) {
        float csh[48], sj[16];
        load_sh_row(in.shs + 3 * (size_t)s.dir_gidx * in.sh_coeffs, 3 * x.ncoef, x.sh_aligned, csh);
#pragma unroll
        for (int j = 0; j < 16; j++) sj[j] = j < x.ncoef ? csh[3 * j] * s.dir_g0 + csh[3 * j + 1] * s.dir_g1 + csh[3 * j + 2] * s.dir_g2 : 0.f;
        const V3 g = sh_dir_grad(in.sh_degree, sj, s.sdx, s.sdy, s.sdz);
        s.drd_x = g.x; s.drd_y = g.y; s.drd_z = g.z;
    }
    return bwd_next_segment(p, ray, s, s.seg - 1);
}

// Re-composites one gathered chunk of segment s.seg (backward.cu:429-655) for the rays of a warp in step: all 32 lanes call it, `in_chunk`
// marks those with a chunk. key_at(i): the lane's i-th hit of cnt. Returns true for rays that need another enumeration.
template <bool DIAG, bool DIST, class KeyAt>
__device__ __forceinline__ bool bwd_chunk(const BwdParams& p, bool in_chunk, int ray, BwdState& s, KeyAt key_at, int cnt, BwdWarp& ws, TraceCounters& tc) {
    const BwdSegment x = bwd_segment<DIST>(p, in_chunk, ray, s, ws);
    const RowTarget target = row_target(p);
    const float min_depth = s.seg == 0 ? (p.a.in.start_from_first ? 0.2f : 0.0f) : 0.06f;
    if (DIAG && in_chunk && s.chunk == 0) tc.segs++;
    bool stop = !in_chunk;
    const int n = __reduce_max_sync(0xffffffffu, in_chunk ? cnt : 0);
    for (int sl = 0; sl < n; sl++) {
        int gsent = -1;
        if (!stop && sl < cnt) {
            const unsigned long long key = key_at(sl);
            const int pidx = (int)(unsigned int)key;
            const int gidx = pidx >> 1;
            SlotEval e;
            bool ok = false;
            if (gidx != s.last_gidx) {
                if (DIAG) tc.evals++;
                ok = eval_slot(key, s.offset, s.sox, s.soy, s.soz, s.sdx, s.sdy, s.sdz, min_depth, p.cache, gidx, e);
                s.dpt = e.dpt;
            }
            if (ok && (xmul(s.T_prev, xsub(1.0f, e.alpha)) < 0.0001f || ++s.contributor > DST_MAX_INTERSECTION)) { stop = true; ok = false; }
            if (ok) {
                s.last_gidx = gidx;
                if (DIAG) tc.contribs++;
                bwd_hit<DIST>(p, s, x, e, pidx, s.contributor == 1, ws);
                gsent = gidx;
            }
        }
        send_rows(target, ws, gsent, p.tiled != 0);       // linear ray lists: neighbours in the list are not neighbours on a surface
    }
    if (!in_chunk) return false;
    s.chunk++;
    bool seg_done = stop || cnt < DST_CHUNK || s.contributor > DST_MAX_INTERSECTION;
    if (!seg_done && s.chunk >= DST_MAX_CHUNKS) { atomicOr(p.status, DST_STATUS_CHUNK_LIMIT); seg_done = true; }
    if (!seg_done) {
        s.offset = (float)((double)s.dpt + 0.00001);
        return true;
    }
    return bwd_end_segment(p, ray, s, x);
}

__global__ void __launch_bounds__(256) k_bwd_init(const __grid_constant__ BwdParams p, long long slots) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= slots) return;
    if (i == 0) p.counts[0] = (int)slots;
    const int ray = slot_ray(i, p.grid_h, p.grid_w, p.tiled != 0);
    bool alive = false;
    if (ray >= 0) {
        BwdState s;
        alive = bwd_init_state(p, ray, s);
        if (alive) {
            bwd_store_state(p.state, (int)i, s);
            EnumReq q;
            bwd_request(s, q);
            store_req(p.req, (int)i, q);
        }       // else no segment to differentiate: the (zero) ray gradients are already written
    }
    p.list[0][i] = alive ? (int)i : -1;
}

__device__ __forceinline__ void bwd_flush_counters(unsigned long long* counters, const TraceCounters& tc) {
    if (!counters) return;
    if (tc.segs) atomicAdd(counters + 0, tc.segs);
    if (tc.enums) atomicAdd(counters + 1, tc.enums);
    if (tc.nodes) atomicAdd(counters + 2, tc.nodes);
    if (tc.quads) atomicAdd(counters + 3, tc.quads);
    if (tc.evals) atomicAdd(counters + 4, tc.evals);
    if (tc.contribs) atomicAdd(counters + 5, tc.contribs);
}

__device__ __forceinline__ BwdWarp& bwd_warp_mem() {
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    return reinterpret_cast<BwdWarp*>(dyn_smem)[threadIdx.x >> 5];
}

// one round of the re-trace: composites the gathered chunk of every ray on the list
template <bool DIAG, bool DIST>
__global__ void __launch_bounds__(BWD_THREADS, DST_BWD_BLOCKS) k_bwd_shade(const __grid_constant__ BwdParams p, int round) {
    const int n = p.counts[round];
    if (n < p.min_count) return;
    const int* list = p.list[round & 1];
    int* next_list = p.list[(round + 1) & 1];
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    BwdWarp& ws = bwd_warp_mem();
    const int n_pad = (n + 31) & ~31;
    for (int i = blockIdx.x * BWD_THREADS + threadIdx.x; i < n_pad; i += gridDim.x * BWD_THREADS) {
        const int slot = i < n ? list[i] : -1;
        const int ray = slot >= 0 ? slot_ray(slot, p.grid_h, p.grid_w, p.tiled != 0) : -1;
        BwdState s;
        int cnt = 0;
        if (slot >= 0) { bwd_load_state(p.state, slot, s); cnt = p.kcnt[slot]; }
        const bool wide = (cnt & DST_KCNT_WIDE) != 0;
        cnt &= DST_KCNT_WIDE - 1;
        const unsigned long long* kb = p.kbuf + soa(slot >= 0 ? slot : 0, 0, DST_CHUNK);
        const bool alive = bwd_chunk<DIAG, DIST>(p, slot >= 0, ray, s, [&](int k) { return kb[k * 32]; }, cnt, ws, tc);
        int cls = 0;
        if (alive) {
            bwd_store_state(p.state, slot, s);
            EnumReq q;
            bwd_request(s, q);
            if (wide) q.off = -q.off;
            store_req(p.req, slot, q);
            cls = s.seg > 0;
        }
        if (p.lv.stable) live_out(p.lv, round, i, alive, slot, cls);
        else append_alive(alive, slot, next_list, p.counts + round + 1);
    }
    bulk_drain();
    if (DIAG) bwd_flush_counters(p.a.counters, tc);
}

// Runs every ray of the first list the rounds left alone to completion: a warp takes as many rays as it takes to keep all warps busy (one, for the
// few rays the rounds leave), gathers the chunk of one after the other together (knearest_warp) and composites them in step.
template <bool DIAG, bool DIST>
__global__ void __launch_bounds__(BWD_THREADS, DST_BWD_BLOCKS) k_bwd_tail(const __grid_constant__ BwdParams p) {
    constexpr unsigned int FULL = 0xffffffffu;
    __shared__ WalkMem walk_mem[BWD_THREADS / 32];
    __shared__ unsigned long long skeys[BWD_THREADS / 32][32][DST_CHUNK];
    const int round = first_skipped_round(p.counts, p.rounds, p.min_count);
    const int n = p.counts[round];
    const int* list = p.list[round & 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int warps = gridDim.x * (BWD_THREADS / 32);
    const int share = (n + warps - 1) / warps, per = share < 1 ? 1 : share > 32 ? 32 : share;
    const float absmax = __ldg(p.bvh.header + 6);
    BwdWarp& ws = bwd_warp_mem();
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    for (long long i0 = (long long)(blockIdx.x * (BWD_THREADS / 32) + w) * per; i0 < n; i0 += (long long)warps * per) {
        const int slot = lane < per && i0 + lane < n ? list[i0 + lane] : -1;
        const int ray = slot >= 0 ? slot_ray(slot, p.grid_h, p.grid_w, p.tiled != 0) : -1;
        BwdState s;
        bool alive = slot >= 0;
        if (alive) bwd_load_state(p.state, slot, s);
        for (;;) {
            const unsigned int todo = __ballot_sync(FULL, alive);
            if (todo == 0u) break;
            EnumReq q = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
            if (alive) { EnumReq r; bwd_request(s, r); q = r; r.start(q.ox, q.oy, q.oz); if (DIAG) tc.enums++; }
            int cnt = 0;
            for (unsigned int m = todo; m; m &= m - 1u) {
                const int r = __ffs(m) - 1;
                unsigned long long key;
                const int c = knearest_warp<DIAG>(p.bvh, __shfl_sync(FULL, q.ox, r), __shfl_sync(FULL, q.oy, r), __shfl_sync(FULL, q.oz, r), __shfl_sync(FULL, q.dx, r),
                                                  __shfl_sync(FULL, q.dy, r), __shfl_sync(FULL, q.dz, r), DST_T_MAX, absmax, walk_mem[w], key, p.status, tc);
                if (lane < c) skeys[w][r][lane] = key;
                if (lane == r) cnt = c;
                __syncwarp();
            }
            const bool go = bwd_chunk<DIAG, DIST>(p, alive, ray, s, [&](int k) { return skeys[w][lane][k]; }, cnt, ws, tc);
            alive = alive && go;
            __syncwarp();
        }
    }
    bulk_drain();
    if (DIAG) bwd_flush_counters(p.a.counters, tc);
}

// Backward over the contribution log of the matching forward call: every ray composites its logged contributions again, so no
// hierarchy walk is needed; one thread per ray, all segments. Rays whose log is incomplete (log full during the forward) are
// initialised and queued for the re-trace.
//
// A warp composites its rays' contributions in step, entry by entry, and only the lanes whose ray is in the latest segment still
// open in the warp (the backward visits a ray's segments last to first): neighbouring pixels then composite the same surfels in
// the same pass, which is what send_rows() feeds on.
template <bool DIAG, bool DIST, int BLOCKS>
__global__ void __launch_bounds__(BWD_THREADS, BLOCKS) k_bwd_logged(const __grid_constant__ BwdParams p, long long slots, int per) {
    constexpr unsigned int FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long i = ((long long)blockIdx.x * (BWD_THREADS / 32) + (threadIdx.x >> 5)) * per + lane;
    const int slot = lane < per && i < slots ? (int)i : -1;
    const int ray = slot >= 0 ? slot_ray(slot, p.grid_h, p.grid_w, p.tiled != 0) : -1;
    TraceCounters tc = { 0, 0, 0, 0, 0, 0 };
    BwdWarp& ws = bwd_warp_mem();
    const RowTarget target = row_target(p);
    bool requeue = false;
    BwdState s;
    bool active = ray >= 0 && bwd_init_state(p, ray, s);
    if (active && !p.log_ok[slot]) {
        bwd_store_state(p.state, slot, s);
        EnumReq q;
        bwd_request(s, q);
        store_req(p.req, slot, q);
        requeue = true; active = false;
    }
    for (;;) {
        const int cur = __reduce_max_sync(FULL, active ? s.seg : -1);
        if (cur < 0) break;
        const bool in = active && s.seg == cur;
        int num = 0, rec = -1;
        if (in) {
            num = __ldg(p.log_num + cur * p.log_slots + slot);
            if (num > 0) rec = __ldg(p.log_head + cur * p.log_slots + slot);
            if (DIAG) { tc.segs++; tc.contribs += num; tc.evals += num; }
        }
        const BwdSegment x = bwd_segment<DIST>(p, in, ray, s, ws);
        const float min_depth = cur == 0 ? (p.a.in.start_from_first ? 0.2f : 0.0f) : 0.06f;
        unsigned long long key = num > 0 ? __ldg(p.log_keys + soa(rec, 0, DST_CHUNK)) : 0ull;
        const int n = __reduce_max_sync(FULL, num);
        for (int at = 0; at < n; at++) {
            int gsent = -1;
            if (at < num) {
                const int pidx = (int)(unsigned int)key;
                SlotEval e;
                // accepted, as in the forward, unless the caller has changed the surfel since: it then contributes nothing
                const bool ok = eval_slot(key, 0.0f, s.sox, s.soy, s.soz, s.sdx, s.sdy, s.sdz, min_depth, p.cache, pidx >> 1, e);
                if (at + 1 < num) {
                    if (((at + 1) & (DST_CHUNK - 1)) == 0) rec = __ldg(p.log_next + rec);
                    key = __ldg(p.log_keys + soa(rec, (at + 1) & (DST_CHUNK - 1), DST_CHUNK));
                }
                if (ok) {
                    bwd_hit<DIST>(p, s, x, e, pidx, at == 0, ws);
                    gsent = pidx >> 1;
                }
            }
            send_rows(target, ws, gsent, p.tiled != 0);
        }
        if (in) active = bwd_end_segment(p, ray, s, x);
    }
    bulk_drain();
    append_alive(requeue, slot, p.list[0], p.counts);
    if (DIAG) bwd_flush_counters(p.a.counters, tc);
}

// Arena rows -> the caller's gradient tensors. The rows that hold anything are zeroed on the way, so the arena is clean for the next call: a
// call with few rays leaves most of it untouched, and clearing all 80 bytes per surfel first was a fifth of what such a call writes.
__global__ void __launch_bounds__(256) k_unpack(int P, float* __restrict__ arena, float* __restrict__ d_rot, float* __restrict__ d_mean,
                                                float* __restrict__ d_opac, float* __restrict__ d_g3d, float* __restrict__ d_scale,
                                                float* __restrict__ d_others, float* __restrict__ d_color) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P) return;
    float4* r = reinterpret_cast<float4*>(arena + (size_t)g * DST_ARENA_FLOATS);
    const float4 a = r[0], b = r[1], c = r[2], d = r[3], e = r[4];
    auto used = [](const float4& v) { return v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f; };
    if (used(a) || used(b) || used(c) || used(d) || used(e)) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        r[0] = zero; r[1] = zero; r[2] = zero; r[3] = zero; r[4] = zero;
    }
    reinterpret_cast<float4*>(d_rot)[g] = a;
    d_mean[3 * (size_t)g] = b.x; d_mean[3 * (size_t)g + 1] = b.y; d_mean[3 * (size_t)g + 2] = b.z;
    d_opac[g] = b.w;
    d_g3d[3 * (size_t)g] = c.x; d_g3d[3 * (size_t)g + 1] = c.y; d_g3d[3 * (size_t)g + 2] = c.z;
    d_scale[2 * (size_t)g] = d.x; d_scale[2 * (size_t)g + 1] = d.y;
    d_others[2 * (size_t)g] = d.z; d_others[2 * (size_t)g + 1] = d.w;
    d_color[3 * (size_t)g] = e.x; d_color[3 * (size_t)g + 1] = e.y; d_color[3 * (size_t)g + 2] = e.z;
}

}  // namespace

BvhView dst_bvh_view(const dst_handle* h);
int dst_check_inputs(dst_handle* h, const dst_trace_inputs* in);
long long dst_call_signature(const dst_trace_inputs* in);
long long dst_slot_grid(const dst_handle* h, const dst_trace_inputs* in, int* gh, int* gw, int* tiled);

// the staging rows need more dynamic shared memory than a kernel gets by default: raise the limit of every instantiation once per device
template <typename K>
static cudaError_t allow_stage_smem(K kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BWD_STAGE_BYTES); }
static int backward_kernel_setup(dst_handle* h) {
    static bool done[64] = { false };
    if (h->device >= 0 && h->device < 64 && done[h->device]) return DST_OK;
    cudaError_t e = cudaSuccess;
#define DST_SETUP(...) if (e == cudaSuccess) e = allow_stage_smem(__VA_ARGS__);
    DST_SETUP(k_bwd_shade<false, false>) DST_SETUP(k_bwd_shade<false, true>) DST_SETUP(k_bwd_shade<true, false>) DST_SETUP(k_bwd_shade<true, true>)
    DST_SETUP(k_bwd_tail<false, false>) DST_SETUP(k_bwd_tail<false, true>) DST_SETUP(k_bwd_tail<true, false>) DST_SETUP(k_bwd_tail<true, true>)
    DST_SETUP(k_bwd_logged<false, false, 4>) DST_SETUP(k_bwd_logged<false, true, 4>) DST_SETUP(k_bwd_logged<true, false, 4>) DST_SETUP(k_bwd_logged<true, true, 4>)
    DST_SETUP(k_bwd_logged<false, false, 5>) DST_SETUP(k_bwd_logged<false, true, 5>) DST_SETUP(k_bwd_logged<true, false, 5>) DST_SETUP(k_bwd_logged<true, true, 5>)
#undef DST_SETUP
    if (e != cudaSuccess) { cudaGetLastError(); return dst_set_error(h, DST_E_CUDA, "raising the shared-memory limit of the backward kernels failed: %s", cudaGetErrorString(e)); }
    if (h->device >= 0 && h->device < 64) done[h->device] = true;
    return DST_OK;
}

template <int BLOCKS>
static void launch_logged(bool diag, bool dist, unsigned int blocks, cudaStream_t st, const BwdParams& p, long long slots, int per) {
    if (dist) { if (diag) k_bwd_logged<true, true, BLOCKS><<<blocks, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, slots, per); else k_bwd_logged<false, true, BLOCKS><<<blocks, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, slots, per); }
    else { if (diag) k_bwd_logged<true, false, BLOCKS><<<blocks, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, slots, per); else k_bwd_logged<false, false, BLOCKS><<<blocks, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, slots, per); }
}

int dst_backward_impl(dst_handle* h, const dst_bwd_args* a, cudaStream_t st) {
    int rc = dst_check_inputs(h, &a->in);
    if (rc != DST_OK) return rc;
    rc = backward_kernel_setup(h);
    if (rc != DST_OK) return rc;
    if (!a->out_rgb || !a->mid_val) return dst_set_error(h, DST_E_ARG, "a saved forward output pointer is null");
    if (!h->absent_gradients && (!a->dL_drgb || !a->dL_ddpt || !a->dL_dacc || !a->dL_dnorm || !a->dL_daux))
        return dst_set_error(h, DST_E_ARG, "an upstream gradient pointer is null");
    if (!a->dL_dray_o || !a->dL_dray_d || !a->dL_dmeans3D || !a->dL_dgrads3D || !a->dL_dcolors || !a->dL_dothers ||
        !a->dL_dopacities || !a->dL_dscales || !a->dL_drotations || (a->in.shs && !a->dL_dshs))
        return dst_set_error(h, DST_E_ARG, "a gradient output pointer is null");
    if ((reinterpret_cast<uintptr_t>(a->mid_val) & 15) || (reinterpret_cast<uintptr_t>(a->in.vertices) & 15) ||
        (reinterpret_cast<uintptr_t>(a->in.rotations) & 15) || (reinterpret_cast<uintptr_t>(a->dL_drotations) & 15) ||
        (a->in.others_precomp && (reinterpret_cast<uintptr_t>(a->in.others_precomp) & 7)))
        return dst_set_error(h, DST_E_ARG, "mid_val, vertices, rotations and dL_drotations must be 16-byte aligned");
    const int64_t P = a->in.P;
    if (P > h->arena_cap) {
        dst_mem_free(h, h->arena); h->arena = nullptr; h->arena_cap = 0;
        const int64_t cap = P + P / 8 + 1024;
        if (dst_mem_alloc(h, (void**)&h->arena, 4 * DST_ARENA_FLOATS * cap) != cudaSuccess) { cudaGetLastError(); return dst_set_error(h, DST_E_NOMEM, "gradient arena allocation failed"); }
        h->arena_cap = cap; h->arena_clean = false;
    }
    if (!h->arena_clean) DST_CUDA_TRY(h, cudaMemsetAsync(h->arena, 0, 4 * DST_ARENA_FLOATS * (size_t)h->arena_cap, st));
    h->arena_clean = false;      // until k_unpack has been enqueued
    // the records of the forward this belongs to, when they are still there
    const bool same = a->forward_serial != 0 && a->forward_serial == h->cache_serial && h->cache_src[0] == a->in.means3D && h->cache_src[1] == a->in.scales &&
                      h->cache_src[2] == a->in.rotations && h->cache_src[3] == a->in.opacities && h->cache_P == P;
    if (!same) { rc = dst_prepare_cache(h, &a->in, st); if (rc != DST_OK) return rc; }
    if (a->dL_dshs) DST_CUDA_TRY(h, cudaMemsetAsync(a->dL_dshs, 0, 12 * (size_t)P * a->in.sh_coeffs, st));
    BwdParams p;
    p.a = *a; p.bvh = dst_bvh_view(h); p.cache = h->cache; p.arena = h->arena; p.status = h->status;
    p.dist_on = h->distortion;
    dst_handle::Log* log = nullptr;
    if (a->forward_serial != 0) {
        for (int k = 0; k < h->logs_used; k++) {
            dst_handle::Log& l = h->logs[k];
            if (l.serial == a->forward_serial && l.H == a->in.H && l.W == a->in.W && l.depth == a->in.max_trace_depth) log = &l;
        }
        // a log that was overwritten before its backward came: room for the forwards since then next time
        const unsigned long long since = h->serial_counter - a->forward_serial + 1;
        if (!log && h->logs_keep > 1 && since > 1) { h->logs_wanted = since < (unsigned long long)h->logs_keep ? (int)since : h->logs_keep; h->logs_missed = true; }
    }
    long long slots = dst_slot_grid(h, &a->in, &p.grid_h, &p.grid_w, &p.tiled);
    if (log) { p.grid_h = log->grid_h; p.grid_w = log->grid_w; p.tiled = log->tiled; slots = log->slots; log->consumed = true; }       // the log is indexed by its forward's slots
    rc = dst_ensure_wavefront(h, slots, sizeof(BwdState));
    if (rc != DST_OK) return rc;
    p.state = static_cast<float4*>(h->wf_state); p.req = static_cast<float4*>(h->wf_req); p.kbuf = h->wf_kbuf; p.kcnt = h->wf_kcnt;
    p.list[0] = h->wf_list[0]; p.list[1] = h->wf_list[1]; p.counts = h->wf_counts;
    const bool diag = a->counters != nullptr;
    const bool dist = h->distortion != 0 && a->dL_ddist != nullptr && a->out_dist != nullptr;
    const bool use_log = log != nullptr;
    p.log_keys = h->log_keys; p.log_next = h->log_next; p.log_head = log ? log->head : nullptr; p.log_num = log ? log->num : nullptr; p.log_ok = log ? log->ok : nullptr;
    p.log_slots = slots;
    DST_CUDA_TRY(h, cudaMemsetAsync(h->wf_counts, 0, 4 * DST_COUNTS_STRIDE, st));
    h->slices_used = 1;
    const bool wave = slots >= h->wf_min_rays;
    rc = dst_live_lists(h, &p.lv, st);
    if (rc != DST_OK) return rc;
    const int g_compact = (int)((slots + DST_LIVE_BLOCK - 1) / DST_LIVE_BLOCK);
    p.rounds = wave ? DST_WF_ROUNDS : 0;
    p.min_count = wave ? (int)(slots / 512 > 2048 ? slots / 512 : 2048) : 1;
    // With the log the rounds only serve rays it could not hold. When the last completed read-back of a forward of this shape
    // shows that everything fitted, none are enqueued (scheduling only: whatever is left after them is finished by the tail
    // kernel). A dozen rounds of empty launches took 0.15 ms.
    if (wave && use_log && h->log_known_needed > 0 && h->log_known_sig == dst_call_signature(&a->in) && h->log_use <= h->log_cap)
        p.rounds = 0;
    dst_prof_mark(h, 2, 0, st);
    if (use_log) {
        // the forward logged its contributions: composite them again; rays the log could not hold are queued as round 0 of the
        // re-trace below (normally none: the rounds then find an empty list and return at once)
        // Rays per warp: 32, or 16 or 8 (4x4 and 4x2 patches of a tile) where 32 would leave warp slots of the GPU empty. What a small call takes
        // is the chain of one warp's hits, and adding the rows of 8 rays up is shorter than those of 32.
        int per = 32;
        while (per > 8 && slots / per * 2 <= (long long)h->sm_count * DST_BWD_BLOCKS * (BWD_THREADS / 32)) per >>= 1;
        const long long per_block = per * (BWD_THREADS / 32);
        const unsigned int blocks = (unsigned int)((slots + per_block - 1) / per_block);
        // 20 warps an SM at 96 registers where there is twice the work to fill them (a tenth faster there), 16 at 128 registers otherwise
        if (slots / 32 >= 2ll * h->sm_count * 5 * (BWD_THREADS / 32)) launch_logged<5>(diag, dist, blocks, st, p, slots, per);
        else launch_logged<4>(diag, dist, blocks, st, p, slots, per);
    } else {
        k_bwd_init<<<(unsigned int)((slots + 255) / 256), 256, 0, st>>>(p, slots);
    }
    const int g_enum = dst_wavefront_grid(h, slots, ENUM_THREADS, 10), g_shade = dst_wavefront_grid(h, slots, BWD_THREADS, 4);
    for (int r = 0; r < p.rounds; r++) {
        dst_prof_mark(h, 3, 0, st);
        launch_gather(diag, g_enum, h->sm_count, 1, st, p.bvh, p.req, p.list[r & 1], p.counts + r, p.counts + r, p.min_count, p.kbuf, p.kcnt,
                      p.status, a->counters, p.lv.tmp, p.list[(r + 1) & 1]);
        dst_prof_mark(h, 3, 1, st);
        if (dist) { if (diag) k_bwd_shade<true, true><<<g_shade, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, r); else k_bwd_shade<false, true><<<g_shade, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, r); }
        else { if (diag) k_bwd_shade<true, false><<<g_shade, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, r); else k_bwd_shade<false, false><<<g_shade, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p, r); }
        if (p.lv.stable) k_compact<<<g_compact, 256, 0, st>>>(p.lv, p.counts + r, p.counts + r + 1, p.min_count, p.list[(r + 1) & 1], r);
    }
    const int g_tail = dst_wavefront_grid(h, (wave ? p.min_count : slots) * 32, BWD_THREADS, DST_BWD_BLOCKS);
    if (dist) { if (diag) k_bwd_tail<true, true><<<g_tail, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p); else k_bwd_tail<false, true><<<g_tail, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p); }
    else { if (diag) k_bwd_tail<true, false><<<g_tail, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p); else k_bwd_tail<false, false><<<g_tail, BWD_THREADS, BWD_STAGE_BYTES, st>>>(p); }
    dst_prof_mark(h, 2, 1, st);
    DST_CUDA_TRY(h, cudaGetLastError());
    k_unpack<<<(unsigned int)((P + 255) / 256), 256, 0, st>>>((int)P, h->arena, a->dL_drotations, a->dL_dmeans3D, a->dL_dopacities,
                                                              a->dL_dgrads3D, a->dL_dscales, a->dL_dothers, a->dL_dcolors);
    DST_CUDA_TRY(h, cudaGetLastError());
    h->arena_clean = true;
    h->launches += 3 + (p.lv.stable ? 5 : 4) * p.rounds;       // logged re-composite or ray init, the rounds, tail, unpack
    return DST_OK;
}
