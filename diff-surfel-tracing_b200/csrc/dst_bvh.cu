// Hierarchy build / refit over surfel quads: replaces optixAccelBuild as called from
// trace_surfels.cpp:36-159 (OPERATION_BUILD when rebuild > 0, OPERATION_UPDATE otherwise).
//
// Build:  centroid bounds -> 63-bit Morton keys -> LSD radix sort (8 x 8-bit passes, 64-bit key /
//         32-bit value) -> Karras hierarchy -> bottom-up box pass (also writes the per-quad plane
//         frames in leaf order).
// Refit:  the bottom-up pass alone, on the topology and leaf order of the last build.
// All kernels are plain HBM-bound streaming / scatter kernels; nothing waits on another block
// (the bottom-up pass uses arrival counters: the first thread to reach a node leaves, the second
// continues), so there is no device-side spin anywhere.
#include "dst_common.cuh"
#include <math.h>

namespace {

constexpr int REFIT_THREADS = 256;                      // leaves per block of the bottom-up pass
constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;   // 4096 keys per block
constexpr int SORT_WARPS = SORT_THREADS / 32;

__device__ __forceinline__ unsigned int f2ord(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// words 0..2: min of quad-box centres, 3..5: max (ordered-uint encoding)
__global__ void k_init_bounds(unsigned int* bw) {
    if (threadIdx.x < 3) bw[threadIdx.x] = 0xffffffffu;
    else if (threadIdx.x < 6) bw[threadIdx.x] = 0u;
}

__device__ __forceinline__ void quad_box(const float* __restrict__ v, float* lo, float* hi) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
        lo[a] = fminf(fminf(v[a], v[3 + a]), fminf(v[6 + a], v[9 + a]));
        hi[a] = fmaxf(fmaxf(v[a], v[3 + a]), fmaxf(v[6 + a], v[9 + a]));
    }
}

__global__ void __launch_bounds__(256) k_centre_bounds(const float* __restrict__ verts, int P, unsigned int* bw) {
    float lo[3] = { INFINITY, INFINITY, INFINITY }, hi[3] = { -INFINITY, -INFINITY, -INFINITY };
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < P; g += gridDim.x * blockDim.x) {
        float v[12];
        const float4* p = reinterpret_cast<const float4*>(verts + 12 * (size_t)g);
        float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        v[8] = c.x; v[9] = c.y; v[10] = c.z; v[11] = c.w;
        float l[3], h[3];
        quad_box(v, l, h);
#pragma unroll
        for (int a2 = 0; a2 < 3; a2++) {
            float cc = 0.5f * (l[a2] + h[a2]);
            if (isfinite(cc)) { lo[a2] = fminf(lo[a2], cc); hi[a2] = fmaxf(hi[a2], cc); }
        }
    }
    // one atomic per block and bound (as one per warp, 57,000 of them on six addresses, they took longer than the reads)
    __shared__ float red[8][6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; a++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
        if (lane == 0) { red[w][a] = lo[a]; red[w][3 + a] = hi[a]; }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int a = threadIdx.x;
        float l = red[0][a], h = red[0][3 + a];
        for (int k = 1; k < 8; k++) { l = fminf(l, red[k][a]); h = fmaxf(h, red[k][3 + a]); }
        if (l <= h) { atomicMin(&bw[a], f2ord(l)); atomicMax(&bw[3 + a], f2ord(h)); }
    }
}

__device__ __forceinline__ unsigned long long spread21(unsigned long long x) {
    x &= 0x1fffffull;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__global__ void __launch_bounds__(256) k_morton(const float* __restrict__ verts, int P, const unsigned int* __restrict__ bw,
                                                unsigned long long* __restrict__ keys, unsigned int* __restrict__ vals) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P) return;
    float v[12];
    const float4* p = reinterpret_cast<const float4*>(verts + 12 * (size_t)g);
    float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    v[8] = c.x; v[9] = c.y; v[10] = c.z; v[11] = c.w;
    float l[3], h[3];
    quad_box(v, l, h);
    unsigned long long key = 0;
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        const float lo = ord2f(bw[ax]), hi = ord2f(bw[3 + ax]);
        const float ext = hi - lo;
        float cc = 0.5f * (l[ax] + h[ax]);
        float q = (ext > 0.0f && isfinite(cc)) ? (cc - lo) / ext * 2097152.0f : 0.0f;
        q = fminf(fmaxf(q, 0.0f), 2097151.0f);
        key |= spread21((unsigned long long)(unsigned int)q) << (2 - ax);
    }
    keys[g] = key;
    vals[g] = (unsigned int)g;
}

// ---- LSD radix sort, one 8-bit digit per pass --------------------------------------------------
__global__ void __launch_bounds__(SORT_THREADS) k_sort_hist(const unsigned long long* __restrict__ keys, int n, int shift,
                                                            unsigned int* __restrict__ block_hist, int nblocks) {
    __shared__ unsigned int sh[256];
    sh[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * SORT_TILE;
#pragma unroll
    for (int i = 0; i < SORT_ITEMS; i++) {
        const int idx = base + i * SORT_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&sh[(unsigned int)(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
    block_hist[threadIdx.x * nblocks + blockIdx.x] = sh[threadIdx.x];
}

// Exclusive scan of the per-block counts of ONE digit (block d of the grid takes digit d): block_hist[d][0..nblocks)
// becomes the number of keys with digit d in the blocks before, and digit_total[d] their number in all blocks. The
// scatter kernel adds the keys with smaller digits itself (a 256-entry scan every block repeats), so no block of any
// kernel waits for another and no single block walks all 256 x nblocks counters.
__global__ void __launch_bounds__(256) k_sort_scan(unsigned int* __restrict__ block_hist, int nblocks, unsigned int* __restrict__ digit_total) {
    __shared__ unsigned int warp_sum[8];
    __shared__ unsigned int carry_s;
    unsigned int* data = block_hist + (size_t)blockIdx.x * nblocks;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = 0; base < nblocks; base += 256) {
        const int idx = base + threadIdx.x;
        unsigned int x = idx < nblocks ? data[idx] : 0u, incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { unsigned int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
        if (lane == 31) warp_sum[wid] = incl;
        __syncthreads();
        unsigned int before = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) if (k < wid) before += warp_sum[k];
        const unsigned int carry = carry_s;
        if (idx < nblocks) data[idx] = carry + before + incl - x;
        __syncthreads();
        if (threadIdx.x == 255) carry_s = carry + before + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) digit_total[blockIdx.x] = carry_s;
}

// Stable scatter: warp w of a block owns 512 consecutive keys and ranks them 32 at a time. The block's keys are put in digit order in
// shared memory first, so that what a digit gets from this block (16 keys on average) is written as one run: written straight from the
// registers every key was a memory sector of its own (3M keys, mean of the eight passes: 63 -> 42 us under ncu).
struct SortTile { unsigned long long key[SORT_TILE]; unsigned int val[SORT_TILE]; unsigned short wc[SORT_WARPS][256]; unsigned int start[256], base[256], sum[SORT_WARPS]; };
__device__ __forceinline__ unsigned int scan256(unsigned int x, unsigned int* warp_sum) {       // exclusive, over the 256 threads of the block
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { unsigned int y = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += y; }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    unsigned int before = 0;
#pragma unroll
    for (int k = 0; k < SORT_WARPS; k++) if (k < w) before += warp_sum[k];
    __syncthreads();
    return before + incl - x;
}
__global__ void __launch_bounds__(SORT_THREADS) k_sort_scatter(const unsigned long long* __restrict__ keys_in,
                                                               const unsigned int* __restrict__ vals_in,
                                                               unsigned long long* __restrict__ keys_out,
                                                               unsigned int* __restrict__ vals_out, int n, int shift,
                                                               const unsigned int* __restrict__ block_offs, int nblocks,
                                                               const unsigned int* __restrict__ digit_total) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    SortTile& t = *reinterpret_cast<SortTile*>(sort_smem);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // where this block's keys of digit d go: after the keys with a smaller digit, and those of the same digit in the blocks before
    t.base[threadIdx.x] = scan256(digit_total[threadIdx.x], t.sum) + block_offs[threadIdx.x * nblocks + blockIdx.x];
    for (int i = threadIdx.x; i < SORT_WARPS * 256; i += SORT_THREADS) (&t.wc[0][0])[i] = 0;
    __syncthreads();
    const int tile = blockIdx.x * SORT_TILE, base = tile + w * (SORT_ITEMS * 32);
    unsigned long long key[SORT_ITEMS];
    unsigned int val[SORT_ITEMS];
    unsigned short rank[SORT_ITEMS];
#pragma unroll
    for (int s = 0; s < SORT_ITEMS; s++) {
        const int idx = base + s * 32 + lane;
        const bool valid = idx < n;
        key[s] = valid ? keys_in[idx] : ~0ull;
        val[s] = valid ? vals_in[idx] : 0u;
    }
#pragma unroll
    for (int s = 0; s < SORT_ITEMS; s++) {
        const bool valid = base + s * 32 + lane < n;
        const unsigned int d = valid ? ((unsigned int)(key[s] >> shift) & 255u) : 256u;
        const unsigned int mask = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(mask) - 1;
        unsigned int old = 0;
        if (lane == leader && valid) { old = t.wc[w][d]; t.wc[w][d] = (unsigned short)(old + __popc(mask)); }
        old = __shfl_sync(0xffffffffu, old, leader);
        rank[s] = (unsigned short)(old + __popc(mask & ((1u << lane) - 1u)));
        __syncwarp();
    }
    __syncthreads();
    {
        const int d = threadIdx.x;     // SORT_THREADS == 256 digits
        unsigned int count = 0;
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ww++) count += t.wc[ww][d];
        unsigned int sum = scan256(count, t.sum);
        t.start[d] = sum;
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ww++) { const unsigned int c = t.wc[ww][d]; t.wc[ww][d] = (unsigned short)sum; sum += c; }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < SORT_ITEMS; s++) {
        if (base + s * 32 + lane < n) {
            const unsigned int pos = t.wc[w][(unsigned int)(key[s] >> shift) & 255u] + rank[s];
            t.key[pos] = key[s]; t.val[pos] = val[s];
        }
    }
    __syncthreads();
    const int count = n - tile < SORT_TILE ? n - tile : SORT_TILE;
    for (int i = threadIdx.x; i < count; i += SORT_THREADS) {
        const unsigned long long k = t.key[i];
        const unsigned int d = (unsigned int)(k >> shift) & 255u, pos = t.base[d] + (unsigned int)i - t.start[d];
        keys_out[pos] = k;
        vals_out[pos] = t.val[i];
    }
}

// ---- Karras 2012 hierarchy over the sorted keys -----------------------------------------------
__device__ __forceinline__ int key_delta(const unsigned long long* __restrict__ keys, int n, int i, unsigned long long ki, int j) {
    if (j < 0 || j >= n) return -1;
    const unsigned long long x = ki ^ keys[j];
    return x ? __clzll((long long)x) : 64 + __clz(i ^ j);
}

__global__ void __launch_bounds__(256) k_karras(const unsigned long long* __restrict__ keys, int n, BvhNode* __restrict__ nodes,
                                                int* __restrict__ leaf_parent, int* __restrict__ node_parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const unsigned long long ki = keys[i];
    const int d = (key_delta(keys, n, i, ki, i + 1) - key_delta(keys, n, i, ki, i - 1)) >= 0 ? 1 : -1;
    const int dmin = key_delta(keys, n, i, ki, i - d);
    int lmax = 2;
    while (key_delta(keys, n, i, ki, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (key_delta(keys, n, i, ki, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = key_delta(keys, n, i, ki, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (key_delta(keys, n, i, ki, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    int c0, c1;
    if (lo == gamma) { c0 = ~gamma; leaf_parent[gamma] = i; } else { c0 = gamma; node_parent[gamma] = i; }
    if (hi == gamma + 1) { c1 = ~(gamma + 1); leaf_parent[gamma + 1] = i; } else { c1 = gamma + 1; node_parent[gamma + 1] = i; }
    nodes[i].child[0].c = c0; nodes[i].child[1].c = c1;
    nodes[i].child[0].pad = (lo ^ hi) < REFIT_THREADS && lo / REFIT_THREADS == hi / REFIT_THREADS;      // all its leaves in one block of the bottom-up pass
    if (i == 0) node_parent[0] = -1;
}

// single-surfel scene: one node whose second child is an empty box
__global__ void k_single_leaf(BvhNode* nodes, int* leaf_parent, int* node_parent, unsigned int* arrive) {
    nodes[0].child[0].c = ~0; nodes[0].child[1].c = ~0; nodes[0].child[0].pad = 0; node_parent[0] = -1;
    nodes[0].child[1].lox = nodes[0].child[1].loy = nodes[0].child[1].loz = INFINITY;
    nodes[0].child[1].hix = nodes[0].child[1].hiy = nodes[0].child[1].hiz = -INFINITY;
    leaf_parent[0] = 0;
    arrive[0] = 1;      // the lone leaf acts as the second arrival
}

// ---- bottom-up pass: quad frames + leaf boxes, then boxes of all ancestors ----------------------
// The 4 corners of surfel g from its parameters, in the reference's expression order
// (example/utils/gaussian_utils.py:176-210 with build_cov :286-296, build_scaling_rotation :273-282,
// build_rotation :214-249): q = r / |r| in (w,x,y,z) order, tangent columns of R scaled by s_x and
// s_y, corner k = (3 cu_k) L0 + (3 cv_k) L1 + mean, (cu,cv) = (-1,+1), (-1,-1), (+1,+1), (+1,-1).
// One rounding per operation; bit-identical to the reference's CPU tensor ops on the test vectors.
struct SurfelSource { const float* means; const float* scales; const float* rotations; float* v_out; };

__device__ __forceinline__ void surfel_corners(const SurfelSource& src, int g, float* v) {
    const float4 r = __ldg(reinterpret_cast<const float4*>(src.rotations) + g);
    const float2 sc = __ldg(reinterpret_cast<const float2*>(src.scales) + g);
    const float m[3] = { __ldg(src.means + 3 * (size_t)g), __ldg(src.means + 3 * (size_t)g + 1), __ldg(src.means + 3 * (size_t)g + 2) };
    const float n = xsqrt(xadd(xadd(xadd(xmul(r.x, r.x), xmul(r.y, r.y)), xmul(r.z, r.z)), xmul(r.w, r.w)));
    const float w = xdiv(r.x, n), x = xdiv(r.y, n), y = xdiv(r.z, n), z = xdiv(r.w, n);
    float c0[3], c1[3];
    c0[0] = xsub(1.0f, xmul(2.0f, xadd(xmul(y, y), xmul(z, z))));
    c0[1] = xmul(2.0f, xadd(xmul(x, y), xmul(w, z)));
    c0[2] = xmul(2.0f, xsub(xmul(x, z), xmul(w, y)));
    c1[0] = xmul(2.0f, xsub(xmul(x, y), xmul(w, z)));
    c1[1] = xsub(1.0f, xmul(2.0f, xadd(xmul(x, x), xmul(z, z))));
    c1[2] = xmul(2.0f, xadd(xmul(y, z), xmul(w, x)));
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float lu = xmul(c0[a], sc.x), lv = xmul(c1[a], sc.y);
        const float u3 = xmul(lu, 3.0f), v3 = xmul(lv, 3.0f);
        v[0 + a] = xadd(xadd(-u3, v3), m[a]);
        v[3 + a] = xadd(xadd(-u3, -v3), m[a]);
        v[6 + a] = xadd(xadd(u3, v3), m[a]);
        v[9 + a] = xadd(xadd(u3, -v3), m[a]);
    }
}

// get_triangles as one kernel: 36 B of parameters in, 48 B of vertices (+ 24 B of indices) out per surfel
__global__ void __launch_bounds__(256) k_surfel_quads(SurfelSource src, int P, int32_t* __restrict__ tri) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P) return;
    float v[12];
    surfel_corners(src, g, v);
    float4* o = reinterpret_cast<float4*>(src.v_out + 12 * (size_t)g);
    o[0] = make_float4(v[0], v[1], v[2], v[3]); o[1] = make_float4(v[4], v[5], v[6], v[7]); o[2] = make_float4(v[8], v[9], v[10], v[11]);
    if (tri) {
        const int b = 4 * g;
        int2* t = reinterpret_cast<int2*>(tri + 6 * (size_t)g);
        t[0] = make_int2(b, b + 1); t[1] = make_int2(b + 2, b + 1); t[2] = make_int2(b + 2, b + 3);
    }
}

// Bottom-up pass over the hierarchy: leaf level from the quads, then the boxes of every ancestor. FROM_SURFELS: the quad corners are computed from the surfel parameters here and
// written to the caller's vertex buffer on the way (the refit then never reads the vertices).
//
// Nodes whose leaves all lie in one block (all but one in a hundred) are merged through shared memory; only the rest exchange boxes and
// arrivals through the L2, where a level costs a fence and an atomic, about a microsecond (3M surfels, under ncu: 495 -> 319 us).
template <bool FROM_SURFELS>
__global__ void __launch_bounds__(REFIT_THREADS) k_refit(const float* __restrict__ verts, SurfelSource src, int P, const unsigned int* __restrict__ vals,
                                               BvhNode* nodes, const int* __restrict__ leaf_parent, const int* __restrict__ node_parent,
                                               unsigned int* arrive,
                                               float4* __restrict__ quads, float* header) {
    __shared__ float sbox[REFIT_THREADS][2][6];
    __shared__ unsigned int sarrive[REFIT_THREADS];
    sarrive[threadIdx.x] = 0;
    __syncthreads();
    const int pos = blockIdx.x * REFIT_THREADS + threadIdx.x;
    if (pos >= P) return;
    const int gid = (int)vals[pos];
    float v[12];
    if (FROM_SURFELS) {
        surfel_corners(src, gid, v);
        float4* o = reinterpret_cast<float4*>(src.v_out + 12 * (size_t)gid);
        o[0] = make_float4(v[0], v[1], v[2], v[3]); o[1] = make_float4(v[4], v[5], v[6], v[7]); o[2] = make_float4(v[8], v[9], v[10], v[11]);
    } else {
        const float4* p = reinterpret_cast<const float4*>(verts + 12 * (size_t)gid);
        float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        v[8] = c.x; v[9] = c.y; v[10] = c.z; v[11] = c.w;
    }
    const QuadFrame q = make_quad_frame(v);
    quads[4 * (size_t)pos + 0] = make_float4(q.p0x, q.p0y, q.p0z, q.nx);
    quads[4 * (size_t)pos + 1] = make_float4(q.ny, q.nz, q.wux, q.wuy);
    quads[4 * (size_t)pos + 2] = make_float4(q.wuz, q.wvx, q.wvy, q.wvz);
    quads[4 * (size_t)pos + 3] = make_float4(__int_as_float(gid), 0.0f, 0.0f, 0.0f);
    float lo[3], hi[3];
    quad_box(v, lo, hi);
    int child = ~pos;                           // link of the subtree being carried up
    int parent = leaf_parent[pos];
    // the depth of a Karras tree over 64-bit keys with index tie-breaks is below 128
    for (int guard = 0; guard < 128; guard++) {
        BvhNode* nd = nodes + parent;
        const int slot = (nd->child[0].c == child) ? 0 : 1;
        const int local = nd->child[0].pad;
        float4* dst = reinterpret_cast<float4*>(nd->child + slot);
        dst[0] = make_float4(lo[0], lo[1], hi[0], hi[1]); dst[1] = make_float4(lo[2], hi[2], __int_as_float(child), __int_as_float(slot == 0 ? local : 0));
        float slo[3], shi[3];
        if (local) {
            const int k = parent - blockIdx.x * REFIT_THREADS;       // (a node's index is one end of its range of leaves)
#pragma unroll
            for (int a = 0; a < 3; a++) { sbox[k][slot][a] = lo[a]; sbox[k][slot][3 + a] = hi[a]; }
            __threadfence_block();
            if (atomicAdd(&sarrive[k], 1u) == 0u) return;              // the sibling subtree is not done yet
            __threadfence_block();
            const volatile float* sib = sbox[k][1 - slot];
#pragma unroll
            for (int a = 0; a < 3; a++) { slo[a] = sib[a]; shi[a] = sib[3 + a]; }
        } else {
            __threadfence();
            if (atomicAdd(&arrive[parent], 1u) == 0u) return;
            const float4* src = reinterpret_cast<const float4*>(nd->child + (1 - slot));
            const float4 s0 = __ldcg(src), s1 = __ldcg(src + 1);
            slo[0] = s0.x; slo[1] = s0.y; slo[2] = s1.x; shi[0] = s0.z; shi[1] = s0.w; shi[2] = s1.y;
        }
#pragma unroll
        for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], slo[a]); hi[a] = fmaxf(hi[a], shi[a]); }
        if (parent == 0) {
            float am = 0.0f;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                header[a] = lo[a]; header[3 + a] = hi[a];
                if (isfinite(lo[a])) am = fmaxf(am, fabsf(lo[a]));
                if (isfinite(hi[a])) am = fmaxf(am, fabsf(hi[a]));
            }
            header[6] = am;
            return;
        }
        child = parent;
        parent = node_parent[parent];
    }
}

// Four children per node for the warps' walk: the grandchildren, one thread each.
__global__ void __launch_bounds__(256) k_widen(int n, const BvhNode* __restrict__ nodes, BvhChild* __restrict__ wide) {
    const int i = (int)(((long long)blockIdx.x * 256 + threadIdx.x) >> 2), s = threadIdx.x & 3;
    if (i >= n) return;
    const float4* src = reinterpret_cast<const float4*>(nodes[i].child + (s >> 1));
    float4 a = __ldg(src), b = __ldg(src + 1);
    const int c = __float_as_int(b.z);
    if (c >= 0) {
        const float4* g = reinterpret_cast<const float4*>(nodes[c].child + (s & 1));
        a = __ldg(g); b = __ldg(g + 1);
    } else if (s & 1) {       // no second grandchild: an empty box
        a = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY); b = make_float4(INFINITY, -INFINITY, __int_as_float(~0), 0.0f);
    }
    float4* dst = reinterpret_cast<float4*>(wide + 4 * (size_t)i + s);
    dst[0] = a; dst[1] = b;
}

// plane frames back in surfel order, for tests
__global__ void __launch_bounds__(256) k_export_frames(int P, const float4* __restrict__ quads, float* __restrict__ out) {
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= P) return;
    const float4 a = quads[4 * (size_t)pos], b = quads[4 * (size_t)pos + 1], c = quads[4 * (size_t)pos + 2];
    float* o = out + 12 * (size_t)__float_as_int(quads[4 * (size_t)pos + 3].x);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
    o[8] = c.x; o[9] = c.y; o[10] = c.z; o[11] = c.w;
}

int ensure_capacity(dst_handle* h, int64_t P) {
    if (P <= h->cap) return DST_OK;
    // grow-only arena; the old buffers are released first (a rebuild does not need them)
    h->cap = 0; h->built = false;
    const int64_t cap = P + P / 8 + 1024;
    const int64_t nblocks = (cap + SORT_TILE - 1) / SORT_TILE;
    const DstPart parts[] = {
        {(void**)&h->nodes, sizeof(BvhNode) * cap}, {(void**)&h->wide, 4 * sizeof(BvhChild) * cap}, {(void**)&h->quads, 64 * (size_t)cap},
        {(void**)&h->leaf_parent, 4 * (size_t)cap}, {(void**)&h->arrive, 4 * (size_t)cap}, {(void**)&h->node_parent, 4 * (size_t)cap},
        {(void**)&h->keys, 8 * (size_t)cap}, {(void**)&h->keys_alt, 8 * (size_t)cap}, {(void**)&h->vals, 4 * (size_t)cap}, {(void**)&h->vals_alt, 4 * (size_t)cap},
        {(void**)&h->block_hist, 4 * 256 * (size_t)(nblocks + 1)}};       // + the 256 digit totals
    size_t total = 0;
    for (const DstPart& part : parts) total += part.bytes;
    if (total <= DST_SLAB_BUILD) dst_open_slab(h);
    const cudaError_t e = dst_alloc_parts(h, &h->build_block, parts, sizeof(parts) / sizeof(parts[0]));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return dst_set_error(h, DST_E_NOMEM, "device allocation for %lld surfels failed: %s", (long long)P, cudaGetErrorString(e));
    }
    h->cap = cap; h->hist_cap = nblocks;
    return DST_OK;
}

}  // namespace

int dst_surfel_quads_impl(dst_handle* h, const float* means, const float* scales, const float* rotations, int64_t P,
                          float* vertices, int32_t* triangles, cudaStream_t st) {
    if (P <= 0 || P > DST_MAX_SURFELS) return dst_set_error(h, DST_E_ARG, "surfel count must be in [1, 2^26], got %lld", (long long)P);
    if ((reinterpret_cast<uintptr_t>(vertices) & 15) || (reinterpret_cast<uintptr_t>(rotations) & 15) || (reinterpret_cast<uintptr_t>(scales) & 7) ||
        (reinterpret_cast<uintptr_t>(triangles) & 7))
        return dst_set_error(h, DST_E_ARG, "vertices and rotations must be 16-byte aligned, scales and triangles 8-byte aligned");
    const SurfelSource src = { means, scales, rotations, vertices };
    k_surfel_quads<<<(unsigned int)((P + 255) / 256), 256, 0, st>>>(src, (int)P, triangles);
    DST_CUDA_TRY(h, cudaGetLastError());
    h->launches += 1;
    return DST_OK;
}

// v: the vertex buffer. With means/scales/rotations non-null it is an OUTPUT: the quads are expanded
// from the surfel parameters (rebuild: by k_surfel_quads before the sort; refit: inside k_refit).
int dst_bvh_build_impl(dst_handle* h, const float* v, int64_t P, int rebuild, cudaStream_t st,
                       const float* means, const float* scales, const float* rotations) {
    const bool from_surfels = means != nullptr;
    const SurfelSource src = { means, scales, rotations, const_cast<float*>(v) };
    if (from_surfels && ((reinterpret_cast<uintptr_t>(rotations) & 15) || (reinterpret_cast<uintptr_t>(scales) & 7)))
        return dst_set_error(h, DST_E_ARG, "rotations must be 16-byte aligned and scales 8-byte aligned");
    if (P <= 0) return dst_set_error(h, DST_E_ARG, "vertices must hold at least one surfel (4 vertices)");
    if (P > DST_MAX_SURFELS) return dst_set_error(h, DST_E_ARG, "at most 2^26 surfels are supported");
    if ((reinterpret_cast<uintptr_t>(v) & 15) != 0) return dst_set_error(h, DST_E_ARG, "vertices must be 16-byte aligned");
    if (!rebuild) {
        if (!h->built) return dst_set_error(h, DST_E_STATE, "refit (rebuild=0) requested before any build");
        if (P != h->P) return dst_set_error(h, DST_E_ARG, "refit needs the surfel count of the last build (%lld), got %lld",
                                            (long long)h->P, (long long)P);
    }
    const int n = (int)P;
    constexpr int tpb = REFIT_THREADS; const int grid = (n + tpb - 1) / tpb;
    unsigned int* bw = reinterpret_cast<unsigned int*>(h->header + DST_HDR_FLOATS);
    if (rebuild) {
        int rc = ensure_capacity(h, P);
        if (rc != DST_OK) return rc;
    }
    dst_prof_mark(h, 0, 0, st);
    if (rebuild) {
        DST_CUDA_TRY(h, cudaFuncSetAttribute(k_sort_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortTile)));
        h->built = false;
        if (from_surfels) k_surfel_quads<<<grid, tpb, 0, st>>>(src, n, nullptr);
        k_init_bounds<<<1, 32, 0, st>>>(bw);
        const int rgrid = min(grid, h->sm_count * 8);
        k_centre_bounds<<<rgrid, tpb, 0, st>>>(v, n, bw);
        k_morton<<<grid, tpb, 0, st>>>(v, n, bw, h->keys, h->vals);
        const int nblocks = (n + SORT_TILE - 1) / SORT_TILE;
        unsigned long long *kin = h->keys, *kout = h->keys_alt;
        unsigned int *vin = h->vals, *vout = h->vals_alt;
        for (int pass = 0; pass < 8; pass++) {
            const int shift = 8 * pass;
            k_sort_hist<<<nblocks, SORT_THREADS, 0, st>>>(kin, n, shift, h->block_hist, nblocks);
            k_sort_scan<<<256, 256, 0, st>>>(h->block_hist, nblocks, h->block_hist + 256 * (size_t)nblocks);
            k_sort_scatter<<<nblocks, SORT_THREADS, sizeof(SortTile), st>>>(kin, vin, kout, vout, n, shift, h->block_hist, nblocks, h->block_hist + 256 * (size_t)nblocks);
            unsigned long long* tk = kin; kin = kout; kout = tk;
            unsigned int* tv = vin; vin = vout; vout = tv;
        }
        // 8 passes: the sorted data is back in keys / vals
        if (n > 1) k_karras<<<(n - 1 + tpb - 1) / tpb, tpb, 0, st>>>(h->keys, n, h->nodes, h->leaf_parent, h->node_parent);
        h->P = P;
    } else if (from_surfels && !h->single_kernel_refit) {
        // measured at 3M surfels: the coalesced expansion pass (0.07 ms) plus the refit's gathered re-read of the
        // vertices is faster than one kernel that scatters 48-byte vertex writes in Morton order (0.47 vs 0.59 ms)
        k_surfel_quads<<<grid, tpb, 0, st>>>(src, n, nullptr);
    }
    DST_CUDA_TRY(h, cudaMemsetAsync(h->arrive, 0, 4 * (size_t)(n > 1 ? n - 1 : 1), st));
    if (n == 1) k_single_leaf<<<1, 1, 0, st>>>(h->nodes, h->leaf_parent, h->node_parent, h->arrive);
    if (from_surfels && !rebuild && h->single_kernel_refit)
        k_refit<true><<<grid, tpb, 0, st>>>(v, src, n, h->vals, h->nodes, h->leaf_parent, h->node_parent, h->arrive, h->quads, h->header);
    else
        k_refit<false><<<grid, tpb, 0, st>>>(v, src, n, h->vals, h->nodes, h->leaf_parent, h->node_parent, h->arrive, h->quads, h->header);
    const int inner = n > 1 ? n - 1 : 1;
    k_widen<<<(unsigned int)((4ll * inner + 255) / 256), 256, 0, st>>>(inner, h->nodes, h->wide);
    dst_prof_mark(h, 0, 1, st);
    DST_CUDA_TRY(h, cudaGetLastError());
    h->launches += 1 + (rebuild ? 27 + (n > 1 ? 1 : 0) : 0) + (from_surfels && (rebuild || !h->single_kernel_refit) ? 1 : 0) + (n == 1 ? 1 : 0) + 1;
    h->built = true;
    return DST_OK;
}

int dst_export_frames_impl(dst_handle* h, float* out, cudaStream_t st) {
    if (!h->built) return dst_set_error(h, DST_E_STATE, "no hierarchy has been built");
    k_export_frames<<<(unsigned int)((h->P + 255) / 256), 256, 0, st>>>((int)h->P, h->quads, out);
    DST_CUDA_TRY(h, cudaGetLastError());
    return DST_OK;
}
