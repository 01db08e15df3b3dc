// Triangle-triangle discrete collision detection (DCD) for sm_100a.
//
// Broadphase: 24-bit Hilbert-curve codes of the triangles' padded boxes, a
// stable LSD radix sort (8-bit digits, per-warp ranking with
// __match_any_sync), the boxes in that order together with those of every 32
// and every 1024 consecutive leaves, and a block traversal: a warp takes 32
// consecutive triangles and walks down from the 1024-leaf blocks that their
// boxes touch to 32-leaf blocks, and each triangle meets the 32 leaves of a
// block at once.  Two passes (count, scan, fill) list the pairs in a
// deterministic order, by query and partner position.
//
// A binary tree (Karras' construction, a query per thread) needed a build
// launch of 32 us and left 11 of 32 lanes active on chains of dependent node
// loads: 70 us for the counting pass of 105k triangles.  The block traversal
// takes 46 us (692k box pairs in 294k (triangle, block) tests of about 50
// instructions; two queries at a time, half the queries a warp or up to twice
// the resident warps all took 46 to 51 us).
//
// Narrowphase / response / apply restate the reference's UDCF kernels
// (collision/udcf/kernel.py:164-474, 713-822): Moller interval rejection,
// VF/FV/EE candidate depths C1/C2, smaller-positive wins (tie -> C2), equal
// push of the three vertices of each movable face, friction on the
// bary-weighted tangential displacement, Jacobi averaging.
#include <cuda_runtime.h>

#include <algorithm>

#include "xpbd_common.cuh"
#include "xpbd_device.cuh"
#include "xpbd_grid.cuh"

using namespace xpbd;

namespace {

constexpr int kSortThreads = 1024;  // keys per scatter round; the sort's CTA size
constexpr int kScanItems = 4;       // consecutive elements per thread and round of the scan
constexpr int kSlots = 16;  // partners a query keeps from the counting pass
constexpr int kNarrowCtas = 592;  // 4 x 148 SMs
constexpr float kThresh = 1.0e-5f;  // udcf/kernel.py:40 THRESH

__device__ __forceinline__ float4 ld4(const float* p, int i) { return reinterpret_cast<const float4*>(p)[i]; }

// ws_nodes: three float4 arrays of the leaves in curve order: box lo (w: the
// triangle id), box hi (w: its group), vertex ids.  ws_bbox: boxes (lo, hi) of
// the 32-leaf blocks, then of the 1024-leaf blocks.  ws_keys2 (free after the
// sort): pairs per 32-query block, then their offsets.
struct Leaves {
    float4 *lo, *hi;
    int4* verts;
    float4 *b32, *b1k;
    __device__ __forceinline__ explicit Leaves(const XpbdDcd& D)
        : lo(reinterpret_cast<float4*>(D.ws_nodes)),
          hi(lo + D.n_tris),
          verts(reinterpret_cast<int4*>(hi + D.n_tris)),
          b32(reinterpret_cast<float4*>(D.ws_bbox)),
          b1k(b32 + 2 * ((D.n_tris + 31) / 32)) {}
};

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// ---------------------------------------------------------------- boxes
// tri_aabb_kernel (udcf/kernel.py:917-934)
__device__ __forceinline__ void tri_box(const XpbdDcd& D, const float* pos4, int a, int b, int c, float3& lo, float3& hi) {
    const float3 pa = f3(ld4(pos4, a)), pb = f3(ld4(pos4, b)), pc = f3(ld4(pos4, c));
    const float t = D.thickness;
    lo = make_float3(fminf(fminf(pa.x, pb.x), pc.x) - t, fminf(fminf(pa.y, pb.y), pc.y) - t,
                     fminf(fminf(pa.z, pb.z), pc.z) - t);
    hi = make_float3(fmaxf(fmaxf(pa.x, pb.x), pc.x) + t, fmaxf(fmaxf(pa.y, pb.y), pc.y) + t,
                     fmaxf(fmaxf(pa.z, pb.z), pc.z) + t);
}

// Position along the Hilbert curve through the 256^3 grid (J. Skilling,
// "Programming the Hilbert curve", 2004: undo the excess rotations from the top
// bit down, then Gray-decode).  Against Morton order, consecutive cells always
// touch, so no 32 neighbours straddle the scene: of the 3,288 leaf blocks of a
// 105k-triangle body the common box of 32 queries touches 126 at most instead
// of 531, 8.5 on average instead of 11.4, for about 90 more integer operations
// a key.
__device__ __forceinline__ uint32_t hilbert24(uint32_t x, uint32_t y, uint32_t z) {
#pragma unroll
    for (uint32_t q = 128u; q > 1u; q >>= 1) {
        const uint32_t p = q - 1u;
        if (x & q) x ^= p;
        uint32_t t = (x ^ y) & p;
        if (y & q) x ^= p;
        else { x ^= t; y ^= t; }
        t = (x ^ z) & p;
        if (z & q) x ^= p;
        else { x ^= t; z ^= t; }
    }
    y ^= x;
    z ^= y;
    uint32_t t = 0;
#pragma unroll
    for (uint32_t q = 128u; q > 1u; q >>= 1)
        if (z & q) t ^= q - 1u;
    return spread10(x ^ t) << 2 | spread10(y ^ t) << 1 | spread10(z ^ t);
}

// Curve key of triangle i: 8 bits per axis, cells of 3.5 mm on the 0.9-m body,
// about half a triangle (the order only decides how tight the leaf blocks are).
__device__ __forceinline__ uint32_t tri_key(const XpbdDcd& D, const float* __restrict__ pos4, int i) {
    float3 lo, hi;
    tri_box(D, pos4, D.tris[3 * i], D.tris[3 * i + 1], D.tris[3 * i + 2], lo, hi);
    const float q[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t u[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float ext = fmaxf(D.box_hi[k] - D.box_lo[k], 1e-30f);
        u[k] = uint32_t(fminf(fmaxf((q[k] - D.box_lo[k]) / ext * 255.f, 0.f), 255.f));
    }
    return hilbert24(u[0], u[1], u[2]);
}

// The snapshot of the positions by itself, for a broadphase that does not sort.
__global__ void k_snapshot(XpbdDcd D, const float* __restrict__ pos4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < D.n_verts) reinterpret_cast<float4*>(D.x_prev)[i] = ld4(pos4, i);
}

__device__ __forceinline__ uint32_t saturate(unsigned long long v) { return uint32_t(min(v, 0x7fffffffull)); }

// ---------------------------------------------------------- radix sort
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* warp_sums, T* block_total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        T t = lane < int(blockDim.x >> 5) ? warp_sums[lane] : T(0);
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_sums[lane] = t;
    }
    __syncthreads();
    const T incl = x + (w > 0 ? warp_sums[w - 1] : T(0));
    if (block_total && threadIdx.x == blockDim.x - 1) *block_total = incl;
    return incl - v;
}

// One CTA: the pair counts of the query blocks become offsets (a 32nd of the
// triangles: 3,287 values at 105k), their sum the pair count.  n triangles can
// have n (n - 1) / 2 pairs, beyond 32 bits from 65,537 triangles in one place on:
// the sums are 64 bits wide, and what is stored stops at INT32_MAX, which no
// list is longer than.
__global__ void __launch_bounds__(1024) k_scan_pairs(XpbdDcd D) {
    __shared__ unsigned long long warp_sums[32], carry, round_total;
    uint32_t* a = D.ws_keys2;
    const int nb = (D.n_tris + 31) / 32;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < nb; b0 += 1024 * kScanItems) {
        const int base = b0 + int(threadIdx.x) * kScanItems;
        uint32_t v[kScanItems];
        unsigned long long run = 0;
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            v[q] = base + q < nb ? a[base + q] : 0;
            run += v[q];
        }
        unsigned long long off = block_excl_scan(run, warp_sums, &round_total) + carry;
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            if (base + q < nb) a[base + q] = saturate(off);
            off += v[q];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += round_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *D.ws_total = int(saturate(carry));
        *D.n_pairs = int(saturate(carry));
        if (carry > uint32_t(D.max_pairs)) atomicOr(D.status, XPBD_STATUS_PAIR_OVERFLOW);
        *D.n_contacts = 0;
    }
}

// Radix sort of (curve key, triangle id), 3 passes of 8 bits, in one
// cooperative launch: CTA b owns the contiguous chunk [b C, (b+1) C) of the
// pass input.  Per pass: (A) chunk histogram -> hist[b][256]; grid barrier;
// (B) every CTA sums the histograms itself (digit totals, and the counts of
// the chunks before its own) and scans the totals over digits, giving its
// first output slot per digit; (C) stable scatter in rounds of kSortThreads
// keys: warps rank equal digits with __match_any_sync, per-digit prefix over
// the warps in shared memory; grid barrier before the next pass reads.
// The first pass forms the keys as it counts them, in ws_keys2/ws_vals2 (as a
// launch of its own that took 4.8 us for 105k triangles), with the snapshot of the
// positions when asked for; after three passes the sorted data is in
// ws_keys/ws_vals.
__device__ __forceinline__ int add_excl_over_warps(int (*wcnt)[256], int d, int run) {
    for (int ww = 0; ww < kSortThreads / 32; ++ww) {
        const int c = wcnt[ww][d];
        wcnt[ww][d] = run;
        run += c;
    }
    return run;
}

__global__ void __launch_bounds__(kSortThreads) k_sort_coop(XpbdDcd D, const float* __restrict__ pos4,
                                                             int snapshot, int chunk, uint32_t* sync) {
    __shared__ int wcnt[kSortThreads / 32][256];
    __shared__ int run[256];
    __shared__ int part[kSortThreads / 256][256];
    __shared__ int warp_sums[32];
    const int n = D.n_tris, G = gridDim.x, b = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int beg = min(n, b * chunk), end = min(n, beg + chunk);
    int* hist = D.ws_hist;  // [G][256]
    uint32_t* ks = D.ws_keys2;
    int32_t* vs = D.ws_vals2;
    uint32_t* kd = D.ws_keys;
    int32_t* vd = D.ws_vals;
    GridBarrier bar = grid_barrier_begin(sync);
    if (snapshot)
        for (int i = b * kSortThreads + int(threadIdx.x); i < D.n_verts; i += G * kSortThreads)
            reinterpret_cast<float4*>(D.x_prev)[i] = ld4(pos4, i);
    for (int pass = 0; pass < 3; ++pass) {
        const int shift = 8 * pass;
        // (A) chunk histogram
        if (threadIdx.x < 256) run[threadIdx.x] = 0;
        __syncthreads();
        for (int i = beg + int(threadIdx.x); i < end; i += kSortThreads) {
            if (pass == 0) {  // the chunk's keys; (C) reads them in the same CTA
                ks[i] = tri_key(D, pos4, i);
                vs[i] = i;
            }
            const int dig = int((ks[i] >> shift) & 255u);
            const unsigned peers = __match_any_sync(__activemask(), dig);
            if ((peers & ((1u << lane) - 1u)) == 0) atomicAdd(&run[dig], __popc(peers));
        }
        __syncthreads();
        if (threadIdx.x < 256) hist[b * 256 + threadIdx.x] = run[threadIdx.x];
        grid_barrier(bar, D.status);
        // (B) first output slot of each digit for this chunk
        {
            const int d = threadIdx.x & 255, q = threadIdx.x >> 8;
            constexpr int kQ = kSortThreads / 256;
            int tot = 0, pre = 0;
            // the CTAs' counts are independent L2 reads: unrolled so that several
            // are in flight at once instead of one latency per CTA
#pragma unroll 8
            for (int bb = q; bb < G; bb += kQ) {
                const int h = __ldcg(&hist[bb * 256 + d]);
                tot += h;
                pre += bb < b ? h : 0;
            }
            part[q][d] = tot;
            wcnt[q][d] = pre;
            __syncthreads();
            int t_all = 0, p_all = 0;
            if (q == 0) {
                for (int k = 0; k < kQ; ++k) {
                    t_all += part[k][d];
                    p_all += wcnt[k][d];
                }
            }
            const int base = block_excl_scan<int>(q == 0 ? t_all : 0, warp_sums, nullptr);
            if (q == 0) run[d] = base + p_all;
            __syncthreads();
        }
        // (C) stable scatter
        for (int r = beg; r < end; r += kSortThreads) {
            for (int k = threadIdx.x; k < (kSortThreads / 32) * 256; k += kSortThreads) (&wcnt[0][0])[k] = 0;
            __syncthreads();
            const int i = r + int(threadIdx.x);
            const bool valid = i < end;
            const uint32_t key = valid ? ks[i] : 0u;
            const int dig = valid ? int((key >> shift) & 255u) : 256;
            const unsigned peers = __match_any_sync(0xffffffffu, dig);
            const int lrank = __popc(peers & ((1u << lane) - 1u));
            if (valid && lrank == 0) wcnt[w][dig] = __popc(peers);
            __syncthreads();
            if (threadIdx.x < 256) run[threadIdx.x] = add_excl_over_warps(wcnt, threadIdx.x, run[threadIdx.x]);
            __syncthreads();
            const int dst = valid ? wcnt[w][dig] + lrank : -1;
            if (dst >= 0 && dst < n) {  // always, unless a barrier gave up (status bit set)
                kd[dst] = key;
                vd[dst] = vs[i];
            }
            __syncthreads();
        }
        if (pass < 2) grid_barrier(bar, D.status);
        uint32_t* tk = ks; ks = kd; kd = tk;
        int32_t* tv = vs; vs = vd; vd = tv;
    }
    grid_barrier_end(sync, bar);
}

// ---------------------------------------------------------- leaves and blocks
__device__ __forceinline__ void warp_box(float4& lo, float4& hi) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
        hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    }
}

// Leaf records in curve order from the current positions, and the boxes of the
// CTA's 32- and 1024-leaf blocks.  All that a refit-only broadphase runs before
// the traversal (the order of the last rebuild stays; the pair set does not
// depend on it).
__global__ void __launch_bounds__(1024) k_leaves(XpbdDcd D, const float* __restrict__ pos4) {
    __shared__ float4 s_box[32][2];
    const int n = D.n_tris;
    const int s = blockIdx.x * 1024 + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const Leaves L(D);
    float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    if (s < n) {
        const int tri = D.ws_vals[s];
        if (tri >= 0 && tri < n) {  // always, unless the sort gave up
            const int a = D.tris[3 * tri], b = D.tris[3 * tri + 1], c = D.tris[3 * tri + 2];
            float3 l, h;
            tri_box(D, pos4, a, b, c, l, h);
            lo = make_float4(l.x, l.y, l.z, __int_as_float(tri));
            hi = make_float4(h.x, h.y, h.z, __int_as_float(D.tri_group ? D.tri_group[tri] : 0));
            L.verts[s] = make_int4(a, b, c, 0);
        }
        L.lo[s] = lo;
        L.hi[s] = hi;
    }
    warp_box(lo, hi);
    if (lane == 0 && s < n) {
        L.b32[2 * (s >> 5)] = lo;
        L.b32[2 * (s >> 5) + 1] = hi;
    }
    if (lane == 0) {
        s_box[w][0] = lo;
        s_box[w][1] = hi;
    }
    __syncthreads();
    if (w == 0) {
        lo = s_box[lane][0];
        hi = s_box[lane][1];
        warp_box(lo, hi);
        if (lane == 0) {
            L.b1k[2 * blockIdx.x] = lo;
            L.b1k[2 * blockIdx.x + 1] = hi;
        }
    }
}

// ------------------------------------------------------------ traversal
// False for a NaN box (a triangle with an axis on which no corner is a number):
// it pairs with nothing, where the negated test made it a neighbour of all.
__device__ __forceinline__ bool overlap(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    return alo.x <= bhi.x && blo.x <= ahi.x && alo.y <= bhi.y && blo.y <= ahi.y && alo.z <= bhi.z && blo.z <= ahi.z;
}

__device__ __forceinline__ float4 shfl4(float4 v, int src) {
    return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                       __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

struct __align__(16) Query {
    float4 lo, hi;
    int4 verts;
};

// A warp lists the pairs of the 32 triangles at curve positions 32 qb + lane
// with the triangles at later positions (every unordered pair is met once).
// Blocks are found with the common box, 32 per test, and kept only for the
// lanes whose own box touches them: 32 neighbours on the curve can lie on
// different bodies, with a common box much larger than theirs, yet each of them
// touches a dozen 32-leaf blocks at most.  In a block that is kept, each of
// those lanes' boxes in turn meets all 32 leaves, one per lane, so the work is
// the number of (triangle, block) contacts, 3.5 per triangle of a body, however
// large the common box is (a loop over the leaves that touch the common box took
// 1620 us for 105k triangles, in a few warps).
// emit(src, hits, hit, j): for query lane src, in ascending partner position,
// the lanes of the ballot `hits` pair it with their triangle j; `on`: the lanes
// that take part as queries.  Pair rules of broadphase_find_pairs_bvh_kernel
// (udcf/kernel.py:937-981): static-static never, movable-self only when allowed
// and sharing no vertex.  s_q: the warp's queries, read back as broadcasts.
template <class Emit>
__device__ __forceinline__ void walk_blocks(const XpbdDcd& D, int qb, bool on, Query* s_q, Emit emit) {
    const Leaves L(D);
    const int n = D.n_tris, nb = (n + 31) / 32, nk = (n + 1023) / 1024;
    const int lane = threadIdx.x & 31, t = 32 * qb + lane;
    const float4 ulo = L.b32[2 * qb], uhi = L.b32[2 * qb + 1];
    float4 qlo = make_float4(0.f, 0.f, 0.f, 0.f), qhi = qlo;
    on = on && t < n;
    if (on) {
        s_q[lane].lo = qlo = L.lo[t];
        s_q[lane].hi = qhi = L.hi[t];
        s_q[lane].verts = L.verts[t];
    }
    __syncwarp();
    for (int k0 = qb >> 5; k0 < nk; k0 += 32) {
        const int k = min(k0 + lane, nk - 1);
        const float4 klo = L.b1k[2 * k], khi = L.b1k[2 * k + 1];
        unsigned mk = __ballot_sync(0xffffffffu, k0 + lane < nk && overlap(ulo, uhi, klo, khi));
        for (; mk; mk &= mk - 1) {
            const int ks = __ffs(mk) - 1, c0 = 32 * (k0 + ks), c = min(c0 + lane, nb - 1);
            const float4 kl = shfl4(klo, ks), kh = shfl4(khi, ks);
            if (!__any_sync(0xffffffffu, on && overlap(qlo, qhi, kl, kh))) continue;
            const float4 clo = L.b32[2 * c], chi = L.b32[2 * c + 1];
            unsigned mc = __ballot_sync(0xffffffffu, c0 + lane >= qb && c0 + lane < nb && overlap(ulo, uhi, clo, chi));
            for (; mc; mc &= mc - 1) {
                const int cs = __ffs(mc) - 1;
                const float4 cl = shfl4(clo, cs), ch = shfl4(chi, cs);
                unsigned mq = __ballot_sync(0xffffffffu, on && overlap(qlo, qhi, cl, ch));
                if (!mq) continue;
                const int p = 32 * (c0 + cs) + lane, pc = min(p, n - 1);
                const float4 lo = L.lo[pc], hi = L.hi[pc];
                const int4 v = L.verts[pc];
                for (; mq; mq &= mq - 1) {
                    const int src = __ffs(mq) - 1;
                    const float4 alo = s_q[src].lo, ahi = s_q[src].hi;
                    bool hit = p < n && p > 32 * qb + src && overlap(alo, ahi, lo, hi);
                    if (!__any_sync(0xffffffffu, hit)) continue;
                    const int g = __float_as_int(hi.w), ag = __float_as_int(ahi.w);
                    const int4 q = s_q[src].verts;
                    if (g == 1 && ag == 1) hit = false;
                    if (g == 0 && ag == 0)
                        hit = hit && D.allow_self &&
                              !(v.x == q.x || v.x == q.y || v.x == q.z || v.y == q.x || v.y == q.y || v.y == q.z ||
                                v.z == q.x || v.z == q.y || v.z == q.z);
                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                    if (hits) emit(src, hits, hit, __float_as_int(lo.w));
                }
            }
        }
    }
}

// Counting pass: pairs per query (ws_count) and per block of 32 (ws_keys2); a
// query's first kSlots partners are kept for the fill pass.
__global__ void __launch_bounds__(128) k_count_pairs(XpbdDcd D) {
    __shared__ Query s_q[4][32];
    const int qb = int(blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int n = D.n_tris, t = 32 * qb + lane;
    if (32 * qb >= n) return;
    int cnt = 0;
    if (!(*D.status & XPBD_STATUS_BARRIER_TIMEOUT))  // else the sort gave up: no valid order, no pairs
        walk_blocks(D, qb, true, s_q[threadIdx.x >> 5], [&](int src, unsigned hits, bool hit, int j) {
            const int slot = __shfl_sync(0xffffffffu, cnt, src) + __popc(hits & ((1u << lane) - 1u));
            if (hit && slot < kSlots) D.ws_slots[int64_t(slot) * n + 32 * qb + src] = j;
            if (lane == src) cnt += __popc(hits);
        });
    if (t < n) D.ws_count[t] = cnt;
    unsigned long long total = unsigned(cnt);
    for (int o = 16; o >= 1; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) D.ws_keys2[qb] = uint32_t(min(total, 0xffffffffull));
}

// Fill pass: pairs as (min, max) triangle id, grouped by query position; only
// queries with more than kSlots partners walk again.
__global__ void __launch_bounds__(128) k_fill_pairs(XpbdDcd D) {
    __shared__ Query s_q[4][32];
    const int qb = int(blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int n = D.n_tris, t = 32 * qb + lane;
    if (32 * qb >= n) return;
    // unsigned, and stopped at INT32_MAX before each sum: no index wraps into the list
    const uint32_t base = D.ws_keys2[qb], cap = uint32_t(D.max_pairs);
    const uint32_t c = t < n && base < cap ? uint32_t(D.ws_count[t]) : 0u;
    if (!__any_sync(0xffffffffu, c != 0u)) return;
    uint32_t out = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, out, o);
        if (lane >= o) out = min(out + y, 0x7fffffffu);
    }
    out = __shfl_up_sync(0xffffffffu, out, 1);
    out = lane == 0 ? base : min(out + base, 0x7fffffffu);
    const int i = c ? D.ws_vals[t] : 0;
    int2* pairs = reinterpret_cast<int2*>(D.pairs);
    for (uint32_t k = 0; k < c && c <= kSlots; ++k) {
        const int j = D.ws_slots[int64_t(k) * n + t];
        if (out + k < cap) pairs[out + k] = make_int2(min(i, j), max(i, j));
    }
    const bool again = c > kSlots && out < cap;
    if (__any_sync(0xffffffffu, again))
        walk_blocks(D, qb, again, s_q[threadIdx.x >> 5], [&](int src, unsigned hits, bool hit, int j) {
            const uint32_t k = __shfl_sync(0xffffffffu, out, src) + __popc(hits & ((1u << lane) - 1u));
            const int is = __shfl_sync(0xffffffffu, i, src);
            if (hit && k < cap) pairs[k] = make_int2(min(is, j), max(is, j));
            if (lane == src) out += __popc(hits);
        });
}

// ------------------------------------------------------------ narrowphase
__device__ __forceinline__ float3 pick3(float3 a, float3 b, float3 c, int i) { return i == 0 ? a : (i == 1 ? b : c); }

__device__ __forceinline__ bool inside_tri(float3 p1, float3 p2, float3 p3, float3 p) {
    const float3 c1 = cross(p2 - p1, p - p2), c2 = cross(p3 - p2, p - p3), c3 = cross(p1 - p3, p - p1);
    return dot(c1, c2) > 0.f && dot(c1, c3) > 0.f;
}

__device__ __forceinline__ float3 bary(float3 A, float3 B, float3 Cc, float3 P) {
    const float3 v0 = B - A, v1 = Cc - A, v2 = P - A;
    const float d00 = dot(v0, v0), d01 = dot(v0, v1), d11 = dot(v1, v1), d20 = dot(v2, v0), d21 = dot(v2, v1);
    const float den = d00 * d11 - d01 * d01;
    if (den == 0.f) return make_float3(1.f / 3.f, 1.f / 3.f, 1.f / 3.f);
    const float v = (d11 * d20 - d01 * d21) / den, w = (d00 * d21 - d01 * d20) / den;
    return make_float3(1.f - v - w, v, w);
}

__device__ __forceinline__ bool line_isect(float3 p1, float3 p2, float3 p3, float3 p4, float3 v1, float3 v2,
                                           float3& out) {
    const float3 d1 = p2 - p1, d2 = p4 - p3;
    const float3 nrm = cross(d1, d2);
    if (len(nrm) < 1.0e-6f) return false;
    const float den = dot(nrm, nrm);
    if (den < 1.0e-6f) return false;
    const float3 v = p3 - p1;
    const float t1 = dot(cross(v, d2), nrm) / den, t2 = dot(cross(v, d1), nrm) / den;
    if (!(t2 >= 0.f && t2 <= 1.f && t1 >= 0.f && t1 <= 1.f)) return false;
    out = v1 + t1 * (v2 - v1);
    return true;
}

__device__ __forceinline__ bool gen_t(float3 N, float3 v0, float3 v1, float3 v2, float d, float3 D, float2& iv) {
    const float d0 = dot(N, v0) + d, d1 = dot(N, v1) + d, d2 = dot(N, v2) + d;
    if (d0 <= kThresh && d1 <= kThresh && d2 <= kThresh) return false;
    if (d0 >= -kThresh && d1 >= -kThresh && d2 >= -kThresh) return false;
    float3 s0 = v0, s1 = v1, s2 = v2;
    float e0 = d0, e1 = d1, e2 = d2;
    if ((d0 <= 0.f && d1 >= 0.f && d2 >= 0.f) || (d0 >= 0.f && d1 <= 0.f && d2 <= 0.f)) {
        s0 = v1; s1 = v0; e0 = d1; e1 = d0;
    } else if ((d0 >= 0.f && d1 >= 0.f && d2 <= 0.f) || (d0 <= 0.f && d1 <= 0.f && d2 >= 0.f)) {
        s1 = v2; s2 = v1; e1 = d2; e2 = d1;
    }
    const float p0 = dot(D, s0), p1 = dot(D, s1), p2 = dot(D, s2);
    const float tA = p0 + (p1 - p0) * fabsf(e0 / (e0 - e1));
    const float tB = p2 + (p1 - p2) * fabsf(e2 / (e2 - e1));
    iv = tA > tB ? make_float2(tB, tA) : make_float2(tA, tB);
    return true;
}

__device__ __forceinline__ void respond(const XpbdDcd& D, const float* pos4, int4 cu, int4 cl, float4 f0, float4 f1,
                                        float4 f2);

// One pair; a contact is listed and responded to at once (the responses go to
// the accumulator, no position moves before k_dcd_apply).
__device__ __forceinline__ void narrow_pair(const XpbdDcd& D, const float* __restrict__ pos4, int k) {
    const int2 pair = reinterpret_cast<const int2*>(D.pairs)[k];
    const int ta = pair.x, tb = pair.y;
    const float3 q00 = f3(ld4(pos4, D.tris[3 * ta])), q01 = f3(ld4(pos4, D.tris[3 * ta + 1])),
                 q02 = f3(ld4(pos4, D.tris[3 * ta + 2]));
    const float3 q10 = f3(ld4(pos4, D.tris[3 * tb])), q11 = f3(ld4(pos4, D.tris[3 * tb + 1])),
                 q12 = f3(ld4(pos4, D.tris[3 * tb + 2]));
    const float3 n1f = cross(q01 - q00, q02 - q00), n2f = cross(q11 - q10, q12 - q10);
    const float l1 = len(n1f), l2 = len(n2f);
    if (l1 == 0.f || l2 == 0.f) return;
    const float3 N1 = n1f / l1, N2 = n2f / l2;
    const float d1 = -dot(N1, q00), d2 = -dot(N2, q10);
    const float3 cp = cross(N1, N2);
    const float lcp = len(cp);
    if (lcp < 1.0e-8f) return;
    const float3 Dd = cp / lcp;
    float2 iv1, iv2;
    if (!gen_t(N2, q00, q01, q02, d2, Dd, iv1)) return;
    if (!gen_t(N1, q10, q11, q12, d1, Dd, iv2)) return;
    if (!(iv1.y >= iv2.x && iv2.y >= iv1.x)) return;
    float C1 = 0.f, C2 = 0.f;
    float3 b1 = make_float3(0.f, 0.f, 0.f), b2 = b1, b3 = b1, b4 = b1;
    for (int j = 0; j < 3; ++j) {
        const float3 q0j = pick3(q00, q01, q02, j), q1j = pick3(q10, q11, q12, j);
        const float3 P0j = q0j - dot(N2, q0j - q10) * N2;
        if (inside_tri(q10, q11, q12, P0j)) {
            const float cand = dot(N2, q0j) + d2;
            if (C1 < -cand) {
                C1 = -cand;
                b1 = bary(q00, q01, q02, q0j);
                b2 = bary(q10, q11, q12, q0j - cand * N2);
            }
        }
        {
            const float den = dot(N1, N2);
            if (den != 0.f) {
                const float t = dot(N1, q00 - q1j) / den;
                const float3 Q0j = q1j + t * N2;
                if (inside_tri(q00, q01, q02, Q0j)) {
                    const float cand = dot(N2, Q0j) + d2;
                    if (C1 < -cand) {
                        C1 = -cand;
                        b1 = bary(q00, q01, q02, Q0j);
                        b2 = bary(q10, q11, q12, Q0j - cand * N2);
                    }
                }
            }
        }
        const float3 P1j = q1j - dot(N1, q1j - q00) * N1;
        if (inside_tri(q00, q01, q02, P1j)) {
            const float cand = dot(N1, q1j) + d1;
            if (C2 < -cand) {
                C2 = -cand;
                b3 = bary(q10, q11, q12, q1j);
                b4 = bary(q00, q01, q02, q1j - cand * N1);
            }
        }
        {
            const float den = dot(N2, N1);
            if (den != 0.f) {
                const float t = dot(N2, q10 - q0j) / den;
                const float3 Q1j = q0j + t * N1;
                if (inside_tri(q10, q11, q12, Q1j)) {
                    const float cand = dot(N1, Q1j) + d1;
                    if (C2 < -cand) {
                        C2 = -cand;
                        b3 = bary(q10, q11, q12, Q1j);
                        b4 = bary(q00, q01, q02, Q1j - cand * N1);
                    }
                }
            }
        }
        const int jn = (j + 1) % 3;
        const float3 q0jn = pick3(q00, q01, q02, jn), q1jn = pick3(q10, q11, q12, jn);
        const float3 P0jn = q0jn - dot(N2, q0jn - q10) * N2;
        const float3 P1jn = q1jn - dot(N1, q1jn - q00) * N1;
        for (int kk = 0; kk < 3; ++kk) {
            const int kn = (kk + 1) % 3;
            float3 o;
            if (line_isect(P0j, P0jn, pick3(q10, q11, q12, kk), pick3(q10, q11, q12, kn), q0j, q0jn, o)) {
                const float cand = dot(N2, o) + d2;
                if (C1 < -cand) {
                    C1 = -cand;
                    b1 = bary(q00, q01, q02, o);
                    b2 = bary(q10, q11, q12, o - cand * N2);
                }
            }
            if (line_isect(P1j, P1jn, pick3(q00, q01, q02, kk), pick3(q00, q01, q02, kn), q1j, q1jn, o)) {
                const float cand = dot(N1, o) + d1;
                if (C2 < -cand) {
                    C2 = -cand;
                    b3 = bary(q10, q11, q12, o);
                    b4 = bary(q00, q01, q02, o - cand * N1);
                }
            }
        }
    }
    if (C1 <= D.offset_eps || C2 <= D.offset_eps) return;
    const int slot = atomicAdd(D.n_contacts, 1);
    if (slot >= D.max_contacts) {
        atomicOr(D.status, XPBD_STATUS_CONTACT_OVERFLOW);
        return;
    }
    const bool first = C1 < C2;  // tie -> C2 branch
    const int tc = first ? ta : tb, tl = first ? tb : ta;
    int4* cid = reinterpret_cast<int4*>(D.c_ids);
    const int4 cu = make_int4(D.tris[3 * tc], D.tris[3 * tc + 1], D.tris[3 * tc + 2], k);
    const int4 cl = make_int4(D.tris[3 * tl], D.tris[3 * tl + 1], D.tris[3 * tl + 2], 0);
    cid[2 * slot] = cu;
    cid[2 * slot + 1] = cl;
    float4* cf = reinterpret_cast<float4*>(D.c_data);
    const float3 n = first ? N2 : N1;
    const float3 bb1 = first ? b1 : b3, bb2 = first ? b2 : b4;
    const float4 f0 = make_float4(n.x, n.y, n.z, first ? C1 : C2), f1 = make_float4(bb1.x, bb1.y, bb1.z, C1),
                 f2 = make_float4(bb2.x, bb2.y, bb2.z, C2);
    cf[3 * slot] = f0;
    cf[3 * slot + 1] = f1;
    cf[3 * slot + 2] = f2;
    respond(D, pos4, cu, cl, f0, f1, f2);
}

// The pair count is known on the device only: a grid that fills the GPU strides
// over it (a thread per possible pair was 16,384 CTAs, 17 us to find 31k pairs).
__global__ void __launch_bounds__(256) k_narrow(XpbdDcd D, const float* __restrict__ pos4) {
    const uint32_t np = uint32_t(min(*D.n_pairs, D.max_pairs));
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x)
        narrow_pair(D, pos4, int(k));
}

// respond_kernel (udcf/kernel.py:713-806)
__device__ __forceinline__ void respond(const XpbdDcd& D, const float* pos4, int4 cu, int4 cl, float4 f0, float4 f1,
                                        float4 f2) {
    float pen = f0.w;
    if (D.max_push > 0.f && pen > D.max_push) pen = D.max_push;
    float C = pen * D.multiplier;
    if (C == 0.f) return;
    const float3 nrm = make_float3(f0.x, f0.y, f0.z);
    const float4 pu0 = ld4(pos4, cu.x), pu1 = ld4(pos4, cu.y), pu2 = ld4(pos4, cu.z);
    const float4 pl0 = ld4(pos4, cl.x), pl1 = ld4(pos4, cl.y), pl2 = ld4(pos4, cl.z);
    const bool solid_cur = pu0.w == 0.f || pu1.w == 0.f || pu2.w == 0.f;
    const bool solid_clo = pl0.w == 0.f || pl1.w == 0.f || pl2.w == 0.f;
    if (!solid_cur && !solid_clo) C = C * 0.5f;
    const float3 push_clo = solid_clo ? make_float3(0.f, 0.f, 0.f) : (-C) * nrm;
    const float3 push_cur = solid_cur ? make_float3(0.f, 0.f, 0.f) : C * nrm;
    const float4* xp = reinterpret_cast<const float4*>(D.x_prev);
    const float3 v0 = (f3(pl0) + push_clo) - f3(xp[cl.x]), v1 = (f3(pl1) + push_clo) - f3(xp[cl.y]),
                 v2 = (f3(pl2) + push_clo) - f3(xp[cl.z]);
    const float3 v3 = (f3(pu0) + push_cur) - f3(xp[cu.x]), v4 = (f3(pu1) + push_cur) - f3(xp[cu.y]),
                 v5 = (f3(pu2) + push_cur) - f3(xp[cu.z]);
    const float3 g = nrm / len(nrm);
    const float3 b1 = make_float3(f1.x, f1.y, f1.z), b2 = make_float3(f2.x, f2.y, f2.z);
    const float3 vclo = (b1.x * v0 + b1.y * v1) + b1.z * v2;
    const float3 perp_clo = vclo - dot(vclo, g) * g;
    const float3 vcur = (b2.x * v3 + b2.y * v4) + b2.z * v5;
    const float3 perp_cur = vcur - dot(vcur, g) * g;
    float3 diff = perp_cur - perp_clo;
    const float dn = len(diff);
    const float static_norm = pen * D.friction_static;
    if (dn > static_norm && dn > 0.f) diff = (pen * D.friction_dynamic / dn) * diff;
    const float3 diffV = 0.5f * diff;
    const float3 diffT = diff - diffV;
    float4* acc = reinterpret_cast<float4*>(D.dP);
    const float3 mu = push_cur - diffV, ml = push_clo + diffT;
    if (pu0.w > 0.f) atomicAdd(&acc[cu.x], make_float4(mu.x, mu.y, mu.z, 1.f));
    if (pu1.w > 0.f) atomicAdd(&acc[cu.y], make_float4(mu.x, mu.y, mu.z, 1.f));
    if (pu2.w > 0.f) atomicAdd(&acc[cu.z], make_float4(mu.x, mu.y, mu.z, 1.f));
    if (pl0.w > 0.f) atomicAdd(&acc[cl.x], make_float4(ml.x, ml.y, ml.z, 1.f));
    if (pl1.w > 0.f) atomicAdd(&acc[cl.y], make_float4(ml.x, ml.y, ml.z, 1.f));
    if (pl2.w > 0.f) atomicAdd(&acc[cl.z], make_float4(ml.x, ml.y, ml.z, 1.f));
}

// apply_kernel (udcf/kernel.py:809-822), clearing the accumulator it reads
__global__ void k_dcd_apply(XpbdDcd D, float* pos4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.n_verts || *D.n_contacts == 0) return;
    float4* acc = reinterpret_cast<float4*>(D.dP);
    const float4 a = acc[i];
    if (a.w > 0.f) {
        float4 p = reinterpret_cast<float4*>(pos4)[i];
        if (D.jacobi_avg) {
            p.x += a.x / a.w;
            p.y += a.y / a.w;
            p.z += a.z / a.w;
        } else {
            p.x += a.x;
            p.y += a.y;
            p.z += a.z;
        }
        reinterpret_cast<float4*>(pos4)[i] = p;
        acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Sort CTAs: one per kSortThreads keys, at most the co-resident count.
int64_t hist_words(int n) { return int64_t(256) * ((n + kSortThreads - 1) / kSortThreads); }

int launch_sort(const XpbdDcd* D, const float* pos4, int snapshot, uint32_t* sync, cudaStream_t s) {
    static int slots[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cuda_check("xpbd_dcd_broadphase: device");
    if (slots[dev] == 0) {
        int n_sm = 0, per_sm = 0;
        if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sort_coop, kSortThreads, 0) != cudaSuccess)
            return cuda_check("xpbd_dcd_broadphase: sort occupancy");
        if (per_sm < 1) return fail(XPBD_ERR_LIMIT, "xpbd_dcd_broadphase: sort kernel does not fit an SM");
        slots[dev] = per_sm * n_sm;
    }
    const int n = D->n_tris;
    const int need = (n + kSortThreads - 1) / kSortThreads;
    const int G = std::min(need, slots[dev]);
    const int chunk = ((n + G - 1) / G + kSortThreads - 1) / kSortThreads * kSortThreads;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(kSortThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_sort_coop, *D, pos4, snapshot, chunk, sync) != cudaSuccess)
        return cuda_check("xpbd_dcd_broadphase: sort launch");
    return XPBD_OK;
}

int check_dcd(const XpbdDcd* D) {
    if (!D || D->n_tris <= 0 || D->n_verts <= 0 || !D->tris || !D->pairs || !D->n_pairs || !D->n_contacts ||
        !D->c_ids || !D->c_data || !D->x_prev || !D->dP || !D->status || !D->ws_nodes || !D->ws_keys || !D->ws_vals ||
        !D->ws_keys2 || !D->ws_vals2 || !D->ws_hist || !D->ws_bbox || !D->ws_split || !D->ws_count ||
        !D->ws_total || !D->ws_slots)
        return fail(XPBD_ERR_ARG, "XpbdDcd: null member or empty size");
    if (D->max_pairs <= 0 || D->max_contacts <= 0) return fail(XPBD_ERR_ARG, "XpbdDcd: capacities must be > 0");
    if (!aligned16(D->ws_nodes) || !aligned16(D->ws_bbox) || !aligned16(D->ws_split) || !aligned16(D->pairs) || !aligned16(D->c_ids) || !aligned16(D->c_data) || !aligned16(D->x_prev) ||
        !aligned16(D->dP))
        return fail(XPBD_ERR_ALIGN, "XpbdDcd: 16-byte alignment");
    return XPBD_OK;
}

}  // namespace

extern "C" {

int xpbd_dcd_workspace_query(int32_t n_tris, XpbdDcdWorkspaceSizes* out) {
    if (n_tris <= 0 || !out) return fail(XPBD_ERR_ARG, "xpbd_dcd_workspace_query: bad arguments");
    out->nodes_floats = int64_t(12) * n_tris;  // leaf records
    out->keys = n_tris;
    out->hist = hist_words(n_tris) + 4;  // sort histograms [CTAs][256], the sort's barrier words
    out->bbox_floats = int64_t(8) * ((n_tris + 31) / 32 + (n_tris + 1023) / 1024);  // 32- and 1024-leaf block boxes
    out->count = n_tris;
    out->slots = int64_t(kSlots) * n_tris;
    out->split = 4;  // unused
    return XPBD_OK;
}

int xpbd_dcd_broadphase(const XpbdDcd* D, const float* pos4, int32_t snapshot_prev, xpbd_stream_t stream) {
    int rc;
    if ((rc = check_dcd(D))) return rc;
    if (!pos4 || !aligned16(pos4)) return fail(XPBD_ERR_ARG, "xpbd_dcd_broadphase: pos4");
    cudaStream_t s = (cudaStream_t)stream;
    const int n = D->n_tris;
    if (D->refit_only) {
        if (snapshot_prev) k_snapshot<<<(D->n_verts + 255) / 256, 256, 0, s>>>(*D, pos4);
    } else if ((rc = launch_sort(D, pos4, snapshot_prev, reinterpret_cast<uint32_t*>(D->ws_hist + hist_words(n)), s))) {
        return rc;
    }
    k_leaves<<<(n + 1023) / 1024, 1024, 0, s>>>(*D, pos4);
    k_count_pairs<<<(n + 127) / 128, 128, 0, s>>>(*D);
    k_scan_pairs<<<1, 1024, 0, s>>>(*D);
    k_fill_pairs<<<(n + 127) / 128, 128, 0, s>>>(*D);
    return cuda_check("xpbd_dcd_broadphase");
}

int xpbd_dcd_narrow_respond(const XpbdDcd* D, float* pos4, xpbd_stream_t stream) {
    int rc;
    if ((rc = check_dcd(D))) return rc;
    if (!pos4 || !aligned16(pos4)) return fail(XPBD_ERR_ARG, "xpbd_dcd_narrow_respond: pos4");
    cudaStream_t s = (cudaStream_t)stream;
    cudaMemsetAsync(D->n_contacts, 0, sizeof(int32_t), s);
    k_narrow<<<std::min((D->max_pairs + 255) / 256, kNarrowCtas), 256, 0, s>>>(*D, pos4);
    k_dcd_apply<<<(D->n_verts + 255) / 256, 256, 0, s>>>(*D, pos4);
    return cuda_check("xpbd_dcd_narrow_respond");
}

}  // extern "C"
