// Whole frames in one cooperative launch (xpbd_frame_persistent).
//
// Each CTA keeps one tile's vertices in shared memory for all substeps.  Per
// substep every tile takes its own copies of the vertices through the substep
// boundary (push-out, velocity, prediction, pin; it depends on the vertex
// alone, so the copies of a vertex shared by several tiles stay equal bit for
// bit), then runs the Jacobi iterations: project the tile's tets into shared
// accumulators, send the partial sums of the shared vertices to the tiles that
// share them, fetch theirs, and finish all vertices.
//
// The partial sums travel through mailboxes instead of a global accumulator
// behind a grid-wide barrier.  A copy of a shared vertex owns a 16-byte slot
// (two, alternating): the three fixed-point sums and a word with the
// constraint count and the iteration's number.  The tile stores it once; the
// readers poll the slot itself until the number is this iteration's and add the
// integers to their own, so the order does not matter and all copies of a
// vertex get the same total.  One L2 round trip does the work of three
// (reduction, barrier, read-back), no fence waits for the reductions, and no
// tile waits for tiles it shares nothing with.  The barrier alone took 2.2 us of
// a 5.5-us iteration (17.6k tets, clock64 stamps) however small the mesh; with
// the mailboxes and one pass over the vertices per iteration that iteration
// takes 3.8 us, and 3.6 us with the constants of the attachments and the fibre
// and volume terms kept per material.  Frames of 200 iterations, device time
// against a launch per substep boundary and tet pass: 68k tets 1,288 -> 943 us,
// 222k tets 2.06 -> 1.72 ms; a 12,288-tet box of 10 iterations 113 -> 66 us.
//
// Two slots suffice: a tile stores iteration k + 2 only after it has read every
// neighbour's k + 1, which that neighbour sent after it had read k.  The
// iteration number goes on from launch to launch in the tile's own counter.
#include <cuda_runtime.h>

#include "xpbd_common.cuh"
#include "xpbd_grid.cuh"
#include "xpbd_tile.cuh"
#include "xpbd_vertex.cuh"

using namespace xpbd;

namespace {

constexpr int kThreads = 256;
// position, previous position, target, velocity, accumulators, flags
constexpr size_t kSmemPerVert = 4 * sizeof(float4) + 4 * sizeof(int) + sizeof(int);
// Tiles of at most kFixV vertices put the accumulators and the positions at
// compile-time offsets of the shared block (one register plus an immediate per
// shared access of the tet loop).
constexpr int kFixV = 768;

struct FrameArgs {
    int n_sub, n_iters;
    uint32_t first_ops, sub_ops, last_ops;
    int sdf_kind;  // 0 none, 1 one grid, 2 a grid per instance
    XpbdSdf sdf;
    XpbdSdfBatch batch;
    XpbdExchange ex;
};

// A slot is read and written as one 16-byte word, at L2 (its tiles run on other SMs).
__device__ __forceinline__ void st_slot(int4* p, int4 v) {
    asm volatile(
        "{\n .reg .b64 lo, hi;\n .reg .b128 q;\n mov.b64 lo, {%1, %2};\n mov.b64 hi, {%3, %4};\n"
        " mov.b128 q, {lo, hi};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p),
        "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
        : "memory");
}

__device__ __forceinline__ int4 ld_slot(const int4* p) {
    int4 v;
    asm volatile(
        "{\n .reg .b64 lo, hi;\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%4];\n mov.b128 {lo, hi}, q;\n"
        " mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}\n"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}

// The slot's contents of the iteration with this tag; v is what a first load
// gave.  Bounded as the grid barrier: after kSpinLimit polls the status bit is
// set and the wait ends, and a set bit ends every later wait early.
__device__ __forceinline__ int4 wait_slot(const int4* p, int4 v, uint32_t tag, int32_t* status) {
    uint32_t spins = 0;
    while ((uint32_t(v.w) >> 16) != tag) {
        if (++spins % kSpinCheck == 0u) {
            if (spins > kSpinLimit) {
                atomicOr(status, XPBD_STATUS_BARRIER_TIMEOUT);
                break;
            }
            if (*reinterpret_cast<volatile int32_t*>(status) & XPBD_STATUS_BARRIER_TIMEOUT) break;
        }
        v = ld_slot(p);
    }
    return v;
}

// acc += v in shared memory; a sum that leaves the 32-bit range sets the status bit.
__device__ __forceinline__ void add_checked(int* acc, int v, int32_t* status) {
    const int old = atomicAdd(acc, v), sum = int(uint32_t(old) + uint32_t(v));
    if (((old ^ sum) & (v ^ sum)) < 0 && status) atomicOr(status, XPBD_STATUS_ACC_RANGE);
}

// What stays fixed for the launch and is read between the tet loops: kept in
// shared memory, not in registers that the tet loop would spill.
struct TileState {
    int vbeg, nvt, nint, own_lo, own_hi, orph_lo, n_items;
    uint32_t seq0;
};

template <bool DAMP, int MINB, int CSET, bool FIXED>
__global__ void __launch_bounds__(kThreads, MINB)
    k_frame_tiles(const __grid_constant__ XpbdParams prm, const __grid_constant__ XpbdTiles T,
                  const __grid_constant__ XpbdVerts V, const __grid_constant__ XpbdPersist P,
                  const __grid_constant__ FrameArgs F) {
    extern __shared__ float4 smem[];
    __shared__ MatConsts s_mat[XPBD_MAX_MATERIALS];
    __shared__ float2 s_att[XPBD_MAX_ATTACH_MATERIALS];
    __shared__ int s_defer[2 + kDeferCap];
    __shared__ TileState s_tile;
    const int tile = P.tile_begin + int(blockIdx.x);
    const int mtv = T.max_tile_verts;
    float4 *s_pos, *s_prev, *s_tgt, *s_vel;
    int *s_ax, *s_ay, *s_az, *s_cnt, *s_f;
    int2* s_item;  // (other tile's copy, this tile's vertex) of every sum to fetch
    if constexpr (FIXED) {
        // [4 x kFixV accumulator ints][kFixV positions][prev, target, velocity: mtv each][items][flags]
        s_ax = reinterpret_cast<int*>(smem);
        s_ay = s_ax + kFixV;
        s_az = s_ay + kFixV;
        s_cnt = s_az + kFixV;
        s_pos = smem + kFixV;
        s_prev = smem + 2 * kFixV;
        s_tgt = s_prev + mtv;
        s_vel = s_tgt + mtv;
        s_item = reinterpret_cast<int2*>(s_vel + mtv);
        s_f = reinterpret_cast<int*>(s_item + F.ex.max_items);
    } else {
        s_pos = smem;
        s_prev = smem + mtv;
        s_tgt = smem + 2 * mtv;
        s_vel = smem + 3 * mtv;
        s_ax = reinterpret_cast<int*>(smem + 4 * mtv);
        s_ay = s_ax + mtv;
        s_az = s_ay + mtv;
        s_cnt = s_az + mtv;  // (4 mtv ints: the items stay 8-byte aligned)
        s_item = reinterpret_cast<int2*>(s_cnt + mtv);
        s_f = reinterpret_cast<int*>(s_item + F.ex.max_items);
    }
    // re-read after every tet loop (volatile: not kept in registers across it)
    const volatile TileState& S = s_tile;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr uint32_t kFinish = XPBD_APPLY_ATTACH | XPBD_APPLY_DIVIDE | XPBD_APPLY_PIN;
    {
        const int vbeg = T.tile_vptr[tile], nvt = T.tile_vptr[tile + 1] - vbeg;
        const int it0 = F.ex.item_ptr[tile], n_items = F.ex.item_ptr[tile + 1] - it0;
        for (int i = threadIdx.x; i < n_items; i += kThreads)
            s_item[i] = reinterpret_cast<const int2*>(F.ex.items)[it0 + i];
        if (threadIdx.x == 0) {
            s_tile.n_items = n_items;
            s_tile.vbeg = vbeg;
            s_tile.nvt = nvt;
            s_tile.nint = T.tile_nint[tile];
            s_tile.own_lo = P.tile_own[tile];
            s_tile.own_hi = P.tile_own[tile + 1];
            s_tile.orph_lo = P.tile_end == T.n_tiles ? P.tile_own[T.n_tiles] : V.n;  // last range only
            s_tile.seq0 = F.ex.tile_cnt[tile];
            s_defer[0] = s_defer[1] = 0;
        }
        fill_materials(prm, s_mat);
        fill_attach(prm, s_att);
        for (int i = threadIdx.x; i < nvt; i += kThreads) {
            const int g = T.tile_verts[vbeg + i];
            const int f = V.vflags ? V.vflags[g] : 0;
            s_pos[i] = reinterpret_cast<const float4*>(V.pos)[g];
            s_prev[i] = V.pprev ? reinterpret_cast<const float4*>(V.pprev)[g] : z4;
            s_vel[i] = V.vel ? reinterpret_cast<const float4*>(V.vel)[g] : z4;
            // one target per vertex: an active pin ends at its pin whatever an attachment adds
            float4 pin = z4;
            if (f & XPBD_VF_PIN) pin = reinterpret_cast<const float4*>(V.pin_target)[g];
            const bool pinned = pin.w != 0.f;
            s_f[i] = pinned ? XPBD_VF_PIN : (f & XPBD_VF_ATTACH_MASK);
            s_tgt[i] = pinned ? pin
                              : ((f & XPBD_VF_ATTACH_MASK) ? reinterpret_cast<const float4*>(V.attach_target)[g] : z4);
            // zeroed here and again wherever they are read: no clearing pass between iterations
            s_ax[i] = 0;
            s_ay[i] = 0;
            s_az[i] = 0;
            s_cnt[i] = 0;
        }
    }
    __syncthreads();
    const int n_total = F.n_sub * F.n_iters;
    for (int it = 0;; ++it) {
        // One pass over the tile's vertices: the finish of the last iteration (all
        // sums are in) and, between substeps, the substep boundary.  Kept in one
        // place: each phase's code runs once per iteration, and on small tiles its
        // instruction fetch, not its arithmetic, is what it costs.
        const bool boundary = it % F.n_iters == 0;
        const uint32_t vops = !boundary ? 0u : (it == 0 ? F.first_ops : (it == n_total ? F.last_ops : F.sub_ops));
        for (int i = threadIdx.x; i < S.nvt; i += kThreads) {
            float4 p = s_pos[i];
            const int f = s_f[i];
            float4 tg = z4;
            if (f) tg = s_tgt[i];
            if (it > 0) {
                const float4 a = tile_acc(s_ax, s_ay, s_az, s_cnt, i, 1.f / prm.acc_scale);
                s_ax[i] = 0;
                s_ay[i] = 0;
                s_az[i] = 0;
                s_cnt[i] = 0;
                finish_core(prm, f, tg, f ? s_prev[i] : z4, tg, p, a, kFinish, s_att);
            }
            if (vops) {
                uint32_t o = vops;
                float4 v = s_vel[i], q = s_prev[i];
                const int g = (F.sdf_kind == 2 || V.force) ? T.tile_verts[S.vbeg + i] : 0;
                if (F.sdf_kind == 2 && (o & XPBD_OP_SDF)) {
                    XpbdSdf sdf;
                    if (instance_sdf(F.batch, g, sdf)) sdf_push(sdf, p);
                    o &= ~uint32_t(XPBD_OP_SDF);
                }
                vertex_step_regs(prm, V, o, F.sdf, g, p, v, q);
                if ((o & XPBD_OP_PIN) && (f & XPBD_VF_PIN)) {
                    p.x = tg.x;
                    p.y = tg.y;
                    p.z = tg.z;
                }
                s_vel[i] = v;
                s_prev[i] = q;
            }
            s_pos[i] = p;
        }
        // The vertices in no tet, in global memory, each by one thread throughout.
        for (int g = S.orph_lo + int(blockIdx.x) * kThreads + threadIdx.x; g < V.n; g += gridDim.x * kThreads) {
            if (it > 0) {
                float4 pp = reinterpret_cast<const float4*>(V.pos)[g];
                finish_vertex(prm, V, g, pp, z4, kFinish);
                reinterpret_cast<float4*>(V.pos)[g] = pp;
            }
            if (vops) {
                XpbdSdf sdf = F.sdf;
                uint32_t o = vops;
                if (F.sdf_kind == 2 && (o & XPBD_OP_SDF) && !instance_sdf(F.batch, g, sdf)) o &= ~uint32_t(XPBD_OP_SDF);
                vertex_step_at(prm, V, o, sdf, g);
            }
        }
        if (it == n_total) break;
        __syncthreads();  // positions, zeroed accumulators
        project_tile_tets<DAMP, CSET>(prm, T, tile, s_pos, s_prev, s_ax, s_ay, s_az, s_cnt, s_mat, s_defer, it & 1);
        __syncthreads();
        const int nvt = S.nvt, n_items = S.n_items;
        const uint32_t seq = S.seq0 + uint32_t(it) + 1u, tag = seq & 0xffffu;
        int4* slots = reinterpret_cast<int4*>(F.ex.slots) + (seq & 1u ? size_t(F.ex.n_copies) : 0);
        for (int i = S.nint + threadIdx.x; i < nvt; i += kThreads)
            st_slot(slots + S.vbeg + i,
                    make_int4(s_ax[i], s_ay[i], s_az[i], int((tag << 16) | (uint32_t(s_cnt[i]) & 0xffffu))));
        __syncthreads();  // every own sum is in its slot before foreign ones are added to it
        // two fetches in flight per thread
        for (int j = threadIdx.x; j < n_items; j += 2 * kThreads) {
            const bool two = j + kThreads < n_items;
            const int2 e0 = s_item[j], e1 = s_item[two ? j + kThreads : j];
            int4 v0 = ld_slot(slots + e0.x), v1 = ld_slot(slots + e1.x);
            v0 = wait_slot(slots + e0.x, v0, tag, P.status);
            add_checked(&s_ax[e0.y], v0.x, P.status);
            add_checked(&s_ay[e0.y], v0.y, P.status);
            add_checked(&s_az[e0.y], v0.z, P.status);
            atomicAdd(&s_cnt[e0.y], v0.w & 0xffff);
            if (two) {
                v1 = wait_slot(slots + e1.x, v1, tag, P.status);
                add_checked(&s_ax[e1.y], v1.x, P.status);
                add_checked(&s_ay[e1.y], v1.y, P.status);
                add_checked(&s_az[e1.y], v1.z, P.status);
                atomicAdd(&s_cnt[e1.y], v1.w & 0xffff);
            }
        }
        __syncthreads();
    }
    // write-back by the threads that finished the vertices
    for (int i = threadIdx.x; i < S.nvt; i += kThreads) {
        const int g = T.tile_verts[S.vbeg + i];
        if (i < S.nint || (g >= S.own_lo && g < S.own_hi)) {
            if (F.first_ops | F.sub_ops | F.last_ops) {
                reinterpret_cast<float4*>(V.pprev)[g] = s_prev[i];
                reinterpret_cast<float4*>(V.vel)[g] = s_vel[i];
            }
            reinterpret_cast<float4*>(V.pos)[g] = s_pos[i];
        }
    }
    if (threadIdx.x == 0) F.ex.tile_cnt[tile] = S.seq0 + uint32_t(F.n_sub * F.n_iters);
    // The accumulator ring's phase (sync[2]) counts these iterations too.  Its
    // next launch may start on any slot of it, so where one has ever written the
    // ring (sync[3] bit 1), the shared vertices' slots are left zero.
    if (P.ring && P.sync) {
        if (P.sync[3] & 2u) {
            for (int i = S.nint + threadIdx.x; i < S.nvt; i += kThreads) {
                const int g = T.tile_verts[S.vbeg + i];
                if (g < S.own_lo || g >= S.own_hi) continue;
                for (int k = 0; k < 3; ++k) reinterpret_cast<float4*>(P.ring)[size_t(k) * V.n + g] = z4;
            }
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) P.sync[2] = (P.sync[2] + uint32_t(F.n_sub * F.n_iters)) % 3u;
    }
}

uint32_t material_union(const XpbdParams* p) {
    uint32_t u = 0;
    for (int i = 0; i < p->n_materials; ++i) u |= p->materials[i].flags;
    return u;
}

bool has_damped(const XpbdParams* prm) { return (material_union(prm) & XPBD_MAT_DAMPED) != 0; }

// One launch (or, with slots set, one occupancy query) of an instance.
struct Launch {
    const XpbdParams* prm;
    const XpbdTiles* T;
    const XpbdVerts* V;
    const XpbdPersist* P;
    const FrameArgs* F;
    cudaStream_t s;
    int max_items;
    int64_t* slots;
};

template <bool DAMP, int MINB, int CSET, bool FIXED>
int launch_v(const Launch& L) {
    auto kern = k_frame_tiles<DAMP, MINB, CSET, FIXED>;
    const size_t fix = 4 * sizeof(int) + sizeof(float4);  // accumulators and positions
    const size_t smem = (FIXED ? size_t(kFixV) * fix + size_t(L.T->max_tile_verts) * (kSmemPerVert - fix)
                               : size_t(L.T->max_tile_verts) * kSmemPerVert) +
                        size_t(L.max_items) * sizeof(int2);
    if (!allow_smem(kern, smem)) {
        cudaGetLastError();
        if (!L.slots) return fail(XPBD_ERR_LIMIT, "xpbd_frame_persistent: a tile's vertices and items exceed an SM");
        *L.slots = 0;
        return XPBD_OK;
    }
    int dev = 0, n_sm = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess)
        return cuda_check("xpbd_frame_persistent: occupancy");
    const int64_t slots = int64_t(per_sm) * n_sm;
    if (L.slots) {
        *L.slots = slots;
        return XPBD_OK;
    }
    const int ntl = L.P->tile_end - L.P->tile_begin;
    if (ntl > slots) return fail(XPBD_ERR_LIMIT, "xpbd_frame_persistent: tiles exceed the resident CTA slots");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ntl);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = L.s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // tiles wait for one another: all must be resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, *L.prm, *L.T, *L.V, *L.P, *L.F) != cudaSuccess)
        return cuda_check("xpbd_frame_persistent: launch");
    return cuda_check("xpbd_frame_persistent");
}

// The instances of the per-iteration pass (xpbd_project) that a frame has: the
// smallest constraint set covering the materials; bit 0 of tile_variant runs
// undamped volume sets at 3 CTAs per SM instead of 2, bit 4 keeps the runtime
// shared layout for small tiles.
int dispatch(const Launch& L) {
    const uint32_t u = material_union(L.prm);
    const bool damp = has_damped(L.prm);
    const bool flip = (L.prm->tile_variant & 1) != 0;
    const bool fixed = L.T->max_tile_verts <= kFixV && !(L.prm->tile_variant & 16);
#define XPBD_LAUNCH(D, M, C) (fixed ? launch_v<D, M, C, true>(L) : launch_v<D, M, C, false>(L))
    if (u & XPBD_MAT_SNH) return damp ? XPBD_LAUNCH(true, 2, CSET_FULL) : XPBD_LAUNCH(false, 2, CSET_FULL);
    if (u & XPBD_MAT_VOLUME) {
        if (damp) return XPBD_LAUNCH(true, 2, CSET_VOL);
        return flip ? XPBD_LAUNCH(false, 3, CSET_VOL) : XPBD_LAUNCH(false, 2, CSET_VOL);
    }
    return XPBD_LAUNCH(false, 3, CSET_LIGHT);
#undef XPBD_LAUNCH
}

}  // namespace

extern "C" int xpbd_frame_persistent(const XpbdParams* prm, const XpbdTiles* tiles, const XpbdVerts* v,
                                     const XpbdPersist* ps, const XpbdFrame* f, xpbd_stream_t stream) {
    if (!prm || !tiles || !v || !ps || !f || !f->ex) return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: null argument");
    if (f->n_sub < 1 || f->n_iters < 1) return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: n_sub and n_iters >= 1");
    if (int64_t(f->n_sub) * f->n_iters > (1 << 20))
        return fail(XPBD_ERR_LIMIT, "xpbd_frame_persistent: more than 2^20 iterations");
    if (!v->pos || v->n <= 0 || !tiles->tile_vptr || !tiles->tile_nint || !tiles->tile_tptr || !tiles->tile_verts ||
        !tiles->tet_q || !tiles->tet_b0 || !tiles->tet_b1 || !tiles->tet_b2 || tiles->n_tiles <= 0)
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: tiles/verts");
    if (!ps->tile_own || !ps->status || (ps->ring && !aligned16(ps->ring)))
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: XpbdPersist pointers");
    const XpbdExchange& ex = *f->ex;
    if (!ex.item_ptr || !ex.items || !ex.slots || !ex.tile_cnt || ex.n_copies <= 0 || ex.max_items < 0)
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: XpbdExchange");
    if (!aligned16(v->pos) || !aligned16(v->pprev) || !aligned16(v->vel) || !aligned16(v->force) ||
        !aligned16(v->attach_target) || !aligned16(v->pin_target) || !aligned16(ex.slots) || (reinterpret_cast<uintptr_t>(ex.items) & 7u) || !aligned16(tiles->tet_q) ||
        !aligned16(tiles->tet_b0) || !aligned16(tiles->tet_b1) || !aligned16(tiles->tet_fiber))
        return fail(XPBD_ERR_ALIGN, "xpbd_frame_persistent: [n][4] arrays must be 16-byte aligned");
    if (v->vflags && (!v->attach_target || !v->pin_target))
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: vflags given without attach_target/pin_target");
    if (tiles->max_tile_verts <= 0 || tiles->max_tile_verts > XPBD_MAX_TILE_VERTS)
        return fail(XPBD_ERR_LIMIT, "xpbd_frame_persistent: tile size");
    if (prm->n_materials < 1 || prm->n_materials > XPBD_MAX_MATERIALS || prm->n_attach_materials < 0 ||
        prm->n_attach_materials > XPBD_MAX_ATTACH_MATERIALS)
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: material counts");
    if (!(prm->dt > 0.f)) return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: dt must be > 0");
    if (!(prm->acc_scale > 0.f) || !(prm->acc_scale < 3.0e38f))
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: acc_scale must be a finite value > 0");
    if ((material_union(prm) & XPBD_MAT_ANISO) && (!tiles->tet_fiber || !tiles->tet_act))
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: aniso materials need tet_fiber and tet_act");
    const uint32_t ops = f->first_ops | f->sub_ops | f->last_ops;
    if ((ops || has_damped(prm)) && !v->pprev) return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: pprev required");
    if (ops && (!v->vel || (v->force && !v->mass)))
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: vel required, mass with force");
    XpbdPersist P = *ps;
    if (P.tile_begin == 0 && P.tile_end == 0) P.tile_end = tiles->n_tiles;
    if (P.tile_begin < 0 || P.tile_end > tiles->n_tiles || P.tile_begin >= P.tile_end)
        return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: tile range");
    FrameArgs F = {};
    F.n_sub = f->n_sub;
    F.n_iters = f->n_iters;
    F.first_ops = f->first_ops;
    F.sub_ops = f->sub_ops;
    F.last_ops = f->last_ops;
    F.ex = ex;
    if (ops & XPBD_OP_SDF) {
        if (!f->sdf == !f->sdf_batch)
            return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: XPBD_OP_SDF needs sdf or sdf_batch, not both");
        if (f->sdf) {
            if (!f->sdf->phi || f->sdf->nx < 2 || f->sdf->ny < 2 || f->sdf->nz < 2 || !(f->sdf->h > 0.f))
                return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: XpbdSdf");
            F.sdf_kind = 1;
            F.sdf = *f->sdf;
        } else {
            const XpbdSdfBatch& b = *f->sdf_batch;
            if (!b.phi || !b.frame || !b.vert_inst || b.n_inst < 1 || b.nx < 2 || b.ny < 2 || b.nz < 2)
                return fail(XPBD_ERR_ARG, "xpbd_frame_persistent: XpbdSdfBatch");
            if (!aligned16(b.frame)) return fail(XPBD_ERR_ALIGN, "xpbd_frame_persistent: frame");
            F.sdf_kind = 2;
            F.batch = b;
        }
    }
    return dispatch({prm, tiles, v, &P, &F, (cudaStream_t)stream, ex.max_items, nullptr});
}

extern "C" int xpbd_frame_fits(const XpbdParams* prm, const XpbdTiles* tiles, const XpbdExchange* ex, int32_t* fits,
                               int32_t* slots) {
    if (!prm || !tiles || !ex || !fits) return fail(XPBD_ERR_ARG, "xpbd_frame_fits: null argument");
    if (prm->n_materials < 1 || prm->n_materials > XPBD_MAX_MATERIALS)
        return fail(XPBD_ERR_ARG, "xpbd_frame_fits: n_materials");
    int64_t n = 0;
    const int rc = dispatch({prm, tiles, nullptr, nullptr, nullptr, nullptr, ex->max_items, &n});
    *fits = n >= tiles->n_tiles ? 1 : 0;
    if (slots) *slots = int32_t(n);
    return rc;
}
