// batch.cuh -- many independent scenes advanced together (included by
// engine.cu after the single-scene engine).
//
// rfsyn runs its examples one at a time (cli/main.c:362-417); a scene of a
// few hundred thousand cells cannot fill a B200, and each of its steps pays
// the launch latency of four kernels.  A batch keeps every scene resident in
// its own buffers (an engine created as a batch member: fields, slab psi,
// codes, interface list, sources, probes) and advances all of them with the
// same launches per step:
//   k_vsweep_b -- the vector sweep (vsweep.cuh) over (scene, tile, plane
//     range) items of every scene, each CTA copying its scene's parameters
//     (Args) into shared memory; under a plan override k_sweep_qb, the
//     work-queue sweeps of sweep.cuh over queues of such items;
//   k_e_list_b -- the interface-list entries of every scene, one block per
//     256 entries of one scene;
//   k_probe_gather_b -- every probe of every scene, then the shared step
//     counter.
// Steps are captured in CUDA graphs (16 steps per graph); tile shapes and the
// segment length follow from the scenes' sizes (batch_build_vplan).  Scenes
// whose tile halos would wrap around a periodic y or z axis are not admitted.
#pragma once

namespace rfb {

struct BatchItem {
    int scene;
    SweepItem t;
};

// Copies one scene's Args into the CTA's shared copy (32-bit words).
template <typename T>
__device__ __forceinline__ void load_args(Args<T> &dst, const Args<T> *src, int nthreads, int tid) {
    const unsigned *s = reinterpret_cast<const unsigned *>(src);
    unsigned *d = reinterpret_cast<unsigned *>(&dst);
    for (int t = tid; t < (int)(sizeof(Args<T>) / 4); t += nthreads) d[t] = s[t];
}

// Tensor maps written by the host before the launch are read through the
// tensormap proxy: order the generic-proxy copy before their first use.
__device__ __forceinline__ void tensormap_acquire(const TmaMaps *m) {
    const CUtensorMap *maps[14] = {&m->e[0],  &m->e[1],  &m->e[2],  &m->h[0],  &m->h[1],  &m->h[2],  &m->code,
                                   &m->en[0], &m->en[1], &m->en[2], &m->hn[0], &m->hn[1], &m->hn[2], &m->coden};
#pragma unroll
    for (int q = 0; q < 14; q++)
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(maps[q]) : "memory");
}

// Dynamic shared memory of the batched sweep: the single-scene layout, then
// the CTA's copy of the current scene's parameters.  No static shared
// memory: it would precede the dynamic region and break the 128-byte
// alignment the tensor copies need.
template <typename T, int TJ, int NS>
struct QBLayout {
    static constexpr size_t args = round128(QLayout<T, TJ, NS>::total);
    static constexpr size_t total = args + sizeof(Args<T>);
};

template <typename T, int TJ, int NS, int MINB, int KIND>
__global__ void __launch_bounds__(32 * TJ, MINB)
    k_sweep_qb(const Args<T> *args, const FusedDims *dims, const TmaMaps *maps, const BatchItem *items, int n_items,
               int *queue, int *err) {
    static_assert(NS >= 3, "the ring must hold the current, the next and one prefetched plane");
    static_assert(TJ >= 5, "warps 0-3 share the halo recomputation, warp 4 issues the copies");
    using S = QLayout<T, TJ, NS>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if (q_misaligned(smem_raw, err)) return;
    Args<T> &sa = *reinterpret_cast<Args<T> *>(smem_raw + QBLayout<T, TJ, NS>::args);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + S::bars);
    volatile int *s_item = reinterpret_cast<volatile int *>(smem_raw + S::misc);
    const int tid = threadIdx.y * 32 + threadIdx.x;
    q_init_bars<NS>(bars);
    unsigned phase = 0, pending = 0;
    bool failed = false;
    int cur = -1;
    for (;;) {
        if (tid == 0) *s_item = atomicAdd(&queue[0], 1);
        __syncthreads();
        const int w = *s_item;
        if (w >= n_items) break;
        const BatchItem bi = items[w];
        if (bi.scene != cur) {
            load_args(sa, args + bi.scene, 32 * TJ, tid);
            // the fence orders the maps for the thread that issues the copies
            if (tid == kCopyIssueTid) tensormap_acquire(maps + bi.scene);
            __syncthreads();
            q_load_table<T, TJ, NS>(sa, smem_raw);
            __syncthreads();
            cur = bi.scene;
        }
        if (!q_run<T, TJ, NS, KIND>(sa, dims[bi.scene], maps[bi.scene], bi.t, smem_raw, phase, pending, failed)) {
            q_bail<NS>(bars, phase, pending, err);
            break;
        }
        __syncthreads();  // the ring, the tables and the item slot are free again
    }
    q_leave(queue);
}

// Interface-list entries of many scenes: block b updates entries
// blocks[b].y .. +255 of scene blocks[b].x.
template <typename T>
__global__ void __launch_bounds__(256) k_e_list_b(const Args<T> *args, const int2 *blocks) {
    __shared__ Args<T> sa;
    grid_launch_next();
    const int2 b = blocks[blockIdx.x];
    load_args(sa, args + b.x, 256, threadIdx.x);
    __syncthreads();
    grid_wait();
    const int e = b.y + threadIdx.x;
    if (e < 3 * sa.n_cells) e_list_entry(sa, e);
}

template <typename T>
struct ProbeRefB {
    const T *f[2];     // the probed component in field buffer 0 and 1
    long long cell;
    T *ts;             // the probe's time series (n_steps samples)
};

// Records sample n of every probe of every scene from the output buffer of
// the step, then advances the batch's step counter (single block).
template <typename T>
__global__ void k_probe_gather_b(const ProbeRefB<T> *p, int n, int out_buf, long long n_steps, int *d_step) {
    __shared__ int step;
    grid_launch_next();
    grid_wait();
    if (threadIdx.x == 0) step = *d_step;
    __syncthreads();
    if (step < n_steps)
        for (int q = threadIdx.x; q < n; q += blockDim.x) p[q].ts[step] = p[q].f[out_buf][p[q].cell];
    __syncthreads();
    if (threadIdx.x == 0) *d_step = step + 1;
}

// CTAs per SM of the batched sweeps: the interior as in the single-scene
// plan; the FP32 x-slab and edge kinds, which keep the scene's parameters in
// registers loaded from shared memory, at 3 (8-row tiles) or 1 (16-row);
// the FP32 single-queue kind with 8-row tiles at 4 (64 registers, 176 bytes
// of spills, against 80 registers at 3: stalled on waits, barriers and
// instruction fetch, it gains from the extra warps -- C4's step 4.681 ->
// 4.616 ms); FP64 as in the single-scene plan.
#define RFB_QB_MINB(TT, TJ_, MBI_, MBE_, KIND_) \
    ((KIND_) == 0 ? (MBI_) : sizeof(TT) == 8 ? (MBE_) : ((TJ_) == 16 ? 1 : (KIND_) == 5 ? 4 : 3))
#define RFB_LAUNCH_QB(TT, TJ_, NS_, MBI_, MBE_)                                                            \
    if (tj == TJ_ && ns == NS_) {                                                                          \
        constexpr int MB_ = RFB_QB_MINB(TT, TJ_, MBI_, MBE_, KIND);                                                  \
        const int g = std::min(n, qb_grid<TT, TJ_, NS_, MB_, KIND>());                                     \
        k_sweep_qb<TT, TJ_, NS_, MB_, KIND><<<g, dim3(32, TJ_), QBLayout<TT, TJ_, NS_>::total, st>>>(      \
            args, dims, maps, items, n, queue, err);                                                       \
    }

template <typename T, int TJ, int NS, int MINB, int KIND>
inline int qb_grid() {
    static int g = 0;
    if (!g) {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sweep_qb<T, TJ, NS, MINB, KIND>, 32 * TJ,
                                                      QBLayout<T, TJ, NS>::total);
        g = (sms > 0 ? sms : 148) * (per > 0 ? per : 1);
    }
    return g;
}

template <int KIND, typename T>
inline void launch_qb(const Args<T> *args, const FusedDims *dims, const TmaMaps *maps, int tj, int ns,
                      const BatchItem *items, int n, int *queue, int *err, cudaStream_t st) {
    if (n <= 0) return;
    if constexpr (sizeof(T) == 4) {
        RFB_Q_VARIANTS_FP32(RFB_LAUNCH_QB)
    } else {
        RFB_Q_VARIANTS_FP64(RFB_LAUNCH_QB)
    }
}

#define RFB_PREP_QB(TT, TJ_, NS_, MBI_, MBE_)                                                               \
    if (e == cudaSuccess)                                                                                   \
        e = cudaFuncSetAttribute(k_sweep_qb<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 0), 0>,                   \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QBLayout<TT, TJ_, NS_>::total); \
    if (e == cudaSuccess)                                                                                   \
        e = cudaFuncSetAttribute(k_sweep_qb<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 1), 1>,                   \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QBLayout<TT, TJ_, NS_>::total); \
    if (e == cudaSuccess)                                                                                   \
        e = cudaFuncSetAttribute(k_sweep_qb<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 2), 2>,                   \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QBLayout<TT, TJ_, NS_>::total); \
    if (e == cudaSuccess)                                                                                   \
        e = cudaFuncSetAttribute(k_sweep_qb<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 5), 5>,                   \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QBLayout<TT, TJ_, NS_>::total); \
    if (e == cudaSuccess) {                                                                                 \
        (void)qb_grid<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 5), 5>();                                       \
        (void)qb_grid<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 0), 0>();                                       \
        (void)qb_grid<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 1), 1>();                                       \
        (void)qb_grid<TT, TJ_, NS_, RFB_QB_MINB(TT, TJ_, MBI_, MBE_, 2), 2>();                                       \
    }
static inline int qb_prepare() {
    static int done = 0;
    if (done) return 0;
    cudaError_t e = cudaSuccess;
    RFB_Q_VARIANTS_FP32(RFB_PREP_QB)
    RFB_Q_VARIANTS_FP64(RFB_PREP_QB)
    if (e != cudaSuccess) return -1;
    done = 1;
    return 0;
}

}  // namespace rfb

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Threads of the vector sweep's CTAs.  us a step at 192 / best of 160 / best of
// 128 threads (segments 12-32): 96 scenes of 32-96 cells an axis FP32 602 /
// 660 / 623, FP64 1113 / 1167 / 1339; 12 of 60-96 FP32 140 / 151 / 140, FP64
// 226 / 250 / 278; 30 of 40-80 FP32 184 / 202 / 190, FP64 310 / 334 / 377.
// Batches of few small scenes can want fewer: 20 of 32-60 FP32 75 / 79 / 67.
constexpr int V_BATCH_NT = 192;

struct rfb_batch {
    std::vector<rfb_engine *> m;  // members (owned)
    int prec = RFB_FP32;
    size_t n_steps = 0, steps_done = 0;
    int parity = 0;
    cudaStream_t stream = nullptr, stream2 = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    int own_stream = 0;
    int *d_step = nullptr, *d_err = nullptr, *d_queue = nullptr;
    void *d_args[2] = {};          // Args<T>[n] per parity
    FusedDims *d_dims = nullptr;
    TmaMaps *d_maps[2] = {};
    BatchItem *d_items[3] = {};    // interior, x slab, edge (uni: every item in the edge list)
    int n_items[3] = {};
    int uni = 0;
    bool overlap = false;          // launches are being captured as programmatic dependents
    // mode 5: the vector sweep's items of every scene, shapes and maps
    VItem *d_vitems = nullptr;
    int n_vitems = 0, n_vplain = 0, v_nt = 0, v_smem = 0;
    VShape *d_vshapes = nullptr;
    VMaps *d_vmaps[2] = {};
    int2 *d_lblocks = nullptr;
    int n_lblocks = 0;
    void *d_probes = nullptr;
    int n_probes = 0;
    int tj = 8, ns = 4, mode = 2, seg_int = 64, seg_edge = 32;
    size_t cells = 0, list_cells = 0, slab_cell_axes = 0;
    static constexpr int CHUNK = 16;
    cudaGraphExec_t g1[2] = {nullptr, nullptr}, gk[2] = {nullptr, nullptr};
};

static void batch_free_plan(rfb_batch *b) {
    for (int k = 0; k < 3; k++) {
        dfree(b->d_items[k]);
        b->d_items[k] = nullptr;
        b->n_items[k] = 0;
    }
    for (int q = 0; q < 2; q++) {
        if (b->g1[q]) cudaGraphExecDestroy(b->g1[q]);
        if (b->gk[q]) cudaGraphExecDestroy(b->gk[q]);
        b->g1[q] = b->gk[q] = nullptr;
        dfree(b->d_maps[q]);
        b->d_maps[q] = nullptr;
        dfree(b->d_vmaps[q]);
        b->d_vmaps[q] = nullptr;
    }
    dfree(b->d_dims);
    b->d_dims = nullptr;
    dfree(b->d_vitems);
    dfree(b->d_vshapes);
    b->d_vitems = nullptr;
    b->d_vshapes = nullptr;
    b->n_vitems = b->n_vplain = 0;
}

// Plan of mode 5, the vector sweep of every scene in one launch: per scene
// the tile of at most `threads` threads that spends the fewest threads on the
// grid, of those that leave an SM room for V_MB CTAs (one scene's larger tile
// would halve the CTAs of the whole batch), and one segment length for the
// batch: one wave of CTAs where that
// takes at most 16 planes each, else waves of at most 32 (seg and seg_edge,
// for plain and slab items, where a plan override gives them).  Items of one kind
// together, the costly kinds first.  96 scenes of 32-96 cells an axis, FP32:
// 68.5 ms for 96 steps; with 128 threads 68.4-84 (segments of 32-6), with 192
// and 12-32 planes 72.1-68.8.
static int batch_build_vplan(rfb_batch *b, int threads, int seg, int seg_edge) {
    batch_free_plan(b);
    const size_t n = b->m.size();
    std::vector<VShape> shapes(n);
    std::vector<VMaps> maps[2];
    std::vector<VItem> items;
    maps[0].resize(n);
    maps[1].resize(n);
    double planes = 0;
    int smem = 0;
    const int args_bytes = b->prec == RFB_FP64 ? v_args_bytes<double>() : v_args_bytes<float>();
    for (size_t s = 0; s < n; s++) {
        rfb_engine *e = b->m[s];
        if (e->g.periodic & 6u) {
            rfb_set_error("batch scene %zu: a tile halo wraps around a periodic y or z axis", s);
            return -1;
        }
        if (!v_fits(e)) {
            rfb_set_error("batch scene %zu too large for the vector sweep (32-bit offsets)", s);
            return -1;
        }
        const int N = e->prec == RFB_FP64 ? 2 : 4;
        int cj, ck, ci;
        v_extents(e, e->active, &cj, &ck, &ci);
        const int nvk = (ck + N - 1) / N;
        long long best = -1, best_tiles = 0;
        for (int nk = 1, pv = 0; nk <= nvk; nk++) {
            const int nv = (nvk + nk - 1) / nk;
            if (nv == pv) continue;
            pv = nv;
            for (int tr = std::min(cj, threads / (nv + 1) - 1); tr >= 1; tr--) {
                const int nj = (cj + tr - 1) / tr;
                if (tr > 1 && nj == (cj + tr - 2) / (tr - 1)) continue;
                VShape t;
                if (!v_layout(e, t, nv, tr, cj, ck, threads)) continue;
                if (v_slots(threads, (int)round_up(t.smem, 16) + args_bytes) < V_MB) continue;
                const long long tiles = (long long)((nvk + nv - 1) / nv) * nj;
                const long long cost = tiles * ((tr + 1) * (nv + 1) + threads);
                if (best < 0 || cost < best) {
                    best = cost;
                    best_tiles = tiles;
                    shapes[s] = t;
                }
            }
        }
        if (best < 0) {
            rfb_set_error("batch scene %zu: no tile fits", s);
            return -1;
        }
        planes += (double)best_tiles * ci;
        smem = std::max(smem, shapes[s].smem);
        if (v_encode(e, shapes[s]) != 0) return -1;
        maps[0][s] = e->vmaps[0];
        maps[1][s] = e->vmaps[1];
    }
    smem = (int)round_up(smem, 16);
    const double slots = 148.0 * v_slots(threads, smem + args_bytes);
    if (seg <= 0) {
        const double per_slot = planes / slots;
        seg = std::max(1, (int)ceil(per_slot <= 16 ? per_slot : per_slot / std::max(2.0, ceil(per_slot / 32))));
        seg_edge = seg;
    }
    b->n_vplain = 0;
    for (size_t s = 0; s < n; s++) {
        int cj, ck, ci;
        v_extents(b->m[s], b->m[s]->active, &cj, &ck, &ci);
        const int most = v_max_seg(b->m[s]);
        v_items(b->m[s], shapes[s], ci, std::min(seg, most), std::min(seg_edge, most), (int)s, items, &b->n_vplain);
    }
    auto rank = [](const VItem &x) { return x.kind & V_X ? 0 : 4 - x.kind; };
    std::stable_sort(items.begin(), items.end(), [&](const VItem &x, const VItem &y) {
        if (rank(x) != rank(y)) return rank(x) < rank(y);
        return x.ie - x.ib > y.ie - y.ib;
    });
    b->mode = 5;
    b->uni = 1;
    b->tj = threads;
    b->ns = V_NH;
    b->seg_int = seg;
    b->seg_edge = seg_edge;
    b->v_nt = threads;
    b->v_smem = smem;
    b->n_vitems = (int)items.size();
    CK(dmalloc(&b->d_vitems, items.size() * sizeof(VItem)));
    CK(cudaMemcpy(b->d_vitems, items.data(), items.size() * sizeof(VItem), cudaMemcpyHostToDevice));
    CK(dmalloc(&b->d_vshapes, n * sizeof(VShape)));
    CK(cudaMemcpy(b->d_vshapes, shapes.data(), n * sizeof(VShape), cudaMemcpyHostToDevice));
    for (int q = 0; q < 2; q++) {
        CK(dmalloc(&b->d_vmaps[q], n * sizeof(VMaps)));
        CK(cudaMemcpy(b->d_vmaps[q], maps[q].data(), n * sizeof(VMaps), cudaMemcpyHostToDevice));
    }
    return 0;
fail:
    return -1;
}

// Work lists and per-scene tensor maps / dims of one plan.
static int batch_build_plan(rfb_batch *b, int tj, int ns, int mode, int seg_int, int seg_edge, int uni = 0) {
    batch_free_plan(b);
    b->tj = tj;
    b->ns = ns;
    b->mode = mode;
    b->uni = uni;
    b->seg_int = seg_int;
    b->seg_edge = seg_edge;
    const size_t n = b->m.size();
    std::vector<BatchItem> lists[3];
    std::vector<FusedDims> dims(n);
    std::vector<TmaMaps> maps[2];
    maps[0].resize(n);
    maps[1].resize(n);
    for (size_t s = 0; s < n; s++) {
        rfb_engine *e = b->m[s];
        if (mode == 4 && (e->g.periodic & 6u)) {
            rfb_set_error("batch scene %zu: sweep mode 4 needs non-periodic y and z axes", s);
            return -1;
        }
        PlanLists pl;
        plan_items(e, e->active, tj, mode, seg_int, seg_edge, pl);
        if (!pl.ve.empty()) {
            rfb_set_error("batch scene %zu: a tile halo wraps around a periodic y or z axis", s);
            return -1;
        }
        dims[s] = pl.d;
        for (const SweepItem &it : pl.vi) lists[0].push_back(BatchItem{(int)s, it});
        for (const SweepItem &it : pl.vx) lists[1].push_back(BatchItem{(int)s, it});
        for (const SweepItem &it : pl.vq) lists[2].push_back(BatchItem{(int)s, it});
        if (build_tma_maps(e, tj) != 0) return -1;
        maps[0][s] = e->tmaps[0];
        maps[1][s] = e->tmaps[1];
    }
    if (uni) {
        // one queue for every item (interior sub 5, x slab sub 6)
        for (BatchItem it : lists[0]) it.t.sub = 5, lists[2].push_back(it);
        for (BatchItem it : lists[1]) it.t.sub = 6, lists[2].push_back(it);
        lists[0].clear();
        lists[1].clear();
    }
    for (int k = 0; k < 3; k++) {
        // costliest items first across the whole batch (a slab or boundary
        // plane costs about four interior planes); among equal costs, items
        // of one body together, so that the SMs run few bodies at a time
        // (fewer instruction-fetch stalls: 4 % faster on C4)
        auto cost = [](const BatchItem &x) { return (x.t.ie - x.t.ib) * (x.t.sub == 5 ? 1 : 4); };
        std::stable_sort(lists[k].begin(), lists[k].end(), [&](const BatchItem &x, const BatchItem &y) {
            if (cost(x) != cost(y)) return cost(x) > cost(y);
            return x.t.sub < y.t.sub;
        });
        b->n_items[k] = (int)lists[k].size();
        if (b->n_items[k]) {
            CK(dmalloc(&b->d_items[k], lists[k].size() * sizeof(BatchItem)));
            CK(cudaMemcpy(b->d_items[k], lists[k].data(), lists[k].size() * sizeof(BatchItem),
                          cudaMemcpyHostToDevice));
        }
    }
    CK(dmalloc(&b->d_dims, n * sizeof(FusedDims)));
    CK(cudaMemcpy(b->d_dims, dims.data(), n * sizeof(FusedDims), cudaMemcpyHostToDevice));
    for (int q = 0; q < 2; q++) {
        CK(dmalloc(&b->d_maps[q], n * sizeof(TmaMaps)));
        CK(cudaMemcpy(b->d_maps[q], maps[q].data(), n * sizeof(TmaMaps), cudaMemcpyHostToDevice));
    }
    return 0;
fail:
    return -1;
}

template <typename T>
static void batch_sweep(rfb_batch *b, int par) {
    const Args<T> *args = (const Args<T> *)b->d_args[par];
    if (b->mode == 5) {
        v_launch_b<T>(args, b->d_vshapes, b->d_vmaps[par], b->d_vitems, b->n_vitems, b->v_nt, b->v_smem, b->d_err,
                      b->stream, b->overlap);
        return;
    }
    const TmaMaps *maps = b->d_maps[par];
    if (b->uni) {
        launch_qb<5, T>(args, b->d_dims, maps, b->tj, b->ns, b->d_items[2], b->n_items[2], b->d_queue + 2, b->d_err,
                        b->stream);
        return;
    }
    cudaEventRecord(b->ev_fork, b->stream);
    cudaStreamWaitEvent(b->stream2, b->ev_fork, 0);
    launch_qb<0, T>(args, b->d_dims, maps, b->tj, b->ns, b->d_items[0], b->n_items[0], b->d_queue, b->d_err,
                    b->stream);
    launch_qb<1, T>(args, b->d_dims, maps, b->tj, b->ns, b->d_items[1], b->n_items[1], b->d_queue + 4, b->d_err,
                    b->stream);
    launch_qb<2, T>(args, b->d_dims, maps, b->tj, b->ns, b->d_items[2], b->n_items[2], b->d_queue + 2, b->d_err,
                    b->stream2);
    cudaEventRecord(b->ev_join, b->stream2);
    cudaStreamWaitEvent(b->stream, b->ev_join, 0);
}

template <typename T>
static void batch_rest(rfb_batch *b, int par) {
    if (b->n_lblocks)
        launch_step(k_e_list_b<T>, dim3(b->n_lblocks), dim3(256), 0, b->stream, b->overlap,
                    (const Args<T> *)b->d_args[par], b->d_lblocks);
    launch_step(k_probe_gather_b<T>, dim3(1), dim3(1024), 0, b->stream, b->overlap,
                (const ProbeRefB<T> *)b->d_probes, b->n_probes, 1 - par, (long long)b->n_steps, b->d_step);
}

static int batch_launches_per_step(const rfb_batch *b) {
    const int sweep = b->mode == 5 ? 1 : (b->n_items[0] > 0) + (b->n_items[1] > 0) + (b->n_items[2] > 0);
    return sweep + (b->n_lblocks > 0) + 1;
}

static void batch_enqueue_step(rfb_batch *b, int par) {
    if (b->prec == RFB_FP64) {
        batch_sweep<double>(b, par);
        batch_rest<double>(b, par);
    } else {
        batch_sweep<float>(b, par);
        batch_rest<float>(b, par);
    }
}

static int batch_graph(rfb_batch *b, int par, int steps, cudaGraphExec_t *out) {
    cudaGraph_t graph = nullptr;
    int p = par;
    CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    b->overlap = b->mode == 5 && b->cells <= (1 << 21) && 3 * b->list_cells <= (1 << 17);  // as overlap_pays
    for (int s = 0; s < steps; s++) {
        batch_enqueue_step(b, p);
        p ^= 1;
    }
    b->overlap = false;
    CK(cudaStreamEndCapture(b->stream, &graph));
    CK(cudaGraphInstantiate(out, graph, 0));
    cudaGraphDestroy(graph);
    return 0;
fail:
    if (graph) cudaGraphDestroy(graph);
    return -1;
}

extern "C" int rfb_batch_reset(rfb_batch_t *b) {
    for (rfb_engine *e : b->m)
        if (rfb_engine_reset(e) != 0) return -1;
    CK(cudaMemsetAsync(b->d_step, 0, sizeof(int), b->stream));
    b->steps_done = 0;
    b->parity = 0;
    return 0;
fail:
    return -1;
}

// A work-queue plan, where every scene is within its sweep's limits.
static int batch_queue_plan(rfb_batch *b, int tj, int ns, int mode, int seg_int, int seg_edge, int uni) {
    if (qb_prepare() != 0) {
        rfb_set_error("cannot configure the batched sweep kernels' shared memory");
        return -1;
    }
    for (size_t s = 0; s < b->m.size(); s++)
        if (!q_fits(b->m[s])) {
            rfb_set_error("batch scene %zu too large for the work-queue sweep (32-bit offsets)", s);
            return -1;
        }
    return batch_build_plan(b, tj, ns, mode, seg_int, seg_edge, uni);
}

// The plan: mode 5 by rule, or the one RFSYN_FDTD_PLAN names -- a work-queue
// sweep, or "threads,stages,seg_interior,seg_edge,5".  A batch with a scene
// past the vector sweep's limits (v_fits: psi arrays of 2^32 bytes, planes of
// 2^29) runs on the work-queue sweep, whose limits are wider (q_fits: 2^31
// elements), by the plan that timing picked for most batches before the vector
// sweep.  Every plan computes bit-identical fields.
static int batch_plan(rfb_batch *b) {
    const char *ov = rfb_plan_override();
    if (!ov) {
        // (a periodic y or z axis is refused by either)
        const bool fits = std::all_of(b->m.begin(), b->m.end(),
                                      [](const rfb_engine *e) { return (e->g.periodic & 6u) || v_fits(e); });
        if (fits) return batch_build_vplan(b, V_BATCH_NT, 0, 0);
        const InteriorVariant v = b->prec == RFB_FP32 ? kQVariantsFp32[0] : kQVariantsFp64[0];
        return batch_queue_plan(b, v.tj, v.ns, 4, 64, 32, 0);
    }
    int a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0, a6 = 0;
    const int nov = sscanf(ov, "%d,%d,%d,%d,%d,%d", &a1, &a2, &a3, &a4, &a5, &a6);
    if (nov >= 5 && a5 == 5 && a2 == V_NH && a3 > 0 && a4 > 0 && a6 >= 0 && a6 <= 1 && a1 >= 32 && a1 <= V_NT && a1 % 32 == 0)
        return batch_build_vplan(b, a1, a3, a4);
    if (nov < 5 || a5 < 2 || a5 > 4 || a3 <= 0 || a4 <= 0 || a6 < 0 || a6 > 1 ||
        !plan_variant_known(b->prec, a1, a2, a5)) {
        rfb_set_error("sweep plan \"%s\" names no work-queue or vector sweep variant", ov);
        return -1;
    }
    return batch_queue_plan(b, a1, a2, a5, a3, a4, a6);
}

extern "C" void rfb_batch_destroy(rfb_batch_t *b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    batch_free_plan(b);
    for (rfb_engine *e : b->m) rfb_engine_destroy(e);
    dfree(b->d_step); dfree(b->d_err); dfree(b->d_queue);
    dfree(b->d_args[0]); dfree(b->d_args[1]);
    dfree(b->d_lblocks); dfree(b->d_probes);
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->ev_join) cudaEventDestroy(b->ev_join);
    if (b->stream2) cudaStreamDestroy(b->stream2);
    if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

template <typename T>
static int batch_upload_args(rfb_batch *b) {
    const size_t n = b->m.size();
    std::vector<Args<T>> a[2];
    std::vector<ProbeRefB<T>> probes;
    std::vector<int2> lblocks;
    for (int par = 0; par < 2; par++) {
        a[par].resize(n);
        for (size_t s = 0; s < n; s++) {
            a[par][s] = engine_args<T>(b->m[s], par);
            a[par][s].d_step = b->d_step;
        }
        CK(dmalloc(&b->d_args[par], n * sizeof(Args<T>)));
        CK(cudaMemcpy(b->d_args[par], a[par].data(), n * sizeof(Args<T>), cudaMemcpyHostToDevice));
    }
    for (size_t s = 0; s < n; s++) {
        rfb_engine *e = b->m[s];
        const int ne = 3 * e->scene.n_cells;
        for (int e0 = 0; e0 < ne; e0 += 256) lblocks.push_back(make_int2((int)s, e0));
        std::vector<long long> cell(e->n_probes);
        std::vector<int> comp(e->n_probes);
        if (e->n_probes) {
            CK(cudaMemcpy(cell.data(), e->probe_cell, e->n_probes * sizeof(long long), cudaMemcpyDeviceToHost));
            CK(cudaMemcpy(comp.data(), e->probe_comp, e->n_probes * sizeof(int), cudaMemcpyDeviceToHost));
        }
        for (int q = 0; q < e->n_probes; q++) {
            ProbeRefB<T> r;
            r.f[0] = (const T *)e->fld[0][comp[q]];
            r.f[1] = (const T *)e->fld[1][comp[q]];
            r.cell = cell[q];
            r.ts = (T *)e->ts + (size_t)q * e->n_steps;
            probes.push_back(r);
        }
    }
    b->n_lblocks = (int)lblocks.size();
    if (b->n_lblocks) {
        CK(dmalloc(&b->d_lblocks, lblocks.size() * sizeof(int2)));
        CK(cudaMemcpy(b->d_lblocks, lblocks.data(), lblocks.size() * sizeof(int2), cudaMemcpyHostToDevice));
    }
    b->n_probes = (int)probes.size();
    if (b->n_probes) {
        CK(dmalloc(&b->d_probes, probes.size() * sizeof(ProbeRefB<T>)));
        CK(cudaMemcpy(b->d_probes, probes.data(), probes.size() * sizeof(ProbeRefB<T>), cudaMemcpyHostToDevice));
    }
    return 0;
fail:
    return -1;
}

extern "C" void *rfb_stream_create(void) {
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
        rfb_set_error("cannot create a CUDA stream");
        return nullptr;
    }
    return (void *)st;
}
extern "C" void rfb_stream_destroy(void *stream) {
    if (stream) cudaStreamDestroy((cudaStream_t)stream);
}

extern "C" rfb_batch_t *rfb_batch_create(rfb_engine_t **members, size_t n, void *stream, int own_stream) {
    rfb_batch *b = new rfb_batch();
    b->stream = (cudaStream_t)stream;
    b->own_stream = own_stream;
    for (size_t s = 0; s < n; s++) b->m.push_back(members[s]);
    if (n == 0) {
        rfb_set_error("a batch needs at least one scene");
        goto fail;
    }
    b->prec = members[0]->prec;
    b->n_steps = members[0]->n_steps;
    for (size_t s = 0; s < n; s++) {
        rfb_engine *e = members[s];
        if (!e->member || e->prec != b->prec || e->n_steps != b->n_steps || e->nbuf != 2) {
            rfb_set_error("batch scene %zu: scenes must be batch members of one precision and step count", s);
            goto fail;
        }
        b->cells += (size_t)e->g.nx * e->g.ny * e->g.nz;
        b->list_cells += (size_t)e->scene.n_cells;
        if (e->cpml.on) {
            const int nn[3] = {e->g.nx, e->g.ny, e->g.nz};
            for (int a = 0; a < 3; a++)
                b->slab_cell_axes += (size_t)e->cpml.eh[a].ns * ((size_t)e->g.nx * e->g.ny * e->g.nz / nn[a]);
        }
    }
    if (!b->stream) {
        rfb_set_error("a batch needs the stream its scenes were created on");
        goto fail;
    }
    CK(cudaStreamCreateWithFlags(&b->stream2, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming));
    CK(dmalloc(&b->d_step, sizeof(int)));
    CK(cudaMemset(b->d_step, 0, sizeof(int)));
    CK(dmalloc(&b->d_err, sizeof(int)));
    CK(cudaMemset(b->d_err, 0, sizeof(int)));
    CK(dmalloc(&b->d_queue, 6 * sizeof(int)));
    CK(cudaMemset(b->d_queue, 0, 6 * sizeof(int)));
    if ((b->prec == RFB_FP64 ? batch_upload_args<double>(b) : batch_upload_args<float>(b)) != 0) goto fail;
    CK(cudaDeviceSynchronize());
    {
        const double t_plan = rfb_now();
        const int rc = batch_plan(b);
        rfb_trace("batch: plan", t_plan);
        if (rc != 0) goto fail;
    }
    return b;
fail:
    rfb_batch_destroy(b);
    return nullptr;
}

static int batch_report(int err) {
    if (err) {
        rfb_set_error("batch: %s", sweep_error_text(err));
        return -1;
    }
    return 0;
}

static int batch_check_error(rfb_batch *b) {
    int err = 0;
    if (cudaMemcpy(&err, b->d_err, sizeof err, cudaMemcpyDeviceToHost) != cudaSuccess) {
        rfb_set_error("batch: %s", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    return batch_report(err);
}

extern "C" int rfb_batch_advance(rfb_batch_t *b, size_t n) {
    if (b->steps_done + n > b->n_steps) {
        rfb_set_error("advance past the configured step count (%zu + %zu > %zu)", b->steps_done, n, b->n_steps);
        return -1;
    }
    const int lps = batch_launches_per_step(b);
    while (n > 0) {
        const int par = b->parity;
        if (n >= (size_t)rfb_batch::CHUNK) {
            if (!b->gk[par] && batch_graph(b, par, rfb_batch::CHUNK, &b->gk[par]) != 0) return -1;
            CK(cudaGraphLaunch(b->gk[par], b->stream));
            g_launches += (unsigned long long)rfb_batch::CHUNK * lps;
            n -= rfb_batch::CHUNK;
            b->steps_done += rfb_batch::CHUNK;
        } else {
            if (!b->g1[par] && batch_graph(b, par, 1, &b->g1[par]) != 0) return -1;
            CK(cudaGraphLaunch(b->g1[par], b->stream));
            g_launches += lps;
            n -= 1;
            b->steps_done += 1;
            b->parity ^= 1;
        }
    }
    for (rfb_engine *e : b->m) {
        e->steps_done = b->steps_done;
        e->parity = b->parity;
    }
    return 0;
fail:
    return -1;
}

extern "C" int rfb_batch_sync(rfb_batch_t *b) {
    int err = 0;  // comes back behind the stream's work
    CK(cudaMemcpyAsync(&err, b->d_err, sizeof err, cudaMemcpyDeviceToHost, b->stream));
    CK(cudaStreamSynchronize(b->stream));
    return batch_report(err);
fail:
    return -1;
}

// A scene's series: the batch's sweeps are the only ones that ran on it, so
// the batch's wait and check cover it.
extern "C" int rfb_batch_read_probes(rfb_batch_t *b, size_t scene, double *out) {
    if (rfb_batch_sync(b) != 0) return -1;
    return copy_series(b->m[scene], out);
}

extern "C" int rfb_batch_advance_timed(rfb_batch_t *b, size_t n, double *ms) {
    cudaEvent_t a = nullptr, c = nullptr;
    float t = 0.f;
    int rc = -1;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&c));
    CK(cudaEventRecord(a, b->stream));
    if (rfb_batch_advance(b, n) != 0) goto out;
    CK(cudaEventRecord(c, b->stream));
    CK(cudaEventSynchronize(c));
    CK(cudaEventElapsedTime(&t, a, c));
    if (ms) *ms = t;
    rc = batch_check_error(b);
    goto out;
fail:
out:
    if (a) cudaEventDestroy(a);
    if (c) cudaEventDestroy(c);
    return rc;
}

// Runs n more steps launching each kernel separately (no graph) with events
// around the sweep and around the rest, to attribute GPU time.
extern "C" int rfb_batch_time_kernels(rfb_batch_t *b, size_t n, double *sweep_ms, double *other_ms) {
    cudaEvent_t ev[3] = {};
    double sw = 0.0, ot = 0.0;
    int rc = -1;
    if (b->steps_done + n > b->n_steps) {
        rfb_set_error("advance past the configured step count");
        return -1;
    }
    for (int q = 0; q < 3; q++) CK(cudaEventCreate(&ev[q]));
    for (size_t s = 0; s < n; s++) {
        const int par = b->parity;
        CK(cudaEventRecord(ev[0], b->stream));
        if (b->prec == RFB_FP64) batch_sweep<double>(b, par);
        else batch_sweep<float>(b, par);
        CK(cudaEventRecord(ev[1], b->stream));
        if (b->prec == RFB_FP64) batch_rest<double>(b, par);
        else batch_rest<float>(b, par);
        CK(cudaEventRecord(ev[2], b->stream));
        CK(cudaEventSynchronize(ev[2]));
        float a = 0.f, c = 0.f;
        CK(cudaEventElapsedTime(&a, ev[0], ev[1]));
        CK(cudaEventElapsedTime(&c, ev[1], ev[2]));
        sw += a;
        ot += c;
        g_launches += batch_launches_per_step(b);
        b->steps_done++;
        b->parity ^= 1;
    }
    for (rfb_engine *e : b->m) {
        e->steps_done = b->steps_done;
        e->parity = b->parity;
    }
    *sweep_ms = sw;
    *other_ms = ot;
    rc = batch_check_error(b);
fail:
    for (int q = 0; q < 3; q++)
        if (ev[q]) cudaEventDestroy(ev[q]);
    return rc;
}

extern "C" rfb_engine_t *rfb_batch_member(rfb_batch_t *b, size_t s) {
    return s < b->m.size() ? b->m[s] : nullptr;
}
extern "C" size_t rfb_batch_size(rfb_batch_t *b) { return b->m.size(); }
extern "C" size_t rfb_batch_steps_done(rfb_batch_t *b) { return b->steps_done; }
extern "C" void *rfb_batch_stream(rfb_batch_t *b) { return (void *)b->stream; }

extern "C" int rfb_batch_info(rfb_batch_t *b, rfb_batch_info_t *out) {
    out->scenes = b->m.size();
    out->cells = b->cells;
    out->list_cells = b->list_cells;
    out->slab_cell_axes = b->slab_cell_axes;
    out->tile_j = b->tj;
    out->ring_depth = b->ns;
    out->mode = b->mode;
    out->unified = b->uni;
    out->seg_interior = b->seg_int;
    out->seg_edge = b->seg_edge;
    out->items_interior = b->mode == 5 ? b->n_vplain : b->n_items[0];
    out->items_xslab = b->n_items[1];
    out->items_edge = b->mode == 5 ? b->n_vitems - b->n_vplain : b->n_items[2];
    out->launches_per_step = batch_launches_per_step(b);
    return 0;
}
