// dem_steps.cuh -- many steps of a small world in one kernel.
//
// A launch a step costs a small world more than the step: at 16,384 bonded
// particles the Simulation kernel's chain of dependent loads, restarted from
// a cold L1 in every launch, takes ~12 us, the graph's conditional node and
// the launch ~4 us more, for ~1 us of arithmetic.  Here one thread owns one
// particle for the whole run: its state stays in registers, its contact
// slots and candidate list in shared memory, and a step costs one gather of
// the partners' records from L2 and one barrier over the grid.  The grid is
// at most one block per SM, launched cooperatively, so every block is
// resident while it waits; up to 4,096 particles it is one cluster, whose
// blocks read each other's records in shared memory.
//
// A particle that moves beyond its candidate list has all lists rebuilt, most
// often within the run (rebuild_lists).  A run ends when the call's steps are
// done, or for the rebuild that also reorders the particle arrays; the graph
// around it (World::capture_run) then runs that rebuild and starts the kernel
// again for the remaining steps.
//
// The step itself is interact_particle and lom_core of dem_kernels.cu, with
// the particle's state behind ResidentOwn instead of HbmOwn: the same
// expressions in the same order, so the results are the same bit for bit.
#pragma once
#define DEM_STEP_DEVICE_CODE
#include "dem_kernels.cu"

#include <climits>

namespace demgb {

// A wait for the other blocks gives up after this many clock cycles (about
// two seconds; a step takes microseconds), sets device error 8 and ends the run.
// (The host reads that word where it waits: a store to host memory here, never
// reached, made every step ~70 ns slower, 1.5 % of a small world's.)
constexpr long long WAIT_CYCLES = 4000000000LL;

// shared memory of a block of TB threads, in words a thread: 5 fields of 14
// slots, the candidate list, the narrow phase's two partner arrays
constexpr int SLOT_WORDS = 5 * K, LIST_WORDS = 8, PARTNER_WORDS = 2 * K;
constexpr int STEP_WORDS = SLOT_WORDS + LIST_WORDS + PARTNER_WORDS;

constexpr uint32_t F_MOVED = 1u, F_BROKE = 2u;  // a block's report at the barrier
constexpr uint32_t F_FAILED = 4u;               // and: a wait gave up

// Every particle in the cells around a position at the rebuild numbered
// `links`, from the cells' chains: visit(b, its record).
// AT_ONCE cells at a time, whose records (read(b)) are in flight together.
template <int AT_ONCE, class Read, class Visit>
__device__ __forceinline__ void walk_cells(const DevWorld &w, Read read, const ScenePar &G, float2 at,
                                           uint32_t number, Visit visit) {
    int gx, gy;
    search_xy(G, at.x, at.y, gx, gy);
    const int cy0 = max(gy - G.stencil, 0), cx0 = max(gx - G.stencil, 0);
    const int wide = min(gx + G.stencil, G.g_w - 1) - cx0 + 1;
    const int cells = wide * (min(gy + G.stencil, G.g_h - 1) - cy0 + 1);
    for (int c0 = 0; c0 < cells; c0 += AT_ONCE) {
        int b[AT_ONCE];
#pragma unroll
        for (int q = 0; q < AT_ONCE; ++q) {
            b[q] = -1;
            if (c0 + q < cells) {
                const int y = (c0 + q) / wide, x = c0 + q - y * wide;
                const unsigned long long h = __ldcg(&w.cell_head[G.cell_base + (cy0 + y) * G.g_w + cx0 + x]);
                if ((uint32_t)(h >> 32) == number) b[q] = (int)(uint32_t)h;
            }
        }
        bool any = true;
        while (any) {
            float4 pb[AT_ONCE];
            int next[AT_ONCE];
#pragma unroll
            for (int q = 0; q < AT_ONCE; ++q)
                if (b[q] >= 0) {
                    pb[q] = read(b[q]);
                    next[q] = __ldcg(w.cell_next + b[q]);
                }
            any = false;
#pragma unroll
            for (int q = 0; q < AT_ONCE; ++q)
                if (b[q] >= 0) {
                    visit(b[q], pb[q]);
                    b[q] = next[q];
                    any |= b[q] >= 0;
                }
        }
    }
}

// A world that one cluster of blocks holds keeps its position and displacement
// records in the blocks' shared memory: particle b is entry b mod TB of block
// b / TB, read through the cluster's shared address space.
__device__ __forceinline__ float4 ld_cluster(const float4 *mine, int rank) {
    uint32_t at = (uint32_t)__cvta_generic_to_shared(mine);
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(at) : "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(at));  // volatile: stays between the barriers, which clobber memory
    return v;
}
__device__ __forceinline__ void or_cluster(uint32_t *mine, int rank, uint32_t bits) {
    uint32_t at = (uint32_t)__cvta_generic_to_shared(mine);
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(at) : "r"(rank));
    asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(at), "r"(bits) : "memory");
}
// every thread of the cluster's blocks; orders shared and global memory among them
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Partner records are written by other blocks during the run: they are read
// through L2 (ld.cg), never through the read-only path, or (CLU) from the
// cluster's shared memory.
template <int TB, bool CLU>
struct ResidentOwn {
    static constexpr bool RESIDENT = true;
    uint32_t m, mask, cm, touched, flags;
    uint64_t cand;  // candidate number of each slot's partner, while cm is not stale
    float4 pa, v, da, half;  // half: data[4..6]
    float2 b0, kns;
    float rho;
    int i, N, own_mat, rec_row;
    int left_run;   // steps the scene has left, 1 at the call's last step
    bool act, det;
    unsigned lanes;  // the warp's lanes that take this step with a radius
    uint32_t links;  // number of the rebuild whose cell chains hold, 0: the cell table does
    long long now;
    int32_t *sl;    // the thread's column of the slot words
    const int4 *nl;
    // the step's and the next one's records: CLU, the block's arrays in shared
    // memory, indexed by thread; else the world's
    const float4 *cur, *dcur;
    float4 *nxt, *dnxt;
    float *rec_out;
    const ScenePar &par;

    __device__ __forceinline__ ResidentOwn(const ScenePar &P) : par(P) {}
    __device__ __forceinline__ const ScenePar &scene(const DevWorld &, int) const { return par; }
    __device__ __forceinline__ bool acts(const DevWorld &, int) const { return act; }
    __device__ __forceinline__ bool detects(const DevWorld &, int) const { return det; }
    __device__ __forceinline__ long long left(const DevWorld &, int) const { return left_run; }
    __device__ __forceinline__ long long step(const DevWorld &) const { return now; }
    __device__ __forceinline__ int4 list(const DevWorld &, int h) const { return nl[h * TB]; }
    __device__ __forceinline__ uint32_t match(const DevWorld &) const { return cm; }
    __device__ __forceinline__ void set_match(const DevWorld &, uint32_t c) { cm = c; }
    __device__ __forceinline__ uint64_t slot_candidates() const { return cand; }
    __device__ __forceinline__ void set_slot_candidates(uint64_t at) { cand = at; }

    __device__ __forceinline__ int32_t &word(int f, int j) const { return sl[(f * K + j) * TB]; }
    __device__ __forceinline__ int slot_b(const DevWorld &, int j) const { return word(0, j); }
    __device__ __forceinline__ int slot_bonded(const DevWorld &, int j) const { return word(1, j); }
    __device__ __forceinline__ float slot_tf(const DevWorld &, int j) const { return __int_as_float(word(2, j)); }
    __device__ __forceinline__ float slot_btf(const DevWorld &, int j) const { return __int_as_float(word(3, j)); }
    __device__ __forceinline__ float slot_thb(const DevWorld &, int j) const { return __int_as_float(word(4, j)); }
    // every slot at the start of a run, so that none is waited for within it:
    // an empty one for the fields that a new contact inherits
    __device__ __forceinline__ void fetch_slots(const DevWorld &w) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const size_t at = (size_t)j * N + i;
            if ((mask >> j) & 1u) {
                word(0, j) = w.s_b[at];
                word(2, j) = __float_as_int(w.s_tf[at]);
            }
            word(1, j) = w.s_bonded[at];
            word(3, j) = __float_as_int(w.s_btf[at]);
            word(4, j) = __float_as_int(w.s_thb[at]);
        }
        touched = mask & SLOT_BITS;
    }
    __device__ __forceinline__ void new_slot(const DevWorld &, int j, int b) {
        touched |= 1u << j;
        word(0, j) = b;
        word(2, j) = 0;
    }
    __device__ __forceinline__ void set_bonded(const DevWorld &, int j, int x) { word(1, j) = x; }
    __device__ __forceinline__ void set_tf(const DevWorld &, int j, float x) { word(2, j) = __float_as_int(x); }
    __device__ __forceinline__ void set_btf(const DevWorld &, int j, float x) { word(3, j) = __float_as_int(x); }
    __device__ __forceinline__ void set_thb(const DevWorld &, int j, float x) { word(4, j) = __float_as_int(x); }
    __device__ __forceinline__ void set_mask(const DevWorld &, uint32_t x, uint32_t) { mask = x; }

    __device__ __forceinline__ float4 record_of(const float4 *a, int b) const {
        return CLU ? ld_cluster(a + (b & (TB - 1)), b / TB) : __ldcg(a + b);
    }
    __device__ __forceinline__ int own() const { return CLU ? (int)threadIdx.x : i; }
    __device__ __forceinline__ float4 partner(const DevWorld &, int b) const { return record_of(cur, b); }
    __device__ __forceinline__ uint32_t partner_range(const DevWorld &, int b) const {
        return __float_as_uint(CLU ? record_of(cur, b).w : __ldcg(reinterpret_cast<const float *>(cur + b) + 3));
    }
    __device__ __forceinline__ float4 partner_disp(const DevWorld &, int b) const { return record_of(dcur, b); }
    __device__ __forceinline__ int bond_status(const DevWorld &w, int g) const { return __ldcg(w.b_status + g); }
    __device__ __forceinline__ void broke() { flags |= F_BROKE; }
    __device__ __forceinline__ unsigned lanes_of_step() const { return lanes; }
    __device__ __forceinline__ float2 stiffness(const DevWorld &w, int n_mat, int at) const {
        return n_mat == 1 ? kns : __ldg(&w.pair[at]);
    }
    __device__ __forceinline__ float density(const DevWorld &w, int at) const {
        return at == own_mat ? rho : w.mats[at].density;
    }
    __device__ __forceinline__ float4 external(const DevWorld &w) const { return __ldg(&w.fx[i]); }
    __device__ __forceinline__ float4 disp(const DevWorld &) const { return da; }
    __device__ __forceinline__ float4 vel(const DevWorld &) const { return v; }
    __device__ __forceinline__ float2 rebuilt_at(const DevWorld &) const { return b0; }
    __device__ __forceinline__ void set_vel(const DevWorld &, float4 x) { v = x; }
    __device__ __forceinline__ void advance(const DevWorld &w, float4 p, float4 vel, float4 d, float4 d4, bool moved,
                                            bool) {
        half = d4;
        nxt[own()] = p;
        dnxt[own()] = d;
        pa = p;
        v = vel;
        da = d;
        if (moved) flags |= F_MOVED;
    }
    __device__ __forceinline__ void stay(const DevWorld &) {
        nxt[own()] = pa;
        dnxt[own()] = da;
    }
    // a particle whose candidates exceed its list goes over its cells
    template <int ST>
    __device__ __forceinline__ bool search_cells(const DevWorld &w, int s, Narrow<ST> &nr) const {
        if (links == 0u) return false;
        walk_cells<TB <= 256 ? 9 : 3>(w, [&](int b) { return record_of(cur, b); }, w.par[s], b0, links,
                                      [&](int b, float4) { narrow_test(w, i, b, *this, nr); });
        return true;
    }
    // the datum of this step (k_gather_datum's row) of a recorded particle
    __device__ __forceinline__ void record(const DevWorld &w, float4 p, float rot, float d0, float d1, float d2) {
        if (rec_row < 0) return;
        float *o = rec_out + 10 * (size_t)rec_row;
        o[0] = p.x;
        o[1] = p.y;
        o[2] = half.x;
        o[3] = half.y;
        o[4] = rot;
        o[5] = half.z;
        o[6] = d0;
        o[7] = d1;
        o[8] = d2;
        o[9] = w.data3[w.run->rec_base + w.orig[i]];
    }
};

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_add(uint32_t *p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// waits until the word's bits `mask` are `want`; the word, or WAIT_FAILED
constexpr uint32_t WAIT_FAILED = ~0u;
__device__ __forceinline__ uint32_t wait_for(const uint32_t *p, uint32_t mask, uint32_t want, StepRun &R, int32_t *err) {
    uint32_t v;
    const long long t0 = clock64();
    do {
        for (int tries = 0; tries < 256; ++tries)
            if (((v = ld_relaxed(p)) & mask) == want) return v;
    } while (clock64() - t0 < WAIT_CYCLES && ld_relaxed(&R.fail) == 0u);
    atomicOr(err, 8);
    st_relaxed(&R.fail, 1u);
    return WAIT_FAILED;
}

// Breaks of the step become visible to the partners (status = min code), as
// end_of_step applies them; by the threads of one block.
__device__ inline void apply_breaks(const DevWorld &w) {
    uint32_t n = *(volatile uint32_t *)w.pend_count;
    if (n > w.pend_cap) n = w.pend_cap;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
        const int2 q = __ldcg(reinterpret_cast<const int2 *>(w.pend) + k);
        atomicMin(&w.b_status[q.x], q.y);
    }
    fence_gpu();
    __syncthreads();
    if (threadIdx.x == 0) *w.pend_count = 0u;
}
static_assert(sizeof(Pending) == sizeof(int2), "a pending break is read as one int2");

// The scenes' words after `done` steps of a run, by the threads of one block.
__device__ inline void end_of_run(const DevWorld &w, long long step0, int done, bool last, bool due, int inner,
                           uint32_t links, bool reorder, cudaGraphConditionalHandle more, cudaGraphConditionalHandle rebuild) {
    const long long next = step0 + done;
    for (int s = threadIdx.x; s < w.S && done > 0; s += blockDim.x) {
        w.cc3[s] = 0;
        const ScenePar &P = w.par[s];
        w.det[s] = detect_at(P.p.collision_interval, P.cc1_0, next - P.step0) ? 1 : 0;
        if (w.act[s]) {
            const long long left = w.remaining[s] - done;
            w.remaining[s] = left > 0 ? left : 0;
            if (left <= 0) w.act[s] = 0;  // a served scene stops at its horizon
        }
    }
    if (threadIdx.x == 0) {
        StepRun &R = *w.run;
        *w.step = next;
        R.todo -= done;
        R.done += done;
        R.lom_done = last ? 0 : 1;
        if (inner || due) *w.rebuild = due ? 1 : 0;
        if (inner) {
            w.stats[4] += (unsigned)inner;
            *w.reorder = reorder ? 1 : 0;
            R.links = links;
            R.linked = 1;
        }
        cudaGraphSetConditional(more, last ? 0u : 1u);
        cudaGraphSetConditional(rebuild, due ? 1u : 0u);
    }
}

// What a block knows of a run, and its meetings with the others (CLU: those of
// its cluster, which is the grid).
template <bool CLU>
struct Run {
    const DevWorld &w;
    StepRun &R;
    uint32_t *s_any;  // three words in shared memory
    const cudaGraphConditionalHandle more, rebuild;
    const long long step0;
    const unsigned long long rebuilds;
    bool reorder_due;
    uint32_t links;
    uint32_t passed = 0u, turn = 0u;  // barriers of this launch; the word and counter in use
    int inner = 0;                    // rebuilds within this launch

    __device__ __forceinline__ Run(const DevWorld &w_, uint32_t *any, cudaGraphConditionalHandle m,
                                   cudaGraphConditionalHandle r, bool lom_done)
        : w(w_), R(*w_.run), s_any(any), more(m), rebuild(r), step0(*w_.step), rebuilds(w_.stats[4]),
          reorder_due(*w_.reorder != 0), links(w_.run->links) {
        if (threadIdx.x == 0) {
            s_any[0] = (!lom_done && *w.rebuild != 0) ? F_MOVED : 0u;
            s_any[1] = s_any[2] = 0u;
        }
        if (CLU) cluster_barrier();
        else __syncthreads();
    }

    // The barrier over the grid; the blocks' reports together.
    // Every block adds itself and its report to a counter (blocks in bits
    // 0-9, of these moved in 10-19 and broke in 20-29) and one of its threads
    // reads that counter until all are in: a trip to L2 out and one back,
    // where a release by the last block takes two more (152 blocks: 2,440
    // against 3,660 cycles; a flag per block read by all of them 8,000, the
    // readers crowding one line).  Three counters are used in turn: block 0
    // clears one after the barrier behind the one that used it, before it
    // enters the next, so it is clear before any block can use it again.
    // In a cluster the hardware barrier does it, the reports written straight to
    // every block's word: ~400 cycles.
    __device__ __forceinline__ uint32_t meet(uint32_t &flags) {
        if (flags) {
            if (CLU)
                for (unsigned q = 0; q < gridDim.x; ++q) or_cluster(&s_any[turn], (int)q, flags);
            else atomicOr(&s_any[turn], flags);
            flags = 0u;
        }
        ++passed;
        if (CLU) cluster_barrier();
        else __syncthreads();
        const uint32_t now = turn, before = turn == 0u ? 2u : turn - 1u;
        turn = turn == 2u ? 0u : turn + 1u;
        if (!CLU && gridDim.x > 1) {
            if (threadIdx.x == 0) {
                const uint32_t f = s_any[now];
                fence_gpu();
                red_add(&R.arrive[now], 1u + ((f & F_MOVED) ? 1u << 10 : 0u) + ((f & F_BROKE) ? 1u << 20 : 0u));
                const uint32_t all = wait_for(&R.arrive[now], 1023u, gridDim.x, R, w.err);
                fence_gpu();
                if (blockIdx.x == 0) st_relaxed(&R.arrive[before], 0u);
                s_any[now] = all == WAIT_FAILED ? F_FAILED
                                                : ((all >> 10 & 1023u) ? F_MOVED : 0u) | ((all >> 20) ? F_BROKE : 0u);
            }
            __syncthreads();
        }
        const uint32_t word = s_any[now];
        if (threadIdx.x == 0) s_any[before] = 0u;
        return word;
    }

    // After `done` steps: meet the other blocks.  Breaks are applied by block 0
    // while the others wait once more (R.gen); the end of the run needs no
    // wait, nothing that block 0 writes then is read again.  A block whose wait
    // for R.gen gave up goes on to the next barrier: the run has failed, and
    // the host hands out none of its state.  If a particle
    // left its list and this rebuild need not reorder the particles, lists(done)
    // rebuilds them (false: a wait failed).  True when the run ends.
    template <class Lists>
    __device__ __forceinline__ bool step_end(uint32_t &flags, int done, bool last, Lists lists) {
        const uint32_t word = meet(flags);
        const bool failed = (word & F_FAILED) != 0u, due = (word & F_MOVED) != 0u && !last && !failed;
        const bool stop = (due && reorder_due) || last || failed;
        if ((word & F_BROKE) && blockIdx.x == 0) apply_breaks(w);
        if (stop && blockIdx.x == 0)
            end_of_run(w, step0, done, last || failed, due, inner, links, reorder_due, more, rebuild);
        if ((word & F_BROKE) && !stop && CLU) cluster_barrier();
        if ((word & F_BROKE) && !stop && !CLU) {
            __syncthreads();
            if (threadIdx.x == 0 && gridDim.x > 1) {
                if (blockIdx.x == 0) {
                    fence_gpu();
                    st_relaxed(&R.gen, passed);
                } else {
                    wait_for(&R.gen, ~0u, passed, R, w.err);
                    fence_gpu();
                }
            }
            __syncthreads();
        }
        if (stop || !due) return stop;
        ++inner;
        ++links;
        if (!lists(done)) {
            if (blockIdx.x == 0) end_of_run(w, step0, done, true, false, inner, links, false, more, rebuild);
            return true;
        }
        const unsigned long long n = rebuilds + (unsigned)inner;
        reorder_due = w.reorder_every <= 1 || n % (unsigned)w.reorder_every == 0u;
        return false;
    }
};

template <int TB, bool CLU, int FORM, int PS>
__global__ void __launch_bounds__(TB, 1) k_steps(DevWorld w, cudaGraphConditionalHandle more,
                                                 cudaGraphConditionalHandle rebuild,
                                                 const __grid_constant__ ScenePar pv) {
    extern __shared__ __align__(16) int32_t sm[];
    __shared__ uint32_t s_any[3];
    StepRun &R = *w.run;
    const int todo = R.todo;
    const bool lom_done = R.lom_done != 0, failed = R.fail == 1u;
    float *rec_out = R.rec_out == nullptr ? nullptr : R.rec_out + (long long)R.rec_per * R.done;
    const int rec_per = R.rec_per;
    if (failed || todo <= 0) {  // uniform over the grid: no block changes these before all have read them
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            cudaGraphSetConditional(more, 0u);
            cudaGraphSetConditional(rebuild, 0u);
        }
        return;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = i < w.N && chunk_live(w, i);
    const uint32_t m = mine ? w.meta[i] : 0u;
    const int s = (int)meta_scene(m);
    // the fields the step reads stay in registers; the others are never loaded
    ScenePar par;
    if (PS != PS_ONE) par = w.par[s];
    const ScenePar &P = PS == PS_ONE ? pv : par;
    const ScenePar &U = PS == PS_SCENE ? P : pv;

    ResidentOwn<TB, CLU> o(P);
    o.m = m;
    o.i = i;
    o.N = w.N;
    o.sl = sm + threadIdx.x;
    int4 *nl = reinterpret_cast<int4 *>(sm + SLOT_WORDS * TB) + threadIdx.x;
    o.nl = nl;
    // the two buffers of the records: positions at [0] and [1], displacements
    // at [2] and [3] of the block's (CLU), or the world's
    float4 *shared_rec = reinterpret_cast<float4 *>(sm + STEP_WORDS * TB);
    const auto buffer = [&](bool second, bool disp) -> float4 * {
        if (CLU) return shared_rec + ((second ? 1 : 0) + (disp ? 2 : 0)) * TB;
        return disp ? (second ? w.dp_n : w.dp) : (second ? w.pr_n : w.pr);
    };
    o.cur = buffer(false, false);
    o.dcur = buffer(false, true);
    o.nxt = buffer(true, false);
    o.dnxt = buffer(true, true);
    o.mask = o.touched = o.cm = o.flags = 0u;
    o.cand = 0u;
    o.rec_row = -1;
    o.act = o.det = false;
    uint32_t *ck = reinterpret_cast<uint32_t *>(sm + (SLOT_WORDS + LIST_WORDS) * TB) + threadIdx.x;
    Narrow<TB> nr{ck, reinterpret_cast<int *>(ck + K * TB)};
    int left = 0;            // steps until the scene stops, from the run's first
    int until_det = 0, det_every = 1;
    if (mine) {
        const long long rem = w.act[s] ? w.remaining[s] : 0;
        left = rem > INT_MAX ? INT_MAX : (int)rem;
        // steps until the narrow phase runs (detect_at)
        const ScenePar &G = w.par[s];  // a launch's parameters carry no schedule
        det_every = G.p.collision_interval > 1 ? G.p.collision_interval : 1;
        long long j1 = (long long)G.p.collision_interval - 1 - G.cc1_0;
        if (j1 < 0) j1 = 0;
        const long long at = *w.step - G.step0;
        until_det = at < j1 ? (int)(j1 - at) : (int)((det_every - (at - j1) % det_every) % det_every);
        o.pa = w.pr[i];
        o.v = w.vw[i];
        o.da = w.dp[i];
        o.half = w.d4[i];
        o.b0 = w.pbuild[i];
        o.mask = w.smask[i];
        o.cm = CM_STALE;  // the slots' candidate numbers come with the first pass
        nl[0] = w.nl[2 * (size_t)i];
        nl[TB] = w.nl[2 * (size_t)i + 1];
        o.own_mat = P.mat_base + (int)meta_mat(m);
        o.rho = w.mats[o.own_mat].density;
        o.kns = w.pair[P.pair_base];
        o.fetch_slots(w);
        if (R.rec_rows != nullptr && s == R.rec_scene) o.rec_row = R.rec_rows[w.orig[i]];
    }
    if (CLU) {
        buffer(false, false)[threadIdx.x] = mine ? o.pa : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        buffer(false, true)[threadIdx.x] = mine ? o.da : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    o.links = R.linked ? R.links : 0u;
    Run<CLU> run(w, s_any, more, rebuild, lom_done);

    // The lists rebuilt within the run.  Nothing of the result depends on the
    // order of a list's candidates, so the particles are only linked by cell
    // -- a word per cell holds the last particle put in and the rebuild's
    // number, so that no cell is ever cleared -- and each walks the chains of
    // its 3 x 3 (or 5 x 5) cells, nine at a time so that a level of all of
    // them costs one trip to L2.  ~5 us, where leaving the kernel for the
    // sorted rebuild, its 16 launches and the way back takes ~150.
    const auto rebuild_lists = [&](int done) -> bool {
        const uint32_t links = run.links;
        const bool in = mine && left > done && o.pa.z != 0.0f;
        const ScenePar &G = w.par[s];
        o.cur = buffer((done & 1) != 0, false);  // the positions of the step to come
        o.links = links;
        if (in) {
            int cx, cy;
            search_xy(G, o.pa.x, o.pa.y, cx, cy);
            const unsigned long long old = atomicExch(&w.cell_head[G.cell_base + cy * G.g_w + cx],
                                                      (unsigned long long)links << 32 | (unsigned)i);
            w.cell_next[i] = (uint32_t)(old >> 32) == links ? (int32_t)(uint32_t)old : -1;
        }
        if (run.meet(o.flags) & F_FAILED) return false;
        if (mine) {
            int16_t *list = reinterpret_cast<int16_t *>(nl);  // entries 0..7; 8..15 are at nl[TB]
            int cnt = 0, h0 = 0;
            bool over = false;
            o.b0 = make_float2(o.pa.x, o.pa.y);
            if (in) {
                const auto read = [&](int b) { return o.record_of(o.cur, b); };
                walk_cells<TB <= 256 ? 9 : 3>(w, read, G, o.b0, links, [&](int b, float4 pb) {
                    if (b == i || pb.z == 0.0f) return;
                    const float dx = pb.x - o.pa.x, dy = pb.y - o.pa.y;
                    const float t = (o.pa.z + pb.z + G.skin) * 1.00001f;
                    if (dx * dx + dy * dy > t * t) return;
                    const int off = b - i;
                    if (cnt < NL && off >= -32768 && off <= 32767) list[cnt < 7 ? cnt + 1 : 8 * TB + cnt - 7] = (int16_t)off;
                    else over = true;
                    ++cnt;
                });
                h0 = over ? NL_OVERFLOW : cnt;
                if (over) atomicAdd(&w.stats[5], 1ull);
            }
            list[0] = (int16_t)h0;
            o.mask = h0 != 0 ? (o.mask | NL_LIVE) : (o.mask & ~NL_LIVE);
            o.cm = CM_STALE;
        }
        return true;
    };

    bool stop = false;
    if (!lom_done) {  // the first step's LOM pass (k_lom)
        if (left > 0 && o.pa.z != 0.0f) {
            const bool ext = w.cc3[s] != 0;
            float4 d;
            bool moved;
            lom_core(P, U, m, o.pa, o.v, w.ac[i], o.b0, ext, o.da, d, o.half, moved);
            buffer(false, false)[o.own()] = o.pa;
            if (!ext) {
                o.da = d;
                buffer(false, true)[o.own()] = d;
            }
            if (moved) o.flags |= F_MOVED;
        }
        stop = run.step_end(o.flags, 0, false, rebuild_lists);
    }
    for (int k = 0; !stop; ++k) {
        const bool last = k + 1 == todo;
        o.act = left > k;
        o.left_run = last ? 1 : left - k;
        o.det = until_det == 0;
        until_det = until_det == 0 ? det_every - 1 : until_det - 1;
        o.now = run.step0 + k;
        // step k reads the buffers that hold its LOM pass's results
        const bool odd = (k & 1) != 0;
        o.cur = buffer(odd, false);
        o.nxt = buffer(!odd, false);
        o.dcur = buffer(odd, true);
        o.dnxt = buffer(!odd, true);
        o.lanes = __ballot_sync(0xffffffffu, o.act && o.pa.z != 0.0f);
        if (o.act) {
            o.rec_out = rec_out + (long long)rec_per * k;
            interact_particle<0, true, FORM, PS>(w, i, o, nr, true, pv);
        }
        stop = run.step_end(o.flags, k + 1, last, rebuild_lists);
    }
    // The particle's state back to device memory, in the buffers that are
    // current between runs (no block reads a partner's record any more).
    if (mine) {
        w.pr[i] = o.pa;
        w.dp[i] = o.da;
        if (CLU) {  // a scene that never steps again reads the same from either
            w.pr_n[i] = o.pa;
            w.dp_n[i] = o.da;
        }
        w.vw[i] = o.v;
        w.d4[i] = o.half;
        w.smask[i] = o.mask;
        w.cmask[i] = o.cm;
        if (run.inner) {
            w.pbuild[i] = o.b0;
            w.nl[2 * (size_t)i] = nl[0];
            w.nl[2 * (size_t)i + 1] = nl[TB];
        }
        const int N = w.N;
        for (uint32_t q = o.touched; q; q &= q - 1) {
            const int j = __ffs(q) - 1;
            w.s_b[j * N + i] = o.word(0, j);
            w.s_bonded[j * N + i] = o.word(1, j);
            w.s_tf[j * N + i] = __int_as_float(o.word(2, j));
            w.s_btf[j * N + i] = __int_as_float(o.word(3, j));
            w.s_thb[j * N + i] = __int_as_float(o.word(4, j));
        }
    }
}

// A particle of a swept world: its state stays in device memory between
// steps, as HbmOwn's does between launches, and its partners' records are
// read through L2.
struct SweptOwn : HbmOwn<0, true> {
    const float4 *cur, *dcur;
    float4 *nxt, *dnxt;
    uint32_t &flags;
    uint32_t links;
    bool act, det;
    int left_run;
    long long now;
    __device__ __forceinline__ SweptOwn(const DevWorld &w, int i_, const float4 *pr, const float4 *dp, float4 *pr_n,
                                        float4 *dp_n, uint32_t &f)
        : HbmOwn<0, true>(w, i_, pr, dp), cur(pr), dcur(dp), nxt(pr_n), dnxt(dp_n), flags(f) {}
    __device__ __forceinline__ bool acts(const DevWorld &, int) const { return act; }
    __device__ __forceinline__ bool detects(const DevWorld &, int) const { return det; }
    __device__ __forceinline__ long long left(const DevWorld &, int) const { return left_run; }
    __device__ __forceinline__ long long step(const DevWorld &) const { return now; }
    __device__ __forceinline__ int4 list(const DevWorld &w, int h) const { return w.nl[2 * (size_t)i + h]; }
    template <int ST>
    __device__ __forceinline__ bool search_cells(const DevWorld &w, int s, Narrow<ST> &nr) const {
        if (links == 0u) return false;
        walk_cells<3>(w, [&](int b) { return __ldcg(cur + b); }, w.par[s], w.pbuild[i], links,
                      [&](int b, float4) { narrow_test(w, i, b, *this, nr); });
        return true;
    }
    __device__ __forceinline__ float4 partner(const DevWorld &, int b) const { return __ldcg(cur + b); }
    __device__ __forceinline__ uint32_t partner_range(const DevWorld &, int b) const {
        return __float_as_uint(__ldcg(reinterpret_cast<const float *>(cur + b) + 3));
    }
    __device__ __forceinline__ float4 partner_disp(const DevWorld &, int b) const { return __ldcg(dcur + b); }
    __device__ __forceinline__ int bond_status(const DevWorld &w, int g) const { return __ldcg(w.b_status + g); }
    __device__ __forceinline__ void broke() { flags |= F_BROKE; }
    __device__ __forceinline__ float4 disp(const DevWorld &) const { return dcur[i]; }
    __device__ __forceinline__ void advance(const DevWorld &w, float4 p, float4 v, float4 d, float4 d4, bool moved,
                                            bool keep_d4) {
        if (keep_d4) w.d4[i] = d4;
        nxt[i] = p;
        w.vw[i] = v;
        dnxt[i] = d;
        if (moved) flags |= F_MOVED;
    }
    __device__ __forceinline__ void stay(const DevWorld &) {
        nxt[i] = pa;
        dnxt[i] = dcur[i];
    }
};

// The same run for worlds of more than a particle a thread: each thread
// sweeps the particles t, t + T, t + 2 T ... (T threads in the grid), whose
// state stays in device memory, in L2.  What it saves over a launch a step is
// the launches, the conditional node and the kernels that end the step.
template <int FORM, int PS>
__global__ void __launch_bounds__(SWEEP_THREADS, 1) k_sweep(DevWorld w, cudaGraphConditionalHandle more,
                                                            cudaGraphConditionalHandle rebuild,
                                                            const __grid_constant__ ScenePar pv) {
    extern __shared__ __align__(16) int32_t sm[];
    __shared__ uint32_t s_any[3];
    StepRun &R = *w.run;
    const int todo = R.todo;
    const bool lom_done = R.lom_done != 0, failed = R.fail == 1u;
    if (failed || todo <= 0) {  // uniform over the grid, as in k_steps
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            cudaGraphSetConditional(more, 0u);
            cudaGraphSetConditional(rebuild, 0u);
        }
        return;
    }
    uint32_t *ck = reinterpret_cast<uint32_t *>(sm) + threadIdx.x;
    Narrow<SWEEP_THREADS> nr{ck, reinterpret_cast<int *>(ck + K * SWEEP_THREADS)};
    const int t0 = blockIdx.x * SWEEP_THREADS + threadIdx.x, T = gridDim.x * SWEEP_THREADS;
    uint32_t flags = 0u;
    uint32_t links = R.linked ? R.links : 0u;
    Run<false> run(w, s_any, more, rebuild, lom_done);
    // steps the particle's scene has left at the run's first
    const auto steps_left = [&](int s) -> int {
        const long long rem = w.act[s] ? w.remaining[s] : 0;
        return rem > INT_MAX ? INT_MAX : (int)rem;
    };
    // frozen scenes' records in both buffers, so that either holds the world
    for (int i = t0; i < w.N; i += T)
        if (chunk_live(w, i) && steps_left((int)meta_scene(w.meta[i])) == 0) {
            w.pr_n[i] = w.pr[i];
            w.dp_n[i] = w.dp[i];
        }
    const auto rebuild_lists = [&](int done) -> bool {
        const float4 *cur = (done & 1) ? w.pr_n : w.pr;
        links = run.links;
        for (int i = t0; i < w.N; i += T) {
            if (!chunk_live(w, i)) continue;
            const int s = (int)meta_scene(w.meta[i]);
            const float4 pa = cur[i];
            if (steps_left(s) <= done || pa.z == 0.0f) continue;
            const ScenePar &G = w.par[s];
            int cx, cy;
            search_xy(G, pa.x, pa.y, cx, cy);
            const unsigned long long old = atomicExch(&w.cell_head[G.cell_base + cy * G.g_w + cx],
                                                      (unsigned long long)links << 32 | (unsigned)i);
            w.cell_next[i] = (uint32_t)(old >> 32) == links ? (int32_t)(uint32_t)old : -1;
        }
        if (run.meet(flags) & F_FAILED) return false;
        for (int i = t0; i < w.N; i += T) {
            if (!chunk_live(w, i)) continue;
            const int s = (int)meta_scene(w.meta[i]);
            const float4 pa = cur[i];
            int16_t *list = reinterpret_cast<int16_t *>(w.nl + 2 * (size_t)i);
            int cnt = 0, h0 = 0;
            bool over = false;
            w.pbuild[i] = make_float2(pa.x, pa.y);
            if (steps_left(s) > done && pa.z != 0.0f) {
                const ScenePar &G = w.par[s];
                const auto read = [&](int b) { return __ldcg(cur + b); };
                walk_cells<5>(w, read, G, make_float2(pa.x, pa.y), links, [&](int b, float4 pb) {
                    if (b == i || pb.z == 0.0f) return;
                    const float dx = pb.x - pa.x, dy = pb.y - pa.y;
                    const float t = (pa.z + pb.z + G.skin) * 1.00001f;
                    if (dx * dx + dy * dy > t * t) return;
                    const int off = b - i;
                    if (cnt < NL && off >= -32768 && off <= 32767) list[1 + cnt] = (int16_t)off;
                    else over = true;
                    ++cnt;
                });
                h0 = over ? NL_OVERFLOW : cnt;
                if (over) atomicAdd(&w.stats[5], 1ull);
            }
            list_head(w, i, list, h0);
        }
        return true;
    };

    bool stop = false;
    if (!lom_done) {
        for (int i = t0; i < w.N; i += T)
            if (chunk_live(w, i)) lom_particle(w, i);
        // lom_particle reports through w.rebuild: read once all have run
        stop = (run.meet(flags) & F_FAILED) != 0u;
        if (threadIdx.x == 0 && *(volatile int32_t *)w.rebuild != 0) flags |= F_MOVED;
        if (run.step_end(flags, 0, false, rebuild_lists)) stop = true;
    }
    int took = 0;
    for (int k = 0; !stop; ++k) {
        const bool last = k + 1 == todo;
        const bool odd = (k & 1) != 0;
        for (int i = t0; i < w.N; i += T) {
            if (!chunk_live(w, i)) continue;
            SweptOwn o(w, i, odd ? w.pr_n : w.pr, odd ? w.dp_n : w.dp, odd ? w.pr : w.pr_n, odd ? w.dp : w.dp_n, flags);
            const int s = (int)meta_scene(o.m);
            const int left = steps_left(s);
            const ScenePar &G = w.par[s];
            o.links = links;
            o.now = run.step0 + k;
            o.act = left > k;
            o.left_run = last ? 1 : left - k;
            const int32_t iv = G.p.collision_interval;
            o.det = iv <= 1 && G.cc1_0 >= 0 ? true : detect_at(iv, G.cc1_0, o.now - G.step0);
            nr.cnt = 0;
            interact_particle<0, true, FORM, PS>(w, i, o, nr, k + 2 == todo, pv);
        }
        took = k + 1;
        stop = run.step_end(flags, k + 1, last, rebuild_lists);
        if (last) took = 0;  // both buffers hold the last step's state
    }
    // back in the buffers that are current between runs
    if (took & 1)
        for (int i = t0; i < w.N; i += T) {
            if (!chunk_live(w, i)) continue;
            w.pr[i] = w.pr_n[i];
            w.dp[i] = w.dp_n[i];
        }
}

using StepsKernel = void (*)(DevWorld, cudaGraphConditionalHandle, cudaGraphConditionalHandle, ScenePar);

// the most threads of a block that a compiled kernel takes: fewer threads may
// hold more registers each (128 at 512 threads, where the bonded forms spill)
constexpr int TB_SMALL = 128, TB_MID = 256, TB_LARGE = 512;

// the kernel of one form (one translation unit each, for the time of a build)
template <int TB, bool CLU, int FORM>
StepsKernel steps_source(int ps) {
    return ps == PS_ONE ? k_steps<TB, CLU, FORM, PS_ONE>
                        : ps == PS_SHARED ? k_steps<TB, CLU, FORM, PS_SHARED> : k_steps<TB, CLU, FORM, PS_SCENE>;
}
template <int FORM>
StepsKernel steps_kernel(int block, bool cluster, int ps) {
    if (block == SWEEP_THREADS)
        return ps == PS_ONE ? k_sweep<FORM, PS_ONE>
                            : ps == PS_SHARED ? k_sweep<FORM, PS_SHARED> : k_sweep<FORM, PS_SCENE>;
    if (cluster) return block == TB_SMALL ? steps_source<TB_SMALL, true, FORM>(ps) : steps_source<TB_MID, true, FORM>(ps);
    return block <= TB_SMALL ? steps_source<TB_SMALL, false, FORM>(ps)
           : block <= TB_MID ? steps_source<TB_MID, false, FORM>(ps)
                             : steps_source<TB_LARGE, false, FORM>(ps);
}

}  // namespace demgb
