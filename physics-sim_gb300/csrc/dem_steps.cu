// dem_steps.cu -- launching the runs of steps of dem_steps.cuh.
#include "dem_steps.cuh"

namespace demgb {

extern template StepsKernel steps_kernel<0>(int, bool, int);
extern template StepsKernel steps_kernel<3>(int, bool, int);
extern template StepsKernel steps_kernel<-1>(int, bool, int);

__global__ void k_run_begin(DevWorld w, int todo, const int32_t *rec_rows, int rec_scene, int rec_base, int rec_per,
                            float *rec_out) {
    StepRun &R = *w.run;
    clear_run_barrier(R);
    R.todo = todo;
    R.done = 0;
    R.lom_done = 0;
    R.rec_rows = rec_rows;
    R.rec_scene = rec_scene;
    R.rec_base = rec_base;
    R.rec_per = rec_per;
    R.rec_out = rec_out;
    if (R.fail == 1u) *(volatile int32_t *)&R.report->failed = 1;
    report_lists(w);
}

void launch_run_begin(const DevWorld &w, int todo, const RunRecord &rec, cudaStream_t st) {
    k_run_begin<<<1, 1, 0, st>>>(w, todo, rec.rows, rec.scene, rec.base, rec.per, rec.out);
}

namespace {

// The most particles a thread of a swept world: with one, a step of a
// 131,000-particle bed goes from 29.3 to 18.9 us and of 129,756 particles of
// the mix from 22.0 to 14.0, with two of a 262,144-particle bed from 38.6 to
// 31.5 (214,475 of the mix 23.8 -> 23.6); with three it gains nothing (400,000:
// 46.0 -> 45.5) and beyond the launches' better balance wins.  Worlds of many
// neighbours a particle stop at one (World::runs_fit).
constexpr int SWEEPS = 2;

// Blocks of the cluster that holds a world of n particles, of tb threads each;
// 0: a grid does.  The hardware's barrier over up to 16 blocks and partner
// records in their shared memory against a barrier through L2 and records
// there, microseconds a step: 512 bonded particles 5.6 -> 4.7, 4,096 falling
// 3.75 -> 2.7, beds of 256 / 2,048 / 4,096 disks 6.7 -> 5.0 / 7.6 -> 6.1 /
// 8.0 -> 6.5.  One block alone loses (128 bonded 4.2 -> 4.75), and beyond 256
// threads a block the warps would share their schedulers.
int cluster_blocks(int n, int &tb) {
    static_assert(16 * TB_MID == CLUSTER_MOST, "a cluster of 16 blocks");
    if (n <= TB_SMALL || n > CLUSTER_MOST) return 0;
    tb = n <= 16 * TB_SMALL ? TB_SMALL : TB_MID;
    int blocks = 1;
    while (blocks * tb < n) blocks *= 2;
    return blocks <= 16 ? blocks : 0;
}

}  // namespace

int steps_block(int n) {
    // one block while it holds the world (its barrier costs a fifth of one over
    // several blocks), else 128 threads or more on every SM
    const int sms = device_sms();
    const int per = n <= TB_SMALL ? n : (n + sms - 1) / sms;
    const int rounded = (per + 31) / 32 * 32;
    const int block = n > TB_SMALL && rounded < TB_SMALL ? TB_SMALL : rounded;
    int dev = 0, coop = 0, smem = 0;
    if (n <= 0 || n > SWEEPS * sms * SWEEP_THREADS || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        smem < 4 * STEP_WORDS * TB_LARGE + 1024)
        return 0;
    if ((n + block - 1) / block >= 1023) return 0;  // the barrier's block count
    return block <= TB_LARGE ? block : SWEEP_THREADS;
}

cudaError_t launch_steps(const DevWorld &w, int block, cudaStream_t st, cudaGraphConditionalHandle more,
                         cudaGraphConditionalHandle rebuild, int form, const ScenePar *pv, int ps, bool *waits) {
    const auto kernel = [&](int threads, bool cluster) {
        return form == 0 ? steps_kernel<0>(threads, cluster, ps)
               : form == 3 ? steps_kernel<3>(threads, cluster, ps)
                           : steps_kernel<-1>(threads, cluster, ps);
    };
    const ScenePar none{};
    const ScenePar &par = ps == PS_SCENE ? none : *pv;
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a = {};
    c.stream = st;
    c.attrs = &a;
    int tb = 0;
    *waits = false;
    const int blocks = cluster_blocks(w.N, tb);
    if (blocks > 0) {
        // records in shared memory; a block an SM (two would share its schedulers)
        const StepsKernel fn = kernel(tb, true);
        const void *f = reinterpret_cast<const void *>(fn);
        int bytes = 4 * STEP_WORDS * tb + 64 * tb, fits = 0;
        if (bytes < 120 * 1024 && blocks > 1) bytes = 120 * 1024;
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = (unsigned)blocks;
        a.val.clusterDim.y = a.val.clusterDim.z = 1;
        c.gridDim = dim3((unsigned)blocks);
        c.blockDim = dim3((unsigned)tb);
        c.dynamicSmemBytes = (size_t)bytes;
        c.numAttrs = 1;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
            cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&fits, f, &c) == cudaSuccess && fits > 0)
            return cudaLaunchKernelEx(&c, fn, w, more, rebuild, par);
        cudaGetLastError();
    }
    const StepsKernel fn = kernel(block, false);
    int grid = (w.N + block - 1) / block;
    int bytes = 4 * STEP_WORDS * (block <= TB_SMALL ? TB_SMALL : block <= TB_MID ? TB_MID : TB_LARGE);
    if (block == SWEEP_THREADS) {
        grid = grid < device_sms() ? grid : device_sms();
        bytes = 4 * PARTNER_WORDS * SWEEP_THREADS;
    }
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void *>(fn),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    int per = 0;
    const cudaError_t o = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, block, (size_t)bytes);
    if (o != cudaSuccess) return o;
    if ((long long)per * device_sms() < grid) return cudaErrorCooperativeLaunchTooLarge;
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = (size_t)bytes;
    a.id = cudaLaunchAttributeCooperative;
    a.val.cooperative = 1;
    c.numAttrs = grid > 1 ? 1 : 0;
    *waits = grid > 1;
    return cudaLaunchKernelEx(&c, fn, w, more, rebuild, par);
}

}  // namespace demgb
