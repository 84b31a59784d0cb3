// dem_noalloc.cu -- the broad phase for callers that cannot allocate device memory.
//
// dem_broad_phase_noalloc() computes, for n particles given as device float4
// {x, y, radius, -}, their search-cell keys, the particle indices in stable
// cell order and the cell start table -- the three outputs of the context's
// broad phase (dem_debug_broad_phase), with one difference: the context keeps
// a scene's large particles out of the search cells (they head its last
// cell), while here every particle with a radius is keyed by its position and
// the last cell holds the zero-radius particles only -- without calling
// cudaMalloc, cudaFree or any allocating routine.  Its only scratch (one
// counter per cell, one sum per scan tile and the sort's per-block digit
// counts) lives in the file-scope device record below, of fixed size, which
// every GPU that loads the library keeps until the process exits.  The
// caller's d_keys buffer is the sort's second buffer (the keys are written
// last).
//
// Who needs this: code that runs where allocation is not allowed or not
// possible -- inside a caller's memory pool that owns the whole device heap,
// under a custom allocator that forbids cudaMalloc, or in a real-time loop
// where an allocation could block -- and therefore hands the library only
// buffers it already owns.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>

#include "dem.h"

namespace {

// The order is a least-significant-digit counting sort of two digits of 9
// bits (the cell limit makes keys 18 bits), one when the grid has at most 512
// cells.  With the first digit's pass also counting the cells and the cell
// table built beside the digits' offsets and scatter, a call is 8 launches,
// each one wave of blocks, and reads the positions three times: they and the
// two index arrays are all that must move, so launches and the trips to
// memory within each bound it.  1,000,003 particles in 509 x 509 cells:
// 50 us, against 152 for three 8-bit passes that read the positions by index
// from the second on, in 15 launches; 65 when each launch starts only after
// the one before has ended.
// (Device time by launch then: zero 2.8, count 11.4, offsets 6.7, scatter
// 16.0, count 4.7, offsets 6.4, scatter 11.7, keys 5.8.)
constexpr int NA_BITS = 9, NA_BINS = 1 << NA_BITS;
constexpr int NA_THREADS = 512, NA_WARPS = NA_THREADS / 32;
constexpr int NA_IPT = 8, NA_CHUNK = NA_THREADS * NA_IPT;  // elements ranked together
constexpr int NA_TILE = NA_THREADS * 4;                    // cells a block scans
constexpr int NA_TILES_MAX = (DEM_NOALLOC_MAX_CELLS + NA_TILE - 1) / NA_TILE;
constexpr int NA_GRID_MAX = 512;                           // blocks of a pass
constexpr int NA_DIGIT_BLOCKS = NA_BINS / (2 * NA_WARPS);  // two digits a warp
static_assert(DEM_NOALLOC_MAX_CELLS <= 1 << (2 * NA_BITS), "two digits cover every key");
// up to here the second digit and the index share the word that the first
// pass leaves, and the second pass reads no positions
constexpr int NA_INDEX_BITS = 32 - NA_BITS;

// cell histogram, then per tile its sum; per digit and block its count, then
// the count of the blocks before it; per digit its total
struct Scratch {
    int32_t cells[DEM_NOALLOC_MAX_CELLS];
    int32_t tiles[NA_TILES_MAX];
    int32_t digits[NA_BINS * NA_GRID_MAX];
    int32_t totals[NA_BINS];
};
static __device__ __align__(256) Scratch g_noalloc_scratch;

constexpr int MAX_DEVICES = 64;
Scratch *g_scratch_ptr[MAX_DEVICES] = {nullptr};
std::mutex g_scratch_mu;
thread_local std::string g_noalloc_error;

int na_fail(int code, const char *msg) {
    g_noalloc_error = msg;
    return code;
}

// Device address of the scratch array on the current device.  The array's
// name in host code is only a host-side handle, so the address is looked up
// once per device with that device current.
int scratch_for_current_device(Scratch **out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES)
        return na_fail(DEM_E_CUDA, "no current CUDA device");
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return na_fail(DEM_E_CUDA, "cudaGetSymbolAddress failed for the scratch array");
        g_scratch_ptr[dev] = static_cast<Scratch *>(p);
    }
    *out = g_scratch_ptr[dev];
    return DEM_OK;
}

__global__ void __launch_bounds__(NA_THREADS) k_na_zero(int32_t *counts, int c) {
    const int i = blockIdx.x * NA_THREADS + threadIdx.x;
    if (i < c) counts[i] = 0;
}

// search-cell key of a particle record
struct NaGrid {
    float x0, y0, inv;
    int gw, gh;
    __device__ __forceinline__ uint32_t key(float4 p) const {
        if (p.z == 0.0f) return (uint32_t)(gw * gh);
        int a = __float2int_rd((p.x - x0) * inv);
        int b = __float2int_rd((p.y - y0) * inv);
        a = a < 0 ? 0 : (a > gw - 1 ? gw - 1 : a);
        b = b < 0 ? 0 : (b > gh - 1 ? gh - 1 : b);
        return (uint32_t)(b * gw + a);
    }
};

// An element of a pass: its digit and its particle.  First: the particles in
// index order, whole keys.  Packed and Listed: what the first pass left.
struct First {
    const float4 *pr;
    NaGrid g;
    __device__ __forceinline__ uint32_t get(int t, int32_t &v) const {
        v = t;
        return g.key(pr[t]);
    }
};
struct Packed {
    const uint32_t *in;
    __device__ __forceinline__ uint32_t get(int t, int32_t &v) const {
        const uint32_t x = in[t];
        v = (int32_t)(x & ((1u << NA_INDEX_BITS) - 1u));
        return x >> NA_INDEX_BITS;
    }
};
struct Listed {
    const int32_t *in;
    const float4 *pr;
    NaGrid g;
    __device__ __forceinline__ uint32_t get(int t, int32_t &v) const {
        v = in[t];
        return g.key(pr[v]) >> NA_BITS;
    }
};

// Start of each kernel after the first: lets the next launch's blocks take
// their places beside this one's, then waits until the launch before is
// complete and its writes are visible.  Every thread of every launch waits, so
// a launch that is complete means that all before it are.
__device__ __forceinline__ void follow() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

// a block's contiguous range of n elements over `blocks` blocks (warp-aligned)
__device__ __forceinline__ void block_range(int n, int blocks, int &beg, int &end) {
    const int per = (int)((((long long)n + blocks - 1) / blocks + 31) & ~31LL);
    beg = (int)min((long long)blockIdx.x * per, (long long)n);
    end = (int)min((long long)beg + per, (long long)n);
}

// the block's count of each digit to digits[digit][block]; CELLS: also the
// cell histogram.  A warp whose elements all share a digit (or cell) adds once.
template <class In, bool CELLS>
__global__ void __launch_bounds__(NA_THREADS) k_na_count(In in, int n, Scratch *s) {
    __shared__ int h[NA_BINS];
    follow();
    for (int d = threadIdx.x; d < NA_BINS; d += NA_THREADS) h[d] = 0;
    __syncthreads();
    int beg, end;
    block_range(n, gridDim.x, beg, end);
    const int lane = threadIdx.x & 31;
    for (int cb = beg; cb < end; cb += NA_CHUNK) {
        uint32_t key[NA_IPT];
#pragma unroll
        for (int k = 0; k < NA_IPT; ++k) {
            const int t = cb + k * NA_THREADS + (int)threadIdx.x;
            int32_t v;
            key[k] = t < end ? in.get(t, v) : ~0u;
        }
#pragma unroll
        for (int k = 0; k < NA_IPT; ++k) {
            int same;
            __match_all_sync(0xffffffffu, key[k], &same);
            if (key[k] == ~0u || (same && lane != 0)) continue;
            const int add = same ? 32 : 1;
            if (CELLS) atomicAdd(&s->cells[key[k]], add);
            atomicAdd(&h[key[k] & (NA_BINS - 1)], add);
        }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < NA_BINS; d += NA_THREADS) s->digits[d * NA_GRID_MAX + blockIdx.x] = h[d];
}

__device__ __forceinline__ int warp_incl(int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)(threadIdx.x & 31) >= o) v += t;
    }
    return v;
}

// exclusive scan of one value a thread over the block; the sum in *total
__device__ __forceinline__ int block_excl(int v, int *total) {
    __shared__ int wsum[NA_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inc = warp_incl(v);
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int x = 0; x < NA_WARPS; ++x) {
        if (x < warp) before += wsum[x];
        all += wsum[x];
    }
    *total = all;
    __syncthreads();
    return before + inc - v;
}

// The first `tiles` blocks: exclusive scan of a tile of cell counts each, and
// its sum.  The others: two digits a warp, each digit's counts turned into
// the counts of the blocks before, and its total.
__global__ void __launch_bounds__(NA_THREADS) k_na_offsets(Scratch *s, int32_t *cell_start, int c, int tiles,
                                                           int blocks) {
    follow();
    if ((int)blockIdx.x < tiles) {
        const int base = blockIdx.x * NA_TILE + threadIdx.x * 4;
        int v[4], sum = 0, total;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = base + k < c ? s->cells[base + k] : 0;
            sum += v[k];
        }
        int off = block_excl(sum, &total);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (base + k < c) cell_start[base + k] = off;
            off += v[k];
        }
        if (threadIdx.x == 0) s->tiles[blockIdx.x] = total;
        return;
    }
    const int lane = threadIdx.x & 31;
    const int warp = ((int)blockIdx.x - tiles) * NA_WARPS + (threadIdx.x >> 5);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int d = 2 * warp + u;
        int32_t *row = s->digits + d * NA_GRID_MAX;
        int v[NA_GRID_MAX / 32];
#pragma unroll
        for (int k = 0; k < NA_GRID_MAX / 32; ++k) v[k] = 32 * k + lane < blocks ? row[32 * k + lane] : 0;
        int run = 0;
#pragma unroll
        for (int k = 0; k < NA_GRID_MAX / 32; ++k) {
            if (32 * k >= blocks) break;
            const int inc = warp_incl(v[k]);
            if (32 * k + lane < blocks) row[32 * k + lane] = run + inc - v[k];
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) s->totals[d] = run;
    }
}

// Stable scatter of a block's range by digit, a chunk at a time: ranks within
// a warp by ballots over the digit's bits, the warps' counts in warp order,
// the chunk put in digit order in shared memory and written out in runs.
// MODE 0: particles; 1: second digit << NA_INDEX_BITS | particle.  Blocks past `blocks` add the sums
// of the tiles before theirs to a tile of the cell table.
template <class In, int MODE>
__global__ void __launch_bounds__(NA_THREADS) k_na_scatter(In in, int n, int blocks, Scratch *s,
                                                           int32_t *__restrict__ out, int32_t *cell_start, int c) {
    __shared__ uint16_t wh[NA_WARPS * NA_BINS];  // per warp and digit: count, then offset within the chunk's digit
    __shared__ int run[NA_BINS];                 // next global position of each digit
    __shared__ int cbase[NA_BINS + 1];
    __shared__ uint32_t sval[NA_CHUNK];
    __shared__ uint16_t sdig[NA_CHUNK];
    int total;
    follow();
    if ((int)blockIdx.x >= blocks) {
        const int tile = (int)blockIdx.x - blocks;
        block_excl((int)threadIdx.x < tile ? s->tiles[threadIdx.x] : 0, &total);
        const int add = total;
        const int base = tile * NA_TILE + threadIdx.x * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (base + k < c) cell_start[base + k] += add;
        if (threadIdx.x == 0 && base + NA_TILE >= c) cell_start[c] = add + s->tiles[tile];
        return;
    }
    const int d0 = threadIdx.x;  // one digit a thread
    run[d0] = block_excl(s->totals[d0], &total) + s->digits[d0 * NA_GRID_MAX + blockIdx.x];
    int beg, end;
    block_range(n, blocks, beg, end);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    uint16_t *my = wh + warp * NA_BINS;
    for (int cb = beg; cb < end; cb += NA_CHUNK) {
        for (int d = lane; d < NA_BINS; d += 32) my[d] = 0;
        __syncwarp();
        uint32_t key[NA_IPT];
        int32_t val[NA_IPT];
        int off[NA_IPT];
        const int w0 = cb + warp * (32 * NA_IPT);
#pragma unroll
        for (int k = 0; k < NA_IPT; ++k) {
            const int t = w0 + k * 32 + lane;
            key[k] = ~0u;
            val[k] = 0;
            if (t < end) key[k] = in.get(t, val[k]);
        }
#pragma unroll
        for (int k = 0; k < NA_IPT; ++k) {
            const bool ok = key[k] != ~0u;
            const int d = (int)(key[k] & (NA_BINS - 1));
            unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
            for (int b = 0; b < NA_BITS; ++b) {
                const bool bit = (d >> b) & 1;
                const unsigned x = __ballot_sync(0xffffffffu, bit);
                peers &= bit ? x : ~x;
            }
            off[k] = ok ? my[d] + __popc(peers & below) : 0;
            __syncwarp();
            if (ok && lane == __ffs(peers) - 1) my[d] = (uint16_t)(my[d] + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        int sum = 0;
#pragma unroll
        for (int x = 0; x < NA_WARPS; ++x) {
            const int cnt = wh[x * NA_BINS + d0];
            wh[x * NA_BINS + d0] = (uint16_t)sum;
            sum += cnt;
        }
        cbase[d0] = block_excl(sum, &total);
        if (threadIdx.x == 0) cbase[NA_BINS] = total;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NA_IPT; ++k) {
            if (key[k] == ~0u) continue;
            const int d = (int)(key[k] & (NA_BINS - 1));
            const int q = cbase[d] + my[d] + off[k];
            sval[q] = MODE == 1 ? (key[k] >> NA_BITS) << NA_INDEX_BITS | (uint32_t)val[k] : (uint32_t)val[k];
            sdig[q] = (uint16_t)d;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < total; q += NA_THREADS) {
            const int d = sdig[q];
            out[run[d] + (q - cbase[d])] = (int32_t)sval[q];
        }
        __syncthreads();
        run[d0] += cbase[d0 + 1] - cbase[d0];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(NA_THREADS) k_na_write_keys(const float4 *__restrict__ pr, int n, NaGrid g,
                                                              int32_t *__restrict__ keys) {
    follow();
    for (int i = blockIdx.x * NA_THREADS + threadIdx.x; i < n; i += gridDim.x * NA_THREADS)
        keys[i] = (int32_t)g.key(pr[i]);
}

}  // namespace

extern "C" {

const char *dem_noalloc_last_error(void) { return g_noalloc_error.c_str(); }

int dem_broad_phase_noalloc(const float *d_pos_radius, int32_t n, float x0, float y0, float inv_cell,
                            int32_t gw, int32_t gh, int32_t *d_keys, int32_t *d_order,
                            int32_t *d_cell_start, void *stream) {
    if (n < 0 || gw <= 0 || gh <= 0) return na_fail(DEM_E_INVALID, "n must be >= 0 and the grid non-empty");
    if (n > (1 << 30)) return na_fail(DEM_E_CAPACITY, "n is above 2^30 particles");
    if ((long long)gw * gh + 1 > DEM_NOALLOC_MAX_CELLS)
        return na_fail(DEM_E_CAPACITY, "grid has more cells than DEM_NOALLOC_MAX_CELLS (262144, incl. the "
                                       "cell of zero-radius particles)");
    if (!(inv_cell > 0.0f)) return na_fail(DEM_E_INVALID, "inv_cell must be > 0");
    if (!d_cell_start || (n > 0 && (!d_pos_radius || !d_keys || !d_order)))
        return na_fail(DEM_E_INVALID, "a buffer pointer is NULL");
    if (reinterpret_cast<uintptr_t>(d_pos_radius) & 15u)
        return na_fail(DEM_E_INVALID, "d_pos_radius must be 16-byte aligned (float4 records)");
    Scratch *x = nullptr;
    int rc = scratch_for_current_device(&x);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int c = gw * gh + 1;
    const int tiles = (c + NA_TILE - 1) / NA_TILE;
    const float4 *pr = reinterpret_cast<const float4 *>(d_pos_radius);
    const NaGrid g{x0, y0, inv_cell, gw, gh};
    // one wave of blocks, two an SM, of at least 1,024 elements each
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
    const int most = 2 * sms < NA_GRID_MAX ? 2 * sms : NA_GRID_MAX;
    const int blocks = (int)(n / 1024 + 1 < most ? n / 1024 + 1 : most);
    const bool two = c > NA_BINS, packed = n <= 1 << NA_INDEX_BITS;
    const First first{pr, g};
    // Each launch after the first may take its places while the one before it
    // runs (its kernel waits), which spares most of the gap between two.
    // Not while the stream is captured: the caller's graph keeps plain edges.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(NA_THREADS);
    cfg.stream = st;
    cfg.attrs = &overlap;
    cfg.numAttrs = cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    cudaError_t e = cudaSuccess;
    auto next = [&](auto kernel, int grid, auto... args) {
        cfg.gridDim = dim3(grid);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kernel, args...);
    };
    k_na_zero<<<(c + NA_THREADS - 1) / NA_THREADS, NA_THREADS, 0, st>>>(x->cells, c);
    next(k_na_count<First, true>, blocks, first, n, x);
    next(k_na_offsets, tiles + NA_DIGIT_BLOCKS, x, d_cell_start, c, tiles, blocks);
    // the first pass into d_keys, the last one into d_order
    next(two && packed ? k_na_scatter<First, 1> : k_na_scatter<First, 0>, blocks + tiles, first, n, blocks, x,
         two ? d_keys : d_order, d_cell_start, c);
    if (two && packed) {
        const Packed in{reinterpret_cast<const uint32_t *>(d_keys)};
        next(k_na_count<Packed, false>, blocks, in, n, x);
        next(k_na_offsets, NA_DIGIT_BLOCKS, x, d_cell_start, c, 0, blocks);
        next(k_na_scatter<Packed, 0>, blocks, in, n, blocks, x, d_order, d_cell_start, c);
    } else if (two) {
        const Listed in{d_keys, pr, g};
        next(k_na_count<Listed, false>, blocks, in, n, x);
        next(k_na_offsets, NA_DIGIT_BLOCKS, x, d_cell_start, c, 0, blocks);
        next(k_na_scatter<Listed, 0>, blocks, in, n, blocks, x, d_order, d_cell_start, c);
    }
    if (n > 0) next(k_na_write_keys, 4 * sms, pr, n, g, d_keys);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return na_fail(DEM_E_CUDA, cudaGetErrorString(e));
    return DEM_OK;
}

}  // extern "C"
