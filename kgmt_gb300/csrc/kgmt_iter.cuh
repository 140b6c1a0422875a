// kgmt_iter.cuh -- device building blocks of one planning iteration: PTX
// helpers (mbarrier, bulk copy), block scans, the device-side schedule, the
// per-sample propagate steps and the propagate tile, region scores and the
// per-query finaliser.  The kernels in kgmt_kernels.cu are built from them.
#pragma once
#include <climits>
#include <cstdint>
#include <type_traits>

#include "kgmt_device.cuh"
#include "kgmt_kernels.h"

namespace kgmt {

// ---------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
    return ok != 0;
}

// bulk global -> shared copy through the TMA engine; bytes % 16 == 0, both
// addresses 16-byte aligned
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// the last-one-in count of a tile or query: a release add at GPU scope
// (everything this thread wrote, and what the block wrote before the last
// __syncthreads, is visible to whoever reads the count afterwards and
// fences) -- lighter than a full fence followed by a relaxed add
__device__ __forceinline__ uint32_t atomic_add_release(uint32_t* p, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.add.release.gpu.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// programmatic dependent launch: the kernel that follows in the stream may
// be scheduled once every block of this one has called pdl_trigger (or
// exited); pdl_wait blocks until the kernel before this one has completed
// and its memory is visible (immediately when launched without the attribute)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// KGMT_CHECK_BOUNDS builds (libkgmt_checked.so) test the kernels' scattered
// indices against their buffers: a failed test records kErrBounds in
// g_bounds_error and the access is skipped -- no trap, no fault -- and the
// host reports KGMT_ERR_INTERNAL.  Other builds compile the tests away.
// (Only kgmt_kernels.cu includes this header: the word is defined once.)
#ifdef KGMT_CHECK_BOUNDS
__device__ uint32_t g_bounds_error;
__device__ __forceinline__ bool bound_ok(bool c)
{
    if(!c) atomicOr(&g_bounds_error, kErrBounds);
    return c;
}
#define KGMT_BOUND(c) bound_ok(c)
#else
#define KGMT_BOUND(c) true
#endif

__device__ __forceinline__ unsigned long long ld_volatile_u64(const unsigned long long* p)
{
    return *(const volatile unsigned long long*)p;
}

__device__ __forceinline__ void st_volatile_u64(unsigned long long* p, unsigned long long v)
{
    *(volatile unsigned long long*)p = v;
}

// Tile bases of up to kBaseCache slots are copied to shared memory once per
// block, so finding a tile's query is a binary search in shared memory
// instead of ~log2(slots) dependent global loads.
constexpr int kBaseCache = 2048;

struct BaseCache {
    const uint32_t* base;  // shared copy, or the global array when too many slots
    int n;
};

__device__ __forceinline__ BaseCache cache_bases(const uint32_t* __restrict__ g, int n, uint32_t* s)
{
    if(n + 1 > kBaseCache) return {g, n};
    for(int i = threadIdx.x; i <= n; i += blockDim.x) s[i] = __ldcg(g + i);
    __syncthreads();
    return {s, n};
}

// last slot q with base[q] <= t (base is an exclusive prefix over n slots,
// base[n] = total, t < total)
__device__ __forceinline__ int find_slot(const uint32_t* __restrict__ base, int n, uint32_t t)
{
    int lo = 0, hi = n;
    while(lo < hi)
        {
            int mid = (lo + hi + 1) >> 1;
            if(base[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
    return lo;
}

// block-wide exclusive scan of one uint32 per thread; returns the exclusive
// prefix, *total the block sum.  scratch: >= 33 words of shared memory.
template <int NT>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* scratch, uint32_t* total)
{
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
        {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += y;
        }
    if(lane == 31) scratch[warp] = x;
    __syncthreads();
    if(warp == 0)
        {
            uint32_t w = lane < NW ? scratch[lane] : 0u;
            uint32_t z = w;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
                {
                    uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
                    if(lane >= o) z += y;
                }
            if(lane < NW) scratch[lane] = z - w;
            if(lane == NW - 1) scratch[32] = z;
        }
    __syncthreads();
    uint32_t excl = scratch[warp] + x - v;
    *total = scratch[32];
    __syncthreads();
    return excl;
}

// block-wide exclusive scan of three uint32 per thread at once; returns the
// exclusive prefixes, *total the block sums.  scratch: >= 33 entries.
template <int NT>
__device__ __forceinline__ uint3 block_exclusive_scan3(uint3 v, uint3* scratch, uint3* total)
{
    constexpr int NW = NT / 32;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint3 x = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
        {
            const uint32_t a = __shfl_up_sync(full, x.x, o), b = __shfl_up_sync(full, x.y, o), c = __shfl_up_sync(full, x.z, o);
            if(lane >= o) x.x += a, x.y += b, x.z += c;
        }
    if(lane == 31) scratch[warp] = x;
    __syncthreads();
    if(warp == 0)
        {
            const uint3 w = lane < NW ? scratch[lane] : make_uint3(0u, 0u, 0u);
            uint3 z = w;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t a = __shfl_up_sync(full, z.x, o), b = __shfl_up_sync(full, z.y, o), c = __shfl_up_sync(full, z.z, o);
                    if(lane >= o) z.x += a, z.y += b, z.z += c;
                }
            if(lane < NW) scratch[lane] = make_uint3(z.x - w.x, z.y - w.y, z.z - w.z);
            if(lane == NW - 1) scratch[32] = z;
        }
    __syncthreads();
    const uint3 e = scratch[warp];
    *total = scratch[32];
    __syncthreads();
    return make_uint3(e.x + x.x - v.x, e.y + x.y - v.y, e.z + x.z - v.z);
}

// ---------------------------------------------------------------------------
// schedule of the next iteration, computed by one block (the last query to
// finalise, or the admission path): tiles per slot, prefix bases, running
// count, and this iteration's tile sizes.  All threads of the calling block
// must enter.
// ---------------------------------------------------------------------------
// TOTALS: the finalisers of this iteration accumulated the running queries'
// samples and tree sizes in Sched::next_samples / next_tree (else a first
// pass over the slots sums them)
template <int NT = kAppendThreads, bool TOTALS = false>
__device__ void compute_schedule(const QueryParams* __restrict__ P, const QueryState* __restrict__ S, Sched* sched, uint32_t* tile_a_base,
                                 uint32_t* tile_c_base, uint32_t* tile_c_old)
{
    __shared__ uint3 s_scan[33];
    const int n = (int)sched->n_slots;
    const uint32_t block = sched->prop_block;
    const uint32_t pair_samples = sched->pair_samples;
    const uint32_t sms = sched->n_sms;
    const uint32_t* order = sched->prop_order;  // tile_a_base is in this order
    // samples per propagate tile: pairs per thread for large iterations; for
    // small ones the smallest power of two from 32 up to the block that keeps
    // the tiles within one per SM, so each tile's warps have an SM to
    // themselves (a tile's time is its slowest sample's)
    auto tile_for = [&](uint32_t total) -> uint32_t {
        if(total >= pair_samples) return kPropPer * block;
        if(sms == 0) return block;
        uint32_t t = 32u;
        while(t < block && (total + t - 1) / t > sms) t <<= 1;
        return t;
    };
    // old nodes per re-activation tile: small tiles while the old nodes of
    // all running queries fill fewer tiles than there are SMs, large ones
    // while they fill many waves of large tiles (each tile's fixed latency --
    // loads, scan, look-back -- spread over more nodes)
    auto old_tile_for = [&](uint32_t tree_total) -> uint32_t {
        if(sms != 0 && tree_total <= sms * (uint32_t)kTileOld) return (uint32_t)kTileOldSmall;
        if(sms != 0 && (unsigned long long)tree_total >= (unsigned long long)kOldLargeWaves * sms * (uint32_t)kTileOldLarge)
            return (uint32_t)kTileOldLarge;
        return (uint32_t)kTileOld;
    };
    // a slot's samples and tree size if it runs (three independent loads:
    // other blocks finalised these states in this kernel, so past L1)
    auto load = [&](int q, uint32_t& ns, uint32_t& tree) -> uint32_t {
        ns = tree = 0u;
        if(q >= n) return 0u;
        const uint32_t st = __ldcg(&S[q].status);
        const uint32_t a = __ldcg(&S[q].n_samples), b = __ldcg(&S[q].tree_size);
        if(st != KGMT_QUERY_RUNNING) return 0u;
        ns = a, tree = b;
        return 1u;
    };
    // totals only steer the tile sizes (thresholds below 2^22): clamped so
    // that no sum can wrap
    constexpr uint32_t kClamp = 1u << 22;
    auto publish = [&](uint32_t tiles_a, uint32_t tiles_c, uint32_t running, uint32_t prop_tile, uint32_t old_tile, uint32_t samples) {
        tile_a_base[n] = tiles_a;
        tile_c_base[n] = tiles_c;
        sched->tiles_a = tiles_a;
        sched->tiles_c = tiles_c;
        sched->running = running;
        sched->ticket_a = 0;
        sched->prop_tile = prop_tile;
        sched->old_tile = old_tile;
        sched->next_samples = 0ull;
        sched->next_tree = 0ull;
        if(running) sched->iterations += 1;
        if(sched->host_running)
            {
                *(volatile uint32_t*)(sched->host_running + 4) = samples;
                *(volatile uint32_t*)sched->host_running = running;
            }
    };
    if(n <= 32)
        {
            // up to 32 slots: one warp, shuffle scans, no block barriers but the last
            if(threadIdx.x < 32)
                {
                    const unsigned full = 0xffffffffu;
                    const int q = (int)threadIdx.x;
                    uint32_t ns, tree;
                    const uint32_t run = load(q, ns, tree);
                    const uint32_t tot_s = __reduce_add_sync(full, ns < kClamp ? ns : kClamp);
                    const uint32_t tot_t = __reduce_add_sync(full, tree < kClamp ? tree : kClamp);
                    const uint32_t prop_tile = tile_for(tot_s), old_tile = old_tile_for(tot_t);
                    uint32_t tc = 0, told = 0;
                    const uint32_t ns_a = __shfl_sync(full, ns, order && q < n ? (int)order[q] : q);
                    // tile sizes are powers of two
                    const uint32_t ta = (ns_a + prop_tile - 1) >> (__ffs(prop_tile) - 1);
                    if(run)
                        {
                            told = (tree + old_tile - 1) >> (__ffs(old_tile) - 1);
                            tc = told + (ns + kTileC - 1) / kTileC;
                        }
                    uint32_t ia = ta, ic = tc, ir = run;
#pragma unroll
                    for(int o = 1; o < 32; o <<= 1)
                        {
                            const uint32_t ya = __shfl_up_sync(full, ia, o);
                            const uint32_t yc = __shfl_up_sync(full, ic, o);
                            const uint32_t yr = __shfl_up_sync(full, ir, o);
                            if(q >= o) ia += ya, ic += yc, ir += yr;
                        }
                    if(q < n)
                        {
                            tile_a_base[q] = ia - ta;
                            tile_c_base[q] = ic - tc;
                            tile_c_old[q] = told;
                        }
                    if(q == 31) publish(ia, ic, ir, prop_tile, old_tile, tot_s);
                }
            __syncthreads();
            return;
        }
    // pass 1: the running queries' samples and tree sizes, for the tile sizes
    // (a block of slots or fewer keeps its loads in registers for pass 2)
    uint32_t ns0 = 0, tree0 = 0, run0 = 0;
    uint3 tot = make_uint3(0u, 0u, 0u);
    if(TOTALS)
        {
            const unsigned long long a = __ldcg(&sched->next_samples), b = __ldcg(&sched->next_tree);
            tot.x = a < kClamp ? (uint32_t)a : kClamp;
            tot.y = b < kClamp ? (uint32_t)b : kClamp;
            if(threadIdx.x < n) run0 = load((int)threadIdx.x, ns0, tree0);
        }
    else
        {
            uint3 part = make_uint3(0u, 0u, 0u);
            for(int q = threadIdx.x; q < n; q += NT)
                {
                    uint32_t ns, tree;
                    const uint32_t run = load(q, ns, tree);
                    if(q == (int)threadIdx.x) ns0 = ns, tree0 = tree, run0 = run;
                    part.x = min(part.x + min(ns, kClamp), kClamp);
                    part.y = min(part.y + min(tree, kClamp), kClamp);
                }
            block_exclusive_scan3<NT>(part, s_scan, &tot);
        }
    const uint32_t prop_tile = tile_for(tot.x), old_tile = old_tile_for(tot.y);
    const int sh_a = __ffs(prop_tile) - 1, sh_o = __ffs(old_tile) - 1;  // tile sizes are powers of two
    // pass 2: tiles per slot and their exclusive prefixes
    uint3 carry = make_uint3(0u, 0u, 0u);
    for(int base = 0; base < n; base += NT)
        {
            const int q = base + (int)threadIdx.x;
            uint32_t ns = ns0, tree = tree0, run = run0;
            if(base > 0) run = load(q, ns, tree);
            uint32_t ns_a = ns, tree_a, tc = 0, told = 0;
            if(order && q < n) load((int)order[q], ns_a, tree_a);
            const uint32_t ta = (ns_a + prop_tile - 1) >> sh_a;
            if(run)
                {
                    told = (tree + old_tile - 1) >> sh_o;
                    tc = told + (ns + kTileC - 1) / kTileC;
                }
            uint3 sum;
            const uint3 e = block_exclusive_scan3<NT>(make_uint3(ta, tc, run), s_scan, &sum);
            if(q < n)
                {
                    tile_a_base[q] = carry.x + e.x;
                    tile_c_base[q] = carry.y + e.y;
                    tile_c_old[q] = told;
                }
            carry.x += sum.x, carry.y += sum.y, carry.z += sum.z;
        }
    if(threadIdx.x == 0) publish(carry.x, carry.y, carry.z, prop_tile, old_tile, tot.x);
    __syncthreads();
}

// frontier entries R, samples per entry and samples of the next iteration
// (KGMT.cu:183-201 with the capacity rule made safe)
__device__ __forceinline__ void plan_samples_vals(uint32_t capacity, uint32_t samples_per_node, uint32_t tree_size, uint32_t R, uint32_t* spe_out,
                                                  uint32_t* n_out)
{
    const uint32_t free_slots = capacity - tree_size;
    uint32_t spe = 0, ruse = R;
    if(R > 0)
        {
            spe = free_slots / R;
            if(spe > samples_per_node) spe = samples_per_node;
            if(spe == 0)
                {
                    spe = 1;
                    ruse = free_slots;
                }
        }
    *spe_out = spe;
    *n_out = ruse * spe;
}

__device__ __forceinline__ void plan_samples(const QueryParams& P, QueryState& st)
{
    plan_samples_vals(P.capacity, P.samples_per_node, st.tree_size, st.n_react + st.w_new, &st.spe, &st.n_samples);
}

// ---------------------------------------------------------------------------
// propagate
// ---------------------------------------------------------------------------
struct PropCtx {
    uint32_t itr, spe, n_react, n_samples;
};

constexpr int kSortBins = 32;  // step-count bins of the in-tile sort (last bin: dead lanes)

struct PropShared {
    uint32_t acc;                // accepted samples of the tile
    uint32_t steps;              // RK4 steps of the tile
    uint32_t tests;              // box tests of the tile
};

// sample rows of a model
// SAMPLE_DIM and the number of control draws (the step draw follows them,
// then the accept draw)
template <int MODEL>
struct ModelDims {
    static constexpr int D = MODEL == KGMT_MODEL_QUADROTOR ? 17 : MODEL == KGMT_MODEL_UNICYCLE ? 7 : 10;
    static constexpr int NC = MODEL == KGMT_MODEL_QUADROTOR ? 4 : 3;
};

// model bits of the MODELS mask a propagate variant is compiled for
constexpr int kBitDI = 1, kBitQuad = 2, kBitDubins = 4, kBitUnicycle = 8, kAllModels = 15;

// calls f(std::integral_constant<int, model>) for the query's model, among
// the models the variant was compiled for (a single-model variant needs no test)
template <int MODELS, typename F>
__device__ __forceinline__ void with_model(int model, F&& f)
{
    if constexpr((MODELS & kBitDI) != 0)
        if(MODELS == kBitDI || model == KGMT_MODEL_DOUBLE_INTEGRATOR) f(std::integral_constant<int, KGMT_MODEL_DOUBLE_INTEGRATOR>{});
    if constexpr((MODELS & kBitQuad) != 0)
        if(MODELS == kBitQuad || model == KGMT_MODEL_QUADROTOR) f(std::integral_constant<int, KGMT_MODEL_QUADROTOR>{});
    if constexpr((MODELS & kBitDubins) != 0)
        if(MODELS == kBitDubins || model == KGMT_MODEL_DUBINS_AIRPLANE) f(std::integral_constant<int, KGMT_MODEL_DUBINS_AIRPLANE>{});
    if constexpr((MODELS & kBitUnicycle) != 0)
        if(MODELS == kBitUnicycle || model == KGMT_MODEL_UNICYCLE) f(std::integral_constant<int, KGMT_MODEL_UNICYCLE>{});
}

template <int MODEL, typename Grid>
__device__ __forceinline__ bool propagate_model(const QueryParams& p, const Grid& grid, const float* x0, const float* u, const float4* obs,
                                                uint32_t n_obs, float* x1, PropCount& cnt)
{
    if constexpr(MODEL == KGMT_MODEL_QUADROTOR) return propagate_quad(p, grid, x0, u, obs, n_obs, x1, cnt);
    else if constexpr(MODEL == KGMT_MODEL_DUBINS_AIRPLANE) return propagate_dubins(p, grid, x0, u, obs, n_obs, x1, cnt);
    else if constexpr(MODEL == KGMT_MODEL_UNICYCLE) return propagate_unicycle(p, grid, x0, u, obs, n_obs, x1, cnt);
    else return propagate_di(p, grid, x0, u, obs, n_obs, x1, cnt);
}

// rows of D floats: with D even every row starts 8-byte aligned (row
// buffers are 256-byte aligned), so they move as float2 pairs.  COHERENT:
// the row may have been written earlier in the same launch by another block
// (the persistent tail kernel), so it is read through L2 instead of the
// read-only path, which is only valid for data no one writes during the launch.
template <int D, bool COHERENT = false>
__device__ __forceinline__ void load_row_ro(const float* __restrict__ src, float* r)
{
    if constexpr(D % 2 == 0)
        {
#pragma unroll
            for(int c = 0; c < D / 2; ++c)
                {
                    const float2 v = COHERENT ? __ldcg((const float2*)src + c) : __ldg((const float2*)src + c);
                    r[2 * c] = v.x, r[2 * c + 1] = v.y;
                }
        }
    else
        {
#pragma unroll
            for(int c = 0; c < D; ++c) r[c] = COHERENT ? __ldcg(src + c) : __ldg(src + c);
        }
}

template <int D>
__device__ __forceinline__ void store_row(float* dst, const float* r)
{
    if constexpr(D % 2 == 0)
        {
#pragma unroll
            for(int c = 0; c < D / 2; ++c) ((float2*)dst)[c] = make_float2(r[2 * c], r[2 * c + 1]);
        }
    else
        {
#pragma unroll
            for(int c = 0; c < D; ++c) dst[c] = r[c];
        }
}

// A sample's eight uniforms come from two Philox blocks, (s, itr, 0, 0) and
// (s, itr, 0, 1): controls first, then the step draw, then the accept draw.
// The block holding the step draw ("key block": the first for three
// controls, the second for four) is drawn once, when the tile is sorted by
// step count, and handed to the thread that propagates the sample.
template <int MODEL>
__device__ __forceinline__ U4 sample_key_block(const QueryParams& p, const PropCtx& c, uint32_t s)
{
    const uint32_t k0 = (uint32_t)p.seed, k1 = (uint32_t)(p.seed >> 32);
    return philox4x32_10(s, c.itr, 0u, ModelDims<MODEL>::NC == 4 ? 1u : 0u, k0, k1);
}

// RK4 steps of the sample whose key block is kb, for ordering the samples of
// a tile so that a warp's lanes loop about equally long
template <int MODEL>
__device__ __forceinline__ int sample_steps(const QueryParams& p, const U4& kb)
{
    return draw_steps(p, u01(ModelDims<MODEL>::NC == 4 ? kb.x : kb.w));
}

// gather the parent row and draw the sample's uniforms (no obstacle access,
// so it runs while the tile's boxes are still in flight); kb: its key block
template <int MODEL, bool COHERENT = false>
__device__ __forceinline__ uint32_t prepare_sample(const QueryParams& p, const PropCtx& c, uint32_t s, const U4& kb, float* x0, float* u)
{
    constexpr int D = ModelDims<MODEL>::D;
    const uint32_t e = s / c.spe;
    uint32_t par = e < c.n_react ? (KGMT_BOUND(e < p.capacity) ? p.rep_old[e] : 0u)
                                 : (KGMT_BOUND(e - c.n_react < p.capacity) ? p.rep_new[e - c.n_react] : 0u);
    if(!KGMT_BOUND(par < p.capacity)) par = 0u;
    load_row_ro<D, COHERENT>(p.tree + (size_t)par * D, x0);
    const uint32_t k0 = (uint32_t)p.seed, k1 = (uint32_t)(p.seed >> 32);
    constexpr bool four = ModelDims<MODEL>::NC == 4;
    const U4 other = philox4x32_10(s, c.itr, 0u, four ? 0u : 1u, k0, k1);
    const U4& a = four ? other : kb;
    const U4& b = four ? kb : other;
    u[0] = u01(a.x), u[1] = u01(a.y), u[2] = u01(a.z), u[3] = u01(a.w);
    u[4] = u01(b.x), u[5] = u01(b.y), u[6] = u01(b.z), u[7] = u01(b.w);
    return par;
}

// row, parent and word: where the sample's end row and parent go if it joins the
// tree, and its region with the accept flag (global arrays, or shared memory)
template <int MODEL>
__device__ __forceinline__ void finish_sample(const QueryParams& p, const GridView& grid, const float4* obs, uint32_t n_obs, uint32_t s,
                                              bool live, uint32_t par, const float* x0, const float* u, PropShared* sh, float* row,
                                              int32_t* parent, uint32_t* word)
{
    constexpr int D = ModelDims<MODEL>::D;
    constexpr int NC = ModelDims<MODEL>::NC;
    const unsigned full = 0xffffffffu;
    int r1 = -1;
    uint64_t bit = 0ull;
    PropCount cnt;
    bool ok = false, acc = false;
    if(live)
        {
            float x1[D];
            ok = propagate_model<MODEL>(p, grid, x0, u, obs, n_obs, x1, cnt);
            const CellIds cid = cell_ids(p, x1);
            r1 = cid.r1;
            bit = 1ull << cid.r2;
            if(!KGMT_BOUND((uint32_t)r1 < p.regions && s < p.capacity)) live = ok = false;
            if(ok)
                {
                    const uint64_t marks = p.marks[r1];
                    const float score = p.score[r1];
                    const bool fresh = (marks & bit) == 0ull;
                    acc = (u[NC + 1] < score) || fresh;
                }
            // only a sample that joins the tree is read again (by the append
            // kernel): its row and parent; every sample's region and accept
            // flag, in one word (region ids are below 2^31)
            if(acc)
                {
                    store_row<D>(row, x1);
                    *parent = (int32_t)par;
                }
            if(live) *word = (uint32_t)r1 | (acc ? 0x80000000u : 0u);
        }
    // histogram updates (KGMT.cu:250-253): counter over all samples, valid
    // count and the fine-cell bit over the valid ones; one fire-and-forget L2
    // atomic per sample (aggregating a warp's equal regions first with
    // match.any cost more than it saved: the batch ran 2.5 % slower); tile
    // totals in shared memory
    if(live) atomicAdd(&p.counter[r1], 1);
    if(ok)
        {
            atomicAdd(&p.valid[r1], 1);
            atomicOr((unsigned long long*)&p.newmarks[r1], (unsigned long long)bit);
        }
    const unsigned acc_mask = __ballot_sync(full, acc);
    const unsigned warp_steps = __reduce_add_sync(full, (unsigned)cnt.steps);
    const unsigned warp_tests = __reduce_add_sync(full, cnt.tests);
    if((threadIdx.x & 31) == 0)
        {
            if(acc_mask) atomicAdd(&sh->acc, (unsigned)__popc(acc_mask));
            if(warp_steps) atomicAdd(&sh->steps, warp_steps);
            if(warp_tests) atomicAdd(&sh->tests, warp_tests);
        }
}

// ---------------------------------------------------------------------------
// propagate tiles: each block keeps two, the one its warps work on and the next,
// so a warp never waits for the block.  A tile's samples are counting-sorted by
// step count and taken 32 at a time, longest first, by whichever warp is free;
// the last warp to leave a tile adds up its counts and prepares the tile after
// the next in the same buffer, while the others go on with the next.
// Bound by instruction issue and, in small iterations, by the latency of the
// few samples a warp has.  With block barriers around each tile the warps of a
// block waited for its longest run and for the sort (2.6 - 2.9 of the 7 - 9
// warps a scheduler had were at a barrier): iterations of the mixed batch with
// few samples issued 40 - 48 % of the time, now 63 %; 256 double-integrator
// queries took 3.12 ms, then 2.81 (2.69 with three blocks an SM); the 2M-node
// quadrotor tree 4.63, then 4.25.
// ---------------------------------------------------------------------------
template <int NT>
struct TileBuf {
    QueryParams p;  // of the tile's query
    uint64_t bar;   // its boxes and grid, copied in bulk
    PropCtx c;
    int q;
    uint32_t first, n;           // samples [first, first + n) of the query
    uint32_t next_run, left;     // runs handed out; warps that are done with the tile
    uint32_t units;              // kSpinLimit polls each: a wait for the buffer's next tile lasts a run of this one
    PropShared sh;
    uint32_t hist[kSortBins];
    uint16_t rank[kPropPer * NT];  // while sorting: step-count bin and rank in it
    uint16_t perm[kPropPer * NT];  // samples in sorted order
};

// Tile `lt` of query q into a buffer, by one warp (BLOCK: by the whole block, for
// a launch's first tile, which nothing overlaps): the query's params and loop
// state, the bulk copies of its boxes and grid (not waited for), and the sorted
// order.  dyn: the buffer's dynamic shared memory.
template <int NT, int MODELS, bool BLOCK>
__device__ __forceinline__ void prepare_tile(TileBuf<NT>& B, char* dyn, const QueryParams* __restrict__ P, const QueryState* S, int q, uint32_t lt,
                                             uint32_t tile, uint32_t smem_boxes)
{
    constexpr uint32_t W = BLOCK ? NT : 32;
    const uint32_t lane = BLOCK ? threadIdx.x : threadIdx.x & 31u;
    auto sync = [] {
        if constexpr(BLOCK) __syncthreads();
        else __syncwarp();
    };
    const unsigned full = 0xffffffffu;
    const QueryParams& gp = P[q];
    const uint32_t* src = (const uint32_t*)&gp;
    uint32_t* dst = (uint32_t*)&B.p;
#pragma unroll
    for(uint32_t i = 0; i < (sizeof(QueryParams) / 4 + W - 1) / W; ++i)
        if(i * W + lane < sizeof(QueryParams) / 4) dst[i * W + lane] = src[i * W + lane];
    if(lane == 0)
        {
            const QueryState& st = S[q];
            const uint32_t ns = st.n_samples;
            B.c.itr = st.itr;
            B.c.spe = st.spe;
            B.c.n_react = st.n_react;
            B.c.n_samples = ns;
            B.q = q;
            B.first = lt * tile;
            B.n = min(tile, ns - lt * tile);
            B.next_run = 0, B.left = 0;
            B.units = wait_units(gp.max_steps, gp.n_obstacles);
            B.sh.acc = 0, B.sh.steps = 0, B.sh.tests = 0;
            // boxes, grid meta, grid starts and the first grid items: one
            // mbarrier transaction of bulk copies (possibly of no bytes)
            const uint32_t n_obs = gp.n_obstacles;
            const bool obs_s = n_obs > 0 && n_obs <= smem_boxes;
            const bool grid = gp.grid_meta != nullptr;
            fence_proxy_async_smem();
            mbar_expect_tx(&B.bar, (obs_s ? n_obs * 32u : 0u) + (grid ? 16u + kSmemStartBytes + kSmemGridItems * 2u : 0u));
            if(obs_s) bulk_copy_g2s(dyn + kSmemGridBytes, gp.obstacles, n_obs * 32u, &B.bar);
            if(grid)
                {
                    bulk_copy_g2s(dyn + kSmemStartBytes + kSmemGridItems * 2u, gp.grid_meta, 16u, &B.bar);
                    bulk_copy_g2s(dyn, gp.grid_start, kSmemStartBytes, &B.bar);
                    bulk_copy_g2s(dyn + kSmemStartBytes, gp.grid_items, kSmemGridItems * 2u, &B.bar);
                }
        }
    if(lane < 32u) B.hist[lane] = 0;
    static_assert(kSortBins == 32 && kPropPer * NT <= 1024, "a bin a lane; bin and rank share 16 bits");
    sync();
    const uint32_t n = B.n, first = B.first;
    const int model = B.p.model;
#pragma unroll 2
    for(uint32_t i = lane; i < n; i += W)
        {
            int k = 1;
            with_model<MODELS>(model, [&](auto m) {
                constexpr int M = decltype(m)::value;
                k = sample_steps<M>(B.p, sample_key_block<M>(B.p, B.c, first + i));
            });
            const uint32_t key = (uint32_t)(k < kSortBins ? k : kSortBins - 1);
            B.rank[i] = (uint16_t)(key << 10 | atomicAdd(&B.hist[key], 1u));
        }
    sync();
    if(!BLOCK || lane < 32u)
        {
            const uint32_t v = B.hist[lane];
            uint32_t x = v;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t y = __shfl_up_sync(full, x, o);
                    if(lane >= (uint32_t)o) x += y;
                }
            B.hist[lane] = x - v;
        }
    sync();
    for(uint32_t i = lane; i < n; i += W)
        {
            const uint32_t r = B.rank[i];
            B.perm[B.hist[r >> 10] + (r & 1023u)] = (uint16_t)i;
        }
}

// The runs of a prepared tile that this warp takes.  parity: of the buffer's
// bulk copies, waited for once, after the first run has gathered its parents.
template <int NT, int MODELS>
__device__ __forceinline__ void run_tile(TileBuf<NT>& B, char* dyn, uint32_t smem_boxes, uint32_t parity, uint32_t* error)
{
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const QueryParams& sp = B.p;
    const int model = sp.model;
    const uint32_t n = B.n, n_runs = (n + 31u) / 32u;
    const uint16_t* gstart = (const uint16_t*)dyn;
    const uint16_t* gitems = (const uint16_t*)(dyn + kSmemStartBytes);
    const uint32_t* gmeta = (const uint32_t*)(dyn + kSmemStartBytes + kSmemGridItems * 2u);
    const float4* obs = sp.n_obstacles <= smem_boxes ? (const float4*)(dyn + kSmemGridBytes) : sp.obstacles;
    bool waited = false;
    for(;;)
        {
            uint32_t run = 0;
            if(lane == 0) run = atomicAdd(&B.next_run, 1u);
            run = __shfl_sync(full, run, 0);
            if(run >= n_runs) break;
            // longest runs first
            const uint32_t slot = (n_runs - 1u - run) * 32u + lane;
            const bool live = slot < n;
            const uint32_t s = B.first + (live ? (uint32_t)B.perm[slot] : 0u);
            float x0[KGMT_MAX_SAMPLE_DIM], u[8];
            uint32_t par = 0;
            if(live)
                with_model<MODELS>(model, [&](auto m) {
                    constexpr int M = decltype(m)::value;
                    par = prepare_sample<M>(sp, B.c, s, sample_key_block<M>(sp, B.c, s), x0, u);
                });
            if(!waited)
                {
                    waited = true;
                    uint32_t spins = 0;
                    while(!mbar_try_wait(&B.bar, parity))
                        if(++spins > kSpinLimit)
                            {
                                if(lane == 0) atomicOr(error, kErrCopyTimeout);
                                break;
                            }
                }
            const GridView grid{(sp.grid_meta != nullptr && gmeta[1] == 1u) ? gstart : nullptr, gitems, sp.grid_items};
            with_model<MODELS>(model, [&](auto m) {
                constexpr int M = decltype(m)::value;
                finish_sample<M>(sp, grid, obs, sp.n_obstacles, s, live, par, x0, u, &B.sh, sp.us + (size_t)s * ModelDims<M>::D, sp.up + s, sp.ur1f + s);
            });
        }
}

// Samples [s0, s0 + n) of one query, one per thread (n <= NT), in index
// order -- no sort: with one such range per block the time of a launch is its
// slowest warp's, which ordering the samples inside a block cannot shorten.
// Parent rows are read coherently (they may have been appended by other
// blocks in the same launch); sample s0 + i leaves its end row, parent and
// region word at rows + i D, parents + i and words + i.  `wait` runs once,
// after the parents and draws are gathered.  Block-uniform call.
template <int NT, int MODELS, typename Wait>
__device__ __forceinline__ void propagate_range(const QueryParams& sp, const PropCtx& sc, uint32_t s0, uint32_t n, uint32_t smem_boxes,
                                                PropShared* sh, const float4* s_obs, const uint16_t* s_gstart, const uint16_t* s_gitems,
                                                const uint32_t* s_gmeta, float* rows, int32_t* parents, uint32_t* words, Wait&& wait)
{
    const int model = sp.model;
    const uint32_t i = threadIdx.x, s = s0 + i;
    const bool live = i < n && s < sc.n_samples;
    float x0[KGMT_MAX_SAMPLE_DIM], u[8];
    uint32_t par = 0;
    if(live)
        with_model<MODELS>(model, [&](auto m) {
            const U4 kb = sample_key_block<decltype(m)::value>(sp, sc, s);
            par = prepare_sample<decltype(m)::value, true>(sp, sc, s, kb, x0, u);
        });
    wait();
    const float4* obs = sp.n_obstacles <= smem_boxes ? s_obs : sp.obstacles;
    const GridView grid{(sp.grid_meta != nullptr && s_gmeta[1] == 1u) ? s_gstart : nullptr, s_gitems, sp.grid_items};
    with_model<MODELS>(model, [&](auto m) {
        constexpr int M = decltype(m)::value;
        finish_sample<M>(sp, grid, obs, sp.n_obstacles, s, live, par, x0, u, sh, rows + (size_t)i * ModelDims<M>::D, parents + i, words + i);
    });
}

// ---------------------------------------------------------------------------
// region scores: Graph::updateVertices (Graph.cu:311-358).  All regions of a query
// are scored, lane l of kScoreLanes sums regions l, l+256, ... in order, then a
// halving tree over the lanes; a small table by update_scores, a large one by
// score_slice and score_finish.  Histograms and marks were updated by other blocks'
// atomics (in the tail launch, in this kernel): read past L1.
// ---------------------------------------------------------------------------
// The fields of QueryParams the scores use, held in registers.
struct ScoreParams
{
    int32_t* counter;
    int32_t* valid;
    float* score;
    uint64_t* marks;
    uint64_t* newmarks;
    uint32_t regions, fine_cells;
    float epsilon, cell_volume;
};

__device__ __forceinline__ ScoreParams score_params(const QueryParams& p)
{
    return {p.counter, p.valid, p.score, p.marks, p.newmarks, p.regions, p.fine_cells, p.epsilon, p.cell_volume};
}

// raw score of a region with n samples, nv of them valid, and the visited fine
// cells m; -1 marks "no valid sample" for the normalisation
__device__ __forceinline__ float raw_score(const ScoreParams& p, float F, uint64_t m, int32_t nv, int32_t n)
{
    if(nv <= 0) return -1.0f;
    const float cov = (float)__popcll(m) / F;
    const float a = p.epsilon + (float)nv;
    const float b = a + (float)(n - nv);
    const float fv = (a / b) * p.cell_volume;
    const float f2 = fv * fv;
    const float f4 = f2 * f2;
    const float nf = (float)n;
    const float den = (1.0f + cov) * (1.0f + nf * nf);
    return f4 / den;
}

// what a raw score adds to the total
__device__ __forceinline__ float scored(float raw) { return raw < 0.0f ? 0.0f : raw; }

// raw score (-1 for regions without valid samples) -> normalised score
__device__ __forceinline__ float norm_score(const ScoreParams& p, float raw, float total)
{
    return raw < 0.0f ? 1.0f : (total > 0.0f ? p.epsilon + raw / total : p.epsilon);
}

// halving tree over the lanes' sums (lane l adds lane l + stride, strides 128 ..
// 1); every thread gets the total.  Block-uniform.  One warp does all levels in
// registers: thread t holds lanes t, t + 32, ..., so the strides of 32 and more
// stay inside it and the rest are shuffles -- no block barrier a level.
__device__ __forceinline__ float lanes_total(float* lanes)
{
    __syncthreads();
    if(threadIdx.x < 32)
        {
            constexpr int K = kScoreLanes / 32;
            static_assert((K & (K - 1)) == 0, "halving levels");
            float v[K];
#pragma unroll
            for(int k = 0; k < K; ++k) v[k] = lanes[threadIdx.x + 32 * k];
#pragma unroll
            for(int h = K / 2; h >= 1; h >>= 1)
#pragma unroll
                for(int k = 0; k < h; ++k) v[k] = v[k] + v[k + h];
#pragma unroll
            for(int stride = 16; stride >= 1; stride >>= 1) v[0] = v[0] + __shfl_down_sync(0xffffffffu, v[0], stride);
            if(threadIdx.x == 0) lanes[0] = v[0];
        }
    __syncthreads();
    return lanes[0];
}

// a table of at most kScoreSmall regions, by one block: a lane a thread
template <int NT>
__device__ void update_scores(const ScoreParams& p, QueryState& st, float* lanes)
{
    static_assert(NT >= kScoreLanes, "a lane a thread");
    const float F = (float)p.fine_cells;
    constexpr int U = (int)kScoreSmall / kScoreLanes;  // a lane's regions: loaded together, their raw scores kept in registers
    const uint32_t l = threadIdx.x;
    float kept[U];
    if(l < (uint32_t)kScoreLanes)
        {
            uint64_t m[U];
            int32_t nv[U], n[U];
#pragma unroll
            for(int k = 0; k < U; ++k)
                {
                    const uint32_t r = l + k * kScoreLanes;
                    if(r < p.regions)
                        {
                            m[k] = __ldcg(&p.marks[r]) | __ldcg(&p.newmarks[r]);
                            nv[k] = __ldcg(&p.valid[r]);
                            n[k] = __ldcg(&p.counter[r]);
                        }
                }
            // regions in increasing order: the lane's sum keeps its fixed order
            float acc = 0.0f;
#pragma unroll
            for(int k = 0; k < U; ++k)
                {
                    const uint32_t r = l + k * kScoreLanes;
                    if(r >= p.regions) break;
                    p.marks[r] = m[k];
                    p.newmarks[r] = 0ull;
                    kept[k] = raw_score(p, F, m[k], nv[k], n[k]);
                    acc = acc + scored(kept[k]);
                }
            lanes[l] = acc;
        }
    const float total = lanes_total(lanes);
    if(l < (uint32_t)kScoreLanes)
        {
#pragma unroll
            for(int k = 0; k < U; ++k)
                if(l + k * kScoreLanes < p.regions) p.score[l + k * kScoreLanes] = norm_score(p, kept[k], total);
        }
    if(threadIdx.x == 0) st.score_total = total;
}

// Slice `slice` of a larger table: its raw scores into the table, the
// iteration's new cells into the marks.  Four consecutive regions a thread and
// round, their counters in 16-byte loads (the tables start 256-byte aligned).
template <int NT, uint32_t SLICE>
__device__ __forceinline__ void score_slice(const ScoreParams& p, uint32_t slice)
{
    const float F = (float)p.fine_cells;
    const uint32_t end = min(p.regions, (slice + 1u) * SLICE);
    for(uint32_t r = slice * SLICE + threadIdx.x * 4u; r < end; r += NT * 4u)
        {
            if(r + 3 < end)
                {
                    const ulonglong2 ma = __ldcg((const ulonglong2*)(p.marks + r)), mb = __ldcg((const ulonglong2*)(p.marks + r) + 1);
                    const ulonglong2 wa = __ldcg((const ulonglong2*)(p.newmarks + r)), wb = __ldcg((const ulonglong2*)(p.newmarks + r) + 1);
                    const int4 nv = __ldcg((const int4*)(p.valid + r)), n = __ldcg((const int4*)(p.counter + r));
                    if(wa.x | wa.y | wb.x | wb.y)
                        {
                            *(ulonglong2*)(p.marks + r) = make_ulonglong2(ma.x | wa.x, ma.y | wa.y);
                            *((ulonglong2*)(p.marks + r) + 1) = make_ulonglong2(mb.x | wb.x, mb.y | wb.y);
                            *(ulonglong2*)(p.newmarks + r) = make_ulonglong2(0ull, 0ull);
                            *((ulonglong2*)(p.newmarks + r) + 1) = make_ulonglong2(0ull, 0ull);
                        }
                    *(float4*)(p.score + r) = make_float4(raw_score(p, F, ma.x | wa.x, nv.x, n.x), raw_score(p, F, ma.y | wa.y, nv.y, n.y),
                                                          raw_score(p, F, mb.x | wb.x, nv.z, n.z), raw_score(p, F, mb.y | wb.y, nv.w, n.w));
                }
            else
                for(uint32_t j = r; j < end; ++j)
                    {
                        const uint64_t m = __ldcg(&p.marks[j]) | __ldcg(&p.newmarks[j]);
                        p.marks[j] = m;
                        p.newmarks[j] = 0ull;
                        p.score[j] = raw_score(p, F, m, __ldcg(&p.valid[j]), __ldcg(&p.counter[j]));
                    }
        }
}

// total and normalisation of a table whose slices are all scored (by other
// blocks: read past L1), by one block
template <int NT>
__device__ __forceinline__ void score_finish(const ScoreParams& p, QueryState& st, float* lanes)
{
    constexpr int U = 32;  // loads in flight a thread
    for(int l = threadIdx.x; l < kScoreLanes; l += NT)
        {
            // regions l, l + 256, ... in order
            float acc = 0.0f;
            uint32_t r = (uint32_t)l;
            for(; r + (U - 1) * kScoreLanes < p.regions; r += U * kScoreLanes)
                {
                    float v[U];
#pragma unroll
                    for(int k = 0; k < U; ++k) v[k] = __ldcg(p.score + r + k * kScoreLanes);
#pragma unroll
                    for(int k = 0; k < U; ++k) acc = acc + scored(v[k]);
                }
            // (the rest in batches too: read one by one, 16^3 regions took 2.6 us longer)
            constexpr int W = 16;
            for(; r < p.regions; r += W * kScoreLanes)
                {
                    float v[W];
#pragma unroll
                    for(int k = 0; k < W; ++k) v[k] = r + k * kScoreLanes < p.regions ? __ldcg(p.score + r + k * kScoreLanes) : 0.0f;
#pragma unroll
                    for(int k = 0; k < W; ++k) acc = acc + scored(v[k]);
                }
            lanes[l] = acc;
        }
    const float total = lanes_total(lanes);
    constexpr int V = 8;  // 16-byte loads in flight a thread
    for(uint32_t r0 = threadIdx.x * 4u; r0 < p.regions; r0 += V * NT * 4u)
        {
            float4 v[V];
#pragma unroll
            for(int k = 0; k < V; ++k)
                if(r0 + k * NT * 4u + 3u < p.regions) v[k] = __ldcg((const float4*)(p.score + r0 + k * NT * 4u));
#pragma unroll
            for(int k = 0; k < V; ++k)
                {
                    const uint32_t r = r0 + k * NT * 4u;
                    if(r + 3u < p.regions)
                        *(float4*)(p.score + r) = make_float4(norm_score(p, v[k].x, total), norm_score(p, v[k].y, total),
                                                              norm_score(p, v[k].z, total), norm_score(p, v[k].w, total));
                    else
                        for(uint32_t j = r; j < p.regions; ++j) p.score[j] = norm_score(p, __ldcg(p.score + j), total);
                }
        }
    if(threadIdx.x == 0) st.score_total = total;
}

// ---------------------------------------------------------------------------
// append / re-activation / frontier build
// ---------------------------------------------------------------------------
__device__ inline void finalize_query(const QueryParams& p, QueryState& st, Sched* sched)
{
    // runs on one thread.  Every input is loaded in one round (the totals
    // were accumulated by other blocks' atomics, so past L1), then the new
    // state is computed in registers and stored.
    const uint32_t acc_total = __ldcg(&st.acc_total), n_next = __ldcg(&st.n_next);
    const int32_t goal_cand = __ldcg(&st.goal_cand);
    const uint32_t react_total = __ldcg(&st.react_total), w_total = __ldcg(&st.w_total);
    const uint32_t tree0 = __ldcg(&st.tree_size), drawn = __ldcg(&st.samples_drawn), ns = __ldcg(&st.n_samples);
    const uint32_t itr = __ldcg(&st.itr);
    const uint32_t max_it = p.max_iterations, cap = p.capacity, spn = p.samples_per_node;
    if(acc_total != n_next) atomicOr(&sched->error, kErrAppendMismatch);
    const uint32_t tree = tree0 + acc_total;
    uint32_t status = KGMT_QUERY_RUNNING;
    if(goal_cand != INT_MAX) status = KGMT_QUERY_SUCCESS;
    else if(itr >= max_it) status = KGMT_QUERY_ITER_LIMIT;
    else if(tree >= cap) status = KGMT_QUERY_CAPACITY;
    st.tree_size = tree;
    st.samples_drawn = drawn + ns;
    // the next frontier's list lengths (kept for a finished query too: the
    // traced plan reports its last frontier)
    st.n_react = react_total;
    st.w_new = w_total;
    // per-iteration accumulators start from zero next iteration
    st.tiles_done = 0;
    st.react_total = 0;
    st.acc_total = 0;
    st.w_total = 0;
    st.goal_cand = INT_MAX;
    if(status != KGMT_QUERY_RUNNING)
        {
            st.status = status;
            if(status == KGMT_QUERY_SUCCESS) st.goal_index = goal_cand;
            st.t_end = globaltimer();
            return;
        }
    st.itr = itr + 1;
    st.n_next = 0;
    uint32_t spe, n_samples;
    plan_samples_vals(cap, spn, tree, react_total + w_total, &spe, &n_samples);
    st.spe = spe;
    st.n_samples = n_samples;
    // the next schedule's totals (it sizes the tiles from them)
    atomicAdd(&sched->next_samples, (unsigned long long)n_samples);
    atomicAdd(&sched->next_tree, (unsigned long long)tree);
}

// Copies one sample row (written by the propagate kernel, read-only here)
// into the tree and returns its goal distance.  The row is read into
// registers before the first store: the two buffers might alias as far as
// the compiler can tell, so interleaved loads would each wait for the
// previous store's turn.
template <int D, bool COHERENT = false>
__device__ __forceinline__ float append_row_d(const QueryParams& p, const float* src, float* dst)
{
    float r[D];
    load_row_ro<D, COHERENT>(src, r);
    store_row<D>(dst, r);
    return goal_distance(p, r);
}

template <bool COHERENT = false>
__device__ __forceinline__ float append_row(const QueryParams& p, const float* src, float* dst, int D)
{
    switch(D)
        {
            case 7: return append_row_d<7, COHERENT>(p, src, dst);
            case 17: return append_row_d<17, COHERENT>(p, src, dst);
            default: return append_row_d<10, COHERENT>(p, src, dst);
        }
}

// KGMT.cu:387-388
__device__ __forceinline__ float f_accept_vals(uint32_t capacity, float epsilon, uint32_t tree_size, uint32_t n_next, uint32_t itr)
{
    const float ta = 1.0f - (float)(tree_size + n_next) / (float)capacity;
    const float ie = (float)itr * epsilon;
    const double t = (double)ta;
    const double t5 = ((t * t) * (t * t)) * t;
    return (float)((double)ie * t5);
}

__device__ __forceinline__ float f_accept_of(const QueryParams& p, const QueryState& st)
{
    return f_accept_vals(p.capacity, p.epsilon, st.tree_size, st.n_next, st.itr);
}


}  // namespace kgmt
