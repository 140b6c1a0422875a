// kgmt_kernels.cu -- the per-iteration kernel chain of the KGMT planning loop.
//
// One iteration of every running query (reference: KGMT::plan loop body,
// src/planners/KGMT.cu:84-95) is three launches with fixed shapes (four where a
// query has a large region table), so the chain can be captured once in a CUDA
// graph and replayed:
//
//   k_propagate  KGMT::propagateFrontier + propagateFrontier_kernel1/2
//                (KGMT.cu:167-299): one thread per sample, persistent blocks
//                taking propagate tiles from a ticket counter, obstacles of
//                the tile's query staged in shared memory by a bulk (TMA)
//                copy, one tile ahead; warp-aggregated counts.
//   k_score      raw region scores of large tables, in slices.
//   k_score_sum  Graph::updateVertices (Graph.cu:207-358): the other tables'
//                scores; sums in a fixed order, normalisation.
//   k_append     KGMT::updateFrontier + updateFrontier_kernel
//                (KGMT.cu:305-403) and the next iteration's frontier
//                compaction / repeat expansion (KGMT.cu:167-181,
//                Planner.cu:52-79): ordered stream compaction with
//                decoupled look-back gives every accepted sample its tree
//                index (an order-preserving "atomic append") and every
//                re-activated node its frontier slot; the last tile of a
//                query finalises it, the last query computes the schedule of
//                the next iteration on the device.
//
// Before the first iteration k_begin (one query) or k_admit and k_build_grid lay
// out a query; k_tail (kgmt_tail.cuh) runs the iterations of few and small
// queries in one launch; k_paths reads the found paths out.
//
// Frontier representation: instead of frontier flags over the whole tree and
// two scans per iteration (KGMT.cu:170-181), the frontier of the next
// iteration is built directly as two index lists -- re-activated old nodes
// (repeat 1) followed by the nodes appended this iteration (repeat 15 or 1) --
// which is the order the reference's scan over node indices produces.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <climits>
#include <type_traits>

#include "kgmt_iter.cuh"
#include "kgmt_tail.cuh"

namespace kgmt {

// ---------------------------------------------------------------------------
// decoupled look-back over one chain of tiles of one query.  Word layout:
// bits 62-63 status (0 empty, 1 aggregate, 2 inclusive prefix), bits 0-61 the
// value (the chains pack their counts so that sums never carry into the
// status bits).  Tiles are taken in ticket order, so every predecessor is
// held by a resident block; waits are bounded all the same.
// ---------------------------------------------------------------------------
constexpr unsigned long long kStAgg = 1ull << 62;
constexpr unsigned long long kStIncl = 2ull << 62;
constexpr unsigned long long kValMask = (1ull << 62) - 1;

// Called by one full warp; lane i inspects predecessor lt-1-i, 32 at a time,
// until the nearest inclusive prefix; every nearer predecessor must have
// published at least its aggregate.  Returns the exclusive prefix on all lanes.
// After `limit` polls without progress it records kErrLookbackTimeout in
// *error and returns (the host reports KGMT_ERR_TIMEOUT).
__device__ unsigned long long lookback_warp(unsigned long long* tiles, int lt, uint32_t* error, uint32_t limit = kSpinLimit)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned long long prefix = 0;
    int base = lt - 1;
    uint32_t spins = 0;
    while(base >= 0)
        {
            const int j = base - lane;
            const unsigned long long w = j >= 0 ? ld_volatile_u64(&tiles[j]) : kStIncl;  // before tile 0: inclusive 0
            const unsigned st = (unsigned)(w >> 62);
            const unsigned incl = __ballot_sync(full, st == 2u);
            const unsigned not_ready = __ballot_sync(full, st == 0u);
            const int stop = incl ? __ffs(incl) - 1 : 31;  // nearest inclusive lane (or the whole window)
            const unsigned upto = stop == 31 ? full : ((2u << stop) - 1u);
            if(not_ready & upto)
                {
                    if(++spins > limit)
                        {
                            if(lane == 0) atomicOr(error, kErrLookbackTimeout);
                            return prefix;
                        }
                    __nanosleep(32);
                    continue;
                }
            unsigned long long v = lane <= stop ? (w & kValMask) : 0ull;
#pragma unroll
            for(int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(full, v, o);
            prefix += v;
            if(incl) break;
            base -= 32;
        }
    return prefix;
}

// Tile lt of a chain with block aggregate `agg`: publishes the aggregate,
// resolves the exclusive prefix (warp 0), publishes the inclusive prefix and
// leaves the exclusive prefix in *s_prefix.  Block-uniform call; the caller
// synchronises before reading *s_prefix.
__device__ __forceinline__ void publish_and_lookback(unsigned long long* tiles, uint32_t lt, unsigned long long agg,
                                                     unsigned long long* s_prefix, uint32_t* error)
{
    if(threadIdx.x >= 32) return;
    if(lt == 0)
        {
            if(threadIdx.x == 0)
                {
                    st_volatile_u64(&tiles[0], kStIncl | agg);
                    *s_prefix = 0;
                }
            return;
        }
    if(threadIdx.x == 0) st_volatile_u64(&tiles[lt], kStAgg | agg);
    __syncwarp();
    const unsigned long long prefix = lookback_warp(tiles, (int)lt, error);
    if(threadIdx.x == 0)
        {
            st_volatile_u64(&tiles[lt], kStIncl | (prefix + agg));
            *s_prefix = prefix;
        }
}

// Failure-detection self-test: the look-back wait of tile 1 of a chain whose
// tile 0 never publishes (a word nothing sets), with a short poll limit; it
// must give up, record the timeout and return.  One warp.
__global__ void k_selftest_wait(unsigned long long* tiles, uint32_t* error, uint32_t polls)
{
    lookback_warp(tiles, 1, error, polls);
}

uint32_t bounds_error_take()
{
#ifdef KGMT_CHECK_BOUNDS
    uint32_t v = 0, z = 0;
    if(cudaMemcpyFromSymbol(&v, g_bounds_error, sizeof(v)) != cudaSuccess) return kErrBounds;
    cudaMemcpyToSymbol(g_bounds_error, &z, sizeof(z));
    return v;
#else
    return 0u;
#endif
}

cudaError_t launch_selftest_wait(unsigned long long* tiles, uint32_t* error, uint32_t polls, cudaStream_t s)
{
    k_selftest_wait<<<1, 32, 0, s>>>(tiles, error, polls);
    return cudaGetLastError();
}

// rows of 2W floats (min corner, max corner; W = 3, or 2 for the planar
// model, whose z extents are then 0 and never tested) -> float4 pairs
__device__ __forceinline__ void stage_box(const float* r, int w, float4* dst)
{
    if(w == 2)
        {
            dst[0] = make_float4(r[0], r[1], 0.0f, 0.0f);
            dst[1] = make_float4(r[2], r[3], 0.0f, 0.0f);
        }
    else
        {
            dst[0] = make_float4(r[0], r[1], r[2], 0.0f);
            dst[1] = make_float4(r[3], r[4], r[5], 0.0f);
        }
}

// region tables and look-back words of a query at zero: this thread's share,
// t of nt
__device__ __forceinline__ void clear_tables(const QueryParams& p, uint32_t t, uint32_t nt)
{
    for(uint32_t r = t; r < p.regions; r += nt)
        {
            p.counter[r] = 0;
            p.valid[r] = 0;
            p.score[r] = 0.0f;
            p.marks[r] = 0ull;
            p.newmarks[r] = 0ull;
        }
    for(uint32_t i = t; i < p.tiles_per_chain; i += nt)
        {
            p.tiles_old[i] = 0ull;
            p.tiles_slot[i] = 0ull;
        }
}

// the root node, the first frontier (root x5) and the loop state of a query;
// by one block
__device__ __forceinline__ void admit_root(const QueryParams& p, QueryState& out)
{
    for(uint32_t j = threadIdx.x; j < p.sample_dim; j += blockDim.x) p.tree[j] = p.init[j];
    if(threadIdx.x < kRootRepeat) p.rep_new[threadIdx.x] = 0u;
    if(threadIdx.x == 0)
        {
            p.parent[0] = -1;
            p.cost[0] = 0.0f;
            p.node_r1[0] = region_of(p, p.init);
            QueryState st = {};
            st.status = KGMT_QUERY_RUNNING;
            st.itr = 1;
            st.tree_size = 1;
            st.n_react = 0;
            st.w_new = kRootRepeat;
            st.goal_cand = INT_MAX;
            st.goal_index = -1;
            st.steps = 0;
            st.tests = 0;
            st.path_at = kNoPath;
            st.t_start = globaltimer();
            plan_samples(p, st);
            out = st;
        }
}

// ---------------------------------------------------------------------------
// admission: root node, cleared region tables, first frontier (root x5); the
// slots are [first, first + count), or slots[0 .. count) when a list is given
// ---------------------------------------------------------------------------
__global__ void k_admit(const QueryParams* __restrict__ P, QueryState* S, uint32_t first, uint32_t count, const uint32_t* __restrict__ slots)
{
    if(blockIdx.x >= count) return;
    const uint32_t q = slots ? slots[blockIdx.x] : first + blockIdx.x;
    const QueryParams& p = P[q];
    if(p.raw_obstacles)
        for(uint32_t o = threadIdx.x; o < p.n_obstacles; o += blockDim.x)
            stage_box(p.raw_obstacles + (size_t)o * 2 * p.raw_w, p.raw_w, p.obstacles + 2 * o);
    clear_tables(p, threadIdx.x, blockDim.x);
    admit_root(p, S[q]);
}

// ---------------------------------------------------------------------------
// Obstacle culling grid of n boxes, built by one block: count boxes per cell,
// scan, fill.  A box is listed in every cell of [cell(min), cell(max)] per
// axis (ordered, so an inverted box is still covered).  NaN coordinates, more
// boxes than 16-bit indices hold, or more entries than `budget` leave the grid
// unusable (false), and every box is tested.
// ---------------------------------------------------------------------------
// The cells' 16-bit counters (two a word) become the fill cursors in place,
// and a filled cell's cursor is the start of the next one: with a zero before
// the first, they are the CSR starts.  Where that takes fewer or shorter rounds,
// four lanes share a box, an x slice each: a lane's chain of shared-memory atomics
// on a box's 8 to 30 cells is the longest part of a small build.  More boxes get a
// lane each: they are smaller, and lanes beyond a box's slices idle.  (49,999 Dubins
// samples, blocks of 128: 80 boxes 17.2 us by four lanes, 17.6 by one; 100 boxes 18.4,
// 17.7; 160 boxes 21.0, 23.3; 256 boxes 24.3, 21.8; 640 boxes 37.0, 25.2.  A plan's first
// iteration with 10,000 boxes 281, 147.)
constexpr uint32_t kGridBuildBytes = 16 + kGridCells * 2;  // shared memory of a build
// The grids of batches, which count their box tests, list the boxes of a cell in
// increasing order when they have at most kGridOrdered of them in at most
// kGridOrderedItems entries: how many tests a step makes before its first hit then
// depends on the scene alone, not on which warp filled the cell first.  The lists
// are filled in shared memory and written out by rank (256 queries of 50 boxes: 10 us
// unordered, 16 ordered).
constexpr uint32_t kGridOrdered = 256;
constexpr uint32_t kGridOrderedItems = 8192;

// calls f(o, cell) for the cells of the boxes o, this thread's share of them;
// true when a box has a NaN coordinate (its cells are skipped)
template <bool GLOBAL, typename F>
__device__ __forceinline__ bool for_box_cells(const QueryParams& p, const float4* obs, uint32_t n, F&& f)
{
    constexpr int G = (int)kGridDim;
    // log2 of the lanes a box: a round of four lanes a box takes 5/16 of one of a lane
    const uint32_t sh = 5u * ((n * 4u + blockDim.x - 1u) / blockDim.x) < 16u * ((n + blockDim.x - 1u) / blockDim.x) ? 2u : 0u;
    const uint32_t step = blockDim.x >> sh;
    bool bad = false;
    // in global memory the next box is on its way while this one's cells are counted
    // (64 queries of 10,000 boxes, admission and an iteration: 432 us without, 411 with)
    uint32_t o = threadIdx.x >> sh;
    float4 na = make_float4(0.0f, 0.0f, 0.0f, 0.0f), nb = na;
    if(GLOBAL && o < n) na = obs[2 * o], nb = obs[2 * o + 1];
#pragma unroll 1
    for(; o < n; o += step)
        {
            if(!GLOBAL) na = obs[2 * o], nb = obs[2 * o + 1];
            const float4 a = na, b = nb;
            if(GLOBAL && o + step < n) na = obs[2 * (o + step)], nb = obs[2 * (o + step) + 1];
            if(isnan(a.x) || isnan(a.y) || isnan(a.z) || isnan(b.x) || isnan(b.y) || isnan(b.z))
                {
                    bad = true;
                    continue;
                }
            const int x0 = grid_cell(p, fminf(a.x, b.x)), x1 = grid_cell(p, fmaxf(a.x, b.x));
            const int y0 = grid_cell(p, fminf(a.y, b.y)), y1 = grid_cell(p, fmaxf(a.y, b.y));
            const int z0 = p.planar ? 0 : grid_cell(p, fminf(a.z, b.z)), z1 = p.planar ? 0 : grid_cell(p, fmaxf(a.z, b.z));
#pragma unroll 1
            for(int cx = x0 + (int)(threadIdx.x & ((1u << sh) - 1u)); cx <= x1; cx += 1 << sh)
#pragma unroll 1
                for(int cy = y0; cy <= y1; ++cy)
                    for(int cz = z0; cz <= z1; ++cz) f(o, (cx * G + cy) * G + cz);
        }
    return bad;
}

// mem: kGridBuildBytes of shared memory, 16-byte aligned; scratch: 34 words;
// items: shared or global memory; listed: kGridOrderedItems of shared memory, or
// null (the order inside a cell is not kept).  All threads of the block (128 or
// 256) must enter.  Returns the starts (kGridCells + 1 of them, inside mem; starts and
// items are complete: the build ends with a block barrier), or nullptr when
// the grid is unusable; *total gets the entries.
// GLOBAL: the boxes are in global memory (else staged).
template <bool GLOBAL>
__device__ __forceinline__ const uint16_t* build_grid(const QueryParams& p, const float4* obs, uint32_t n, uint32_t budget, char* mem,
                                                      uint32_t* scratch, uint16_t* items, uint32_t* total, uint16_t* listed = nullptr)
{
    __shared__ int s_bad;
    uint32_t* cursor = (uint32_t*)(mem + 16);  // cell c: half c & 1 of word c / 2
    for(uint32_t i = threadIdx.x; i < kGridBuildBytes / 16; i += blockDim.x) ((uint4*)mem)[i] = make_uint4(0u, 0u, 0u, 0u);
    if(threadIdx.x < 34) scratch[threadIdx.x] = 0u;
    if(threadIdx.x == 0) s_bad = n > kMaxObstacles ? 1 : 0;
    __syncthreads();
    const uint32_t boxes = n > kMaxObstacles ? 0u : n;
    if(for_box_cells<GLOBAL>(p, obs, boxes, [&](uint32_t, int c) { atomicAdd(&cursor[c >> 1], 1u << ((c & 1) * 16)); })) s_bad = 1;
    __syncthreads();
    // counts -> exclusive prefixes; a thread owns 16 (or, of 128, 32)
    // consecutive cells.  Pairs of 16-bit counts are summed in 32 bits.
    const uint32_t words16 = kGridCells / 8 / blockDim.x;
    uint4* own = (uint4*)cursor + threadIdx.x * words16;
    uint32_t local = 0;
    for(uint32_t i = 0; i < words16; ++i)
        {
            const uint4 v = own[i];
            local += (v.x & 0xffffu) + (v.x >> 16) + (v.y & 0xffffu) + (v.y >> 16) + (v.z & 0xffffu) + (v.z >> 16) + (v.w & 0xffffu) + (v.w >> 16);
        }
    uint32_t run = block_exclusive_scan<256>(local, scratch, total);
    if(s_bad || *total > budget || *total > kMaxGridItems) return nullptr;
    for(uint32_t i = 0; i < words16; ++i)
        {
            uint4 v = own[i];
            auto prefix = [&](uint32_t w) {
                const uint32_t lo = run, hi = run + (w & 0xffffu);
                run = hi + (w >> 16);
                return lo | (hi << 16);
            };
            v.x = prefix(v.x), v.y = prefix(v.y), v.z = prefix(v.z), v.w = prefix(v.w);
            own[i] = v;
        }
    __syncthreads();
    const bool ordered = listed && boxes <= kGridOrdered && *total <= kGridOrderedItems;
    uint16_t* const fill = ordered ? listed : items;
    for_box_cells<GLOBAL>(p, obs, boxes, [&](uint32_t o, int c) {
        const int sh = (c & 1) * 16;
        fill[(atomicAdd(&cursor[c >> 1], 1u << sh) >> sh) & 0xffffu] = (uint16_t)o;
    });
    if(ordered)
        {
            __syncthreads();
            const uint16_t* start = (const uint16_t*)cursor - 1;
            constexpr uint32_t kShort = 6;  // a thread's own cell up to here, a warp's above
            const uint32_t lane = threadIdx.x & 31u;
            for(uint32_t c0 = threadIdx.x & ~31u; c0 < kGridCells; c0 += blockDim.x)
                {
                    const uint32_t at = start[c0 + lane], k = start[c0 + lane + 1u] - at;
                    for(uint32_t i = 0; i < k && k <= kShort; ++i)
                        {
                            const uint16_t v = listed[at + i];
                            uint32_t rank = 0;
                            for(uint32_t j = 0; j < k; ++j) rank += listed[at + j] < v ? 1u : 0u;
                            items[at + rank] = v;
                        }
                    for(unsigned more = __ballot_sync(0xffffffffu, k > kShort); more; more &= more - 1u)
                        {
                            const int from = __ffs((int)more) - 1;
                            const uint32_t ca = __shfl_sync(0xffffffffu, at, from), ck = __shfl_sync(0xffffffffu, k, from);
                            for(uint32_t i = lane; i < ck; i += 32u)
                                {
                                    const uint16_t v = listed[ca + i];
                                    uint32_t rank = 0;
                                    for(uint32_t j = 0; j < ck; ++j) rank += listed[ca + j] < v ? 1u : 0u;
                                    items[ca + rank] = v;
                                }
                        }
                }
        }
    __syncthreads();
    return (const uint16_t*)cursor - 1;
}

// the culling grid of one query per block
__global__ void __launch_bounds__(256) k_build_grid(const QueryParams* __restrict__ P, uint32_t first, uint32_t count,
                                                    const uint32_t* __restrict__ slots)
{
    __shared__ alignas(16) char mem[kGridBuildBytes];
    __shared__ uint16_t listed[kGridOrderedItems];
    __shared__ uint32_t scratch[34];
    if(blockIdx.x >= count) return;
    const QueryParams& p = P[slots ? slots[blockIdx.x] : first + blockIdx.x];
    if(p.grid_start == nullptr) return;
    uint32_t total = 0;
    const uint16_t* start = build_grid<true>(p, p.obstacles, p.n_obstacles, p.grid_budget, mem, scratch, p.grid_items, &total, listed);
    if(start)
        for(uint32_t c = threadIdx.x; c <= kGridCells; c += 256) p.grid_start[c] = start[c];
    if(threadIdx.x == 0)
        {
            p.grid_meta[0] = total;
            p.grid_meta[1] = start ? 1u : 0u;
        }
}

__global__ void k_schedule(const QueryParams* __restrict__ P, const QueryState* __restrict__ S, Sched* sched, uint32_t* tile_a_base,
                           uint32_t* tile_c_base, uint32_t* tile_c_old)
{
    compute_schedule(P, S, sched, tile_a_base, tile_c_base, tile_c_old);
}

// Admission of an engine's only query: what k_stage_obstacles, the params
// upload, k_set_n_slots, k_admit, k_build_grid and k_schedule do in six stream
// operations.  Block 0 takes the query (its build of
// the grid is the longest part), the other blocks clear the region tables.  A
// single plan's first iteration starts about 10 us after the call's first
// launch instead of 45.
__global__ void __launch_bounds__(256) k_begin(const __grid_constant__ QueryParams p, const LaunchArgs a)
{
    __shared__ alignas(16) char mem[kGridBuildBytes];
    __shared__ uint32_t scratch[34];
    if(blockIdx.x > 0)
        {
            clear_tables(p, (blockIdx.x - 1) * blockDim.x + threadIdx.x, (gridDim.x - 1) * blockDim.x);
            return;
        }
    QueryParams* dst = const_cast<QueryParams*>(a.params);
    for(uint32_t i = threadIdx.x; i < sizeof(QueryParams) / 4; i += blockDim.x) ((uint32_t*)dst)[i] = ((const uint32_t*)&p)[i];
    static_assert(sizeof(QueryParams) % 4 == 0 && sizeof(QueryState) % 8 == 0, "copied by words");
    if(p.raw_obstacles)  // (else they are staged)
        for(uint32_t o = threadIdx.x; o < p.n_obstacles; o += blockDim.x)
            stage_box(p.raw_obstacles + (size_t)o * 2 * p.raw_w, p.raw_w, p.obstacles + 2 * o);
    admit_root(p, a.states[0]);
    if(threadIdx.x == 0)
        {
            a.sched->n_slots = 1;
            a.sched->path_words = 0;
        }
    __syncthreads();
    if(threadIdx.x == 0) dst->raw_obstacles = nullptr;  // the caller's array: not kept past this launch
    if(p.grid_start != nullptr)
        {
            uint32_t total = 0;
            const uint16_t* start = build_grid<true>(p, p.obstacles, p.n_obstacles, p.grid_budget, mem, scratch, p.grid_items, &total);
            if(start)
                for(uint32_t c = threadIdx.x; c <= kGridCells; c += blockDim.x) p.grid_start[c] = start[c];
            if(threadIdx.x == 0)
                {
                    p.grid_meta[0] = total;
                    p.grid_meta[1] = start ? 1u : 0u;
                }
        }
    compute_schedule(a.params, a.states, a.sched, a.tile_a_base, a.tile_c_base, a.tile_c_old);
}

// Blocks per SM the registers are shared out for: 24 warps (80 registers) for the
// models with short steps, 16 (128) where the quadrotor may be met.  256
// double-integrator / Dubins / unicycle queries in blocks of 256: 3 blocks an SM
// 2.69 / 2.76 / 0.455 ms of propagate launches, 4 (64 registers, some spilled) 2.76 /
// 2.77 / 0.474, 2 - / 3.00 / 0.494; in blocks of 512 the double integrator takes
// two (one: 3.47 against 2.87).
template <int NT, int MODELS>
constexpr int propagate_blocks()
{
    if(NT == 512) return MODELS == kBitDI ? 2 : 1;
    return (MODELS == kBitDI || MODELS == kBitDubins || MODELS == kBitUnicycle ? 768 : 512) / NT;
}

template <int NT, int MODELS>
__global__ void __launch_bounds__(NT, propagate_blocks<NT, MODELS>()) k_propagate(const QueryParams* __restrict__ P, QueryState* S, Sched* sched,
                                                  const uint32_t* __restrict__ tile_base, uint32_t smem_boxes)
{
    // dynamic shared memory of each of the two buffers: grid starts | grid
    // items | grid meta | boxes (smem_boxes of them; a query with more reads
    // its boxes from global memory)
    extern __shared__ float4 s_dyn[];
    __shared__ TileBuf<NT> s_buf[2];
    __shared__ volatile uint32_t s_ready[2];  // 1 + the number of the block's tile in the buffer, or kEnd
    __shared__ uint32_t s_base[kBaseCache];
    constexpr uint32_t kEnd = 0xFFFFFFFFu, NW = NT / 32;
    // everything here depends on the append kernel before this one (its
    // schedule, frontier and tree); once that is complete the append kernel
    // after this one may be scheduled into the SMs this launch leaves free
    pdl_wait();
    pdl_trigger();
    if(blockIdx.x == 0 && threadIdx.x == 0)
        {
            // counters of the append kernel that follows this one
            sched->ticket_c = 0;
            sched->finalized = 0;
        }
    const uint32_t total = sched->tiles_a;
    const int n_slots = (int)sched->n_slots;
    // samples per tile this iteration (the schedule sized the tiles)
    const uint32_t tile = sched->prop_tile;
    const uint32_t* order = sched->prop_order;
    if(blockIdx.x >= total) return;
    if(threadIdx.x == 0)
        {
            mbar_init(&s_buf[0].bar, 1);
            mbar_init(&s_buf[1].bar, 1);
            s_ready[0] = 0, s_ready[1] = 0;
            s_buf[1].units = 1;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    const BaseCache bases = cache_bases(tile_base, n_slots, s_base);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    auto dyn = [&](uint32_t i) { return (char*)s_dyn + (i & 1u) * (prop_smem_bytes(smem_boxes) / 2); };
    // the block's tile number i, tile t of the iteration; by one warp
    auto prepare = [&](uint32_t i, uint32_t t) {
        if(t < total)
            {
                const int at = find_slot(bases.base, bases.n, t);
                prepare_tile<NT, MODELS, false>(s_buf[i & 1u], dyn(i), P, S, order ? (int)order[at] : at, t - bases.base[at], tile, smem_boxes);
            }
        __syncwarp();
        if(lane == 0)
            {
                __threadfence_block();
                s_ready[i & 1u] = t < total ? i + 1u : kEnd;
            }
    };
    // first tile static, then tickets
    auto ticket = [&] {
        uint32_t t = 0;
        if(lane == 0) t = gridDim.x + atomicAdd(&sched->ticket_a, 1u);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    {
        const int at = find_slot(bases.base, bases.n, blockIdx.x);
        prepare_tile<NT, MODELS, true>(s_buf[0], dyn(0), P, S, order ? (int)order[at] : at, blockIdx.x - bases.base[at], tile, smem_boxes);
    }
    if(threadIdx.x == 0) s_ready[0] = 1u;
    __syncthreads();
    if(warp == 0) prepare(1, ticket());
    for(uint32_t i = 0;; ++i)
        {
            TileBuf<NT>& B = s_buf[i & 1u];
            uint32_t r = 0;
            if(lane == 0)
                {
                    // what keeps the tile is the last warp in the buffer's tile
                    // before, with one run of it at most (its units are still
                    // there, or those of the tile that is now being prepared)
                    uint32_t spins = 0, units = *(volatile uint32_t*)&B.units;
                    while((r = s_ready[i & 1u]) != i + 1u && r != kEnd)
                        {
                            if(++spins > kSpinLimit)
                                {
                                    spins = 0;
                                    if(--units == 0u)
                                        {
                                            atomicOr(&sched->error, kErrCopyTimeout);
                                            r = kEnd;
                                            break;
                                        }
                                }
                            __nanosleep(20);
                        }
                    __threadfence_block();
                }
            if(__shfl_sync(0xffffffffu, r, 0) == kEnd) break;
            __syncwarp();
            run_tile<NT, MODELS>(B, dyn(i), smem_boxes, (i >> 1) & 1u, &sched->error);
            // the last warp to leave has the whole tile behind it
            __syncwarp();
            uint32_t last = 0;
            if(lane == 0)
                {
                    __threadfence_block();
                    last = atomicAdd(&B.left, 1u) == NW - 1u;
                    if(last)
                        {
                            __threadfence_block();
                            QueryState& st = S[B.q];
                            if(B.sh.acc) atomicAdd(&st.n_next, B.sh.acc);
                            if(B.sh.steps) atomicAdd(&st.steps, (unsigned long long)B.sh.steps);
                            if(B.sh.tests) atomicAdd(&st.tests, (unsigned long long)B.sh.tests);
                        }
                }
            last = __shfl_sync(0xffffffffu, last, 0);
            __syncwarp();
            if(last) prepare(i + 2u, ticket());
        }
}

// Region scores, between the propagate and the append launch.  k_score (only in
// chains with a query of more than kScoreSmall regions): raw scores of the large
// tables, their slices round the blocks.  k_score_sum: one block a query scores a
// small table whole, or sums and normalises a large one.  Bound by L2 and DRAM
// latency.  As one launch in which the block that finished a query's last slice
// summed it, 190 queries of up to 32^3 regions took 75 us (some blocks summed
// three of them), now 22 + 16.  (Small tables scored by the propagate block that
// finished the query held that block's next tile up.)  The blocks per SM leave
// each kernel the registers it does not spill.
constexpr int kScoreThreads = 128;
constexpr int kScoreBlocksPerSm = 8;
constexpr int kSumThreads = 384;
constexpr int kSumBlocksPerSm = 2;

// whether slot i has a large table to score in this iteration (the schedule's
// values, complete before the propagate kernel let this launch start)
__device__ __forceinline__ bool has_large_table(const QueryParams* P, const QueryState* S, uint32_t i)
{
    return S[i].status == KGMT_QUERY_RUNNING && S[i].n_samples > 0 && P[i].regions > kScoreSmall;
}

__global__ void __launch_bounds__(kScoreThreads, kScoreBlocksPerSm) k_score(const QueryParams* __restrict__ P, const QueryState* S,
                                                                           const Sched* sched)
{
    __shared__ uint32_t scratch[34];
    __shared__ uint32_t s_pre[kScoreThreads + 1];  // first slice of each slot of the group
    // what the propagate kernel counts is read only past the wait (which every
    // block reaches)
    pdl_trigger();
    const uint32_t n_slots = sched->n_slots;
    bool waited = false;
    uint32_t before = 0;  // slices of earlier groups of slots
    for(uint32_t c0 = 0; c0 < n_slots; c0 += kScoreThreads)
        {
            const uint32_t i = c0 + threadIdx.x;
            const uint32_t slices = i < n_slots && has_large_table(P, S, i) ? (P[i].regions + kScoreSlice - 1) / kScoreSlice : 0u;
            uint32_t total;
            s_pre[threadIdx.x] = block_exclusive_scan<kScoreThreads>(slices, scratch, &total);
            if(threadIdx.x == 0) s_pre[kScoreThreads] = total;
            if(!waited) pdl_wait();
            waited = true;
            __syncthreads();
            for(uint32_t j = (blockIdx.x + gridDim.x - before % gridDim.x) % gridDim.x; j < total; j += gridDim.x)
                {
                    const int g = find_slot(s_pre, kScoreThreads, j);
                    score_slice<kScoreThreads, kScoreSlice>(score_params(P[c0 + (uint32_t)g]), j - s_pre[g]);
                }
            before += total;
            __syncthreads();
        }
    if(!waited) pdl_wait();
}

__global__ void __launch_bounds__(kSumThreads, kSumBlocksPerSm) k_score_sum(const QueryParams* __restrict__ P, QueryState* S, const Sched* sched)
{
    __shared__ float s_lanes[kScoreLanes];
    pdl_trigger();
    const uint32_t n_slots = sched->n_slots;
    bool waited = false;
    for(uint32_t q = blockIdx.x; q < n_slots; q += gridDim.x)
        {
            if(S[q].status != KGMT_QUERY_RUNNING || S[q].n_samples == 0) continue;
            const ScoreParams sp = score_params(P[q]);
            if(!waited) pdl_wait();
            waited = true;
            if(sp.regions > kScoreSmall) score_finish<kSumThreads>(sp, S[q], s_lanes);
            else update_scores<kSumThreads>(sp, S[q], s_lanes);
            __syncthreads();
        }
    if(!waited) pdl_wait();
}

// eight blocks per SM (32 registers; the kernel waits on loads, scans and
// look-back, so more tiles in flight hide more latency: the mixed batch
// +4 %, the double-integrator batch unchanged)
__global__ void __launch_bounds__(kAppendThreads, 8) k_append(const QueryParams* __restrict__ P, QueryState* S, Sched* sched,
                                                           uint32_t* tile_a_base, uint32_t* tile_c_base, uint32_t* tile_c_old)
{
    __shared__ uint32_t scratch[34];
    __shared__ int s_tile, s_q, s_glob, s_fin;
    __shared__ unsigned long long s_prefix;
    __shared__ float s_fa;
    __shared__ uint32_t s_cbase[kBaseCache];
    __shared__ uint32_t s_cold[kBaseCache];
    const uint32_t total = sched->tiles_c;
    const int n_slots = (int)sched->n_slots;
    const uint32_t old_tile = sched->old_tile;
    if(blockIdx.x >= total) return;
    // this iteration's tile bases (the schedule rewrites the global arrays only
    // after every tile is done)
    const BaseCache cbase = cache_bases(tile_c_base, n_slots, s_cbase);
    const BaseCache cold = cache_bases(tile_c_old, n_slots - 1, s_cold);
    // the schedule and tile bases above come from the append kernel of the
    // iteration before (complete before this iteration's propagate kernel, and
    // through it the score kernels, let this one start); this iteration's
    // results are read only from here on
    pdl_wait();
    pdl_trigger();
    // First tile static, then tickets, taken only when the block is free: a
    // ticket taken ahead would hold a tile that its successors' look-back
    // waits for behind the block's current tile.
    uint32_t next = blockIdx.x;
    for(;;)
        {
            if(threadIdx.x == 0)
                {
                    const uint32_t t = next;
                    s_tile = (int)t;
                    s_q = t < total ? find_slot(cbase.base, cbase.n, t) : -1;
                    s_glob = 0;
                    s_fin = 0;
                    if(t < total) s_fa = f_accept_of(P[s_q], S[s_q]);
                }
            __syncthreads();
            const uint32_t t = (uint32_t)s_tile;
            if(t >= total) break;
            const int q = s_q;
            const QueryParams& p = P[q];
            QueryState& st = S[q];
            const uint32_t lt = t - cbase.base[q];
            const uint32_t n_old = cold.base[q];
            const uint32_t itr = st.itr;
            const uint32_t tree_size = st.tree_size;
            if(lt < n_old)
                {
                    // ---- re-activation of old nodes (KGMT.cu:364-377) ----
                    // old_tile / kAppendThreads consecutive nodes a thread (4,
                    // 16 or 32), in rounds of at most kOldPer
                    const uint32_t per_t = old_tile / kAppendThreads;
                    const uint32_t i0 = lt * old_tile + threadIdx.x * per_t;
                    const float fa = s_fa;
                    const uint32_t k0 = (uint32_t)p.seed, k1 = (uint32_t)(p.seed >> 32);
                    uint32_t flags = 0, cnt = 0;
                    static_assert(kOldPer % 4 == 0 && kTileOldLarge / kAppendThreads <= 32, "re-activation: 4-node loads, one flag bit per node");
                    // one round: kOldPer nodes from i0 + r0 -- their regions
                    // four at a time (i0 + r0 is a multiple of 4: the 16-byte
                    // loads are aligned), then the region scores
                    auto round = [&](uint32_t r0) {
                        int32_t reg[kOldPer];
#pragma unroll
                        for(int g = 0; g < kOldPer; g += 4)
                            {
                                const uint32_t ib = i0 + r0 + g;
                                if(r0 + g >= per_t) reg[g] = reg[g + 1] = reg[g + 2] = reg[g + 3] = 0;
                                else if(ib + 3 < tree_size)
                                    {
                                        const int4 v = *(const int4*)(p.node_r1 + ib);
                                        reg[g] = v.x, reg[g + 1] = v.y, reg[g + 2] = v.z, reg[g + 3] = v.w;
                                    }
                                else
                                    {
#pragma unroll
                                        for(int j = 0; j < 4; ++j) reg[g + j] = ib + j < tree_size ? p.node_r1[ib + j] : 0;
                                    }
                            }
#pragma unroll
                        for(int j = 0; j < kOldPer; ++j)
                            {
                                const uint32_t i = i0 + r0 + j;
                                if(r0 + j < per_t && i < tree_size)
                                    {
                                        const U4 r = philox4x32_10(i, itr, 1u, 0u, k0, k1);
                                        const float ur = u01(r.x);
                                        if(ur <= p.score[reg[j]] + fa)
                                            {
                                                flags |= 1u << (r0 + j);
                                                ++cnt;
                                            }
                                    }
                            }
                    };
                    round(0u);
                    if(per_t > (uint32_t)kOldPer) round((uint32_t)kOldPer);
                    uint32_t agg;
                    const uint32_t excl = block_exclusive_scan<kAppendThreads>(cnt, scratch, &agg);
                    publish_and_lookback(p.tiles_old, lt, agg, &s_prefix, &sched->error);
                    if(threadIdx.x == 0) atomicAdd(&st.react_total, agg);
                    __syncthreads();
                    uint32_t pos = (uint32_t)s_prefix + excl;
                    for(uint32_t m = flags; m; m &= m - 1u)
                        {
                            if(KGMT_BOUND(pos < p.capacity)) p.rep_old[pos] = i0 + (uint32_t)(__ffs((int)m) - 1);
                            ++pos;
                        }
                }
            else
                {
                    // ---- ordered append of accepted samples (KGMT.cu:317-362) ----
                    // kAppendPer consecutive samples a thread: their
                    // region-and-flag words four at a time (s0 is a multiple
                    // of 4: 16-byte loads), then the accepted samples' valid
                    // counts -- two round trips; only the flag bits are kept
                    // past the scan (the scatter reads the word again)
                    const uint32_t lts = lt - n_old;
                    const uint32_t s0 = lts * kTileC + threadIdx.x * kAppendPer;
                    const uint32_t ns = st.n_samples;
                    static_assert(kAppendPer % 4 == 0 && kAppendPer <= 32, "16-byte loads of four words, one flag bit per sample");
                    static_assert(kTileC * kRepeatSparse < 65536, "a tile's repeat count fits the scan's low 16 bits");
                    uint32_t rf[kAppendPer];
#pragma unroll
                    for(int g = 0; g < kAppendPer; g += 4)
                        {
                            const uint32_t sb = s0 + g;
                            if(sb + 3 < ns)
                                {
                                    const uint4 v = *(const uint4*)(p.ur1f + sb);
                                    rf[g] = v.x, rf[g + 1] = v.y, rf[g + 2] = v.z, rf[g + 3] = v.w;
                                }
                            else
                                {
#pragma unroll
                                    for(int j = 0; j < 4; ++j) rf[g + j] = sb + j < ns ? p.ur1f[sb + j] : 0u;
                                }
                        }
                    uint32_t acc_bits = 0, sparse_bits = 0, ca = 0, cw = 0;
#pragma unroll
                    for(int j = 0; j < kAppendPer; ++j)
                        if(rf[j] >> 31)
                            {
                                const bool sparse = p.valid[rf[j] & 0x7FFFFFFFu] < kSparseValidLimit;
                                acc_bits |= 1u << j;
                                sparse_bits |= sparse ? 1u << j : 0u;
                                ++ca;
                                cw += sparse ? kRepeatSparse : kRepeatDense;
                            }
                    uint32_t agg;
                    const uint32_t excl = block_exclusive_scan<kAppendThreads>((ca << 16) | cw, scratch, &agg);
                    const uint32_t agg_a = agg >> 16, agg_w = agg & 0xffffu;
                    const unsigned long long val = ((unsigned long long)agg_a << 32) | agg_w;
                    publish_and_lookback(p.tiles_slot, lts, val, &s_prefix, &sched->error);
                    if(threadIdx.x == 0)
                        {
                            atomicAdd(&st.acc_total, agg_a);
                            atomicAdd(&st.w_total, agg_w);
                        }
                    __syncthreads();
                    const unsigned long long pre = s_prefix;
                    uint32_t ia = tree_size + (uint32_t)(pre >> 32) + (excl >> 16);
                    uint32_t iw = (uint32_t)(pre & 0xffffffffull) + (excl & 0xffffu);
                    const int D = (int)p.sample_dim;
                    for(uint32_t m = acc_bits; m; m &= m - 1u)
                        {
                            const int j = __ffs((int)m) - 1;
                            const uint32_t s = s0 + (uint32_t)j;
                            const uint32_t idx = ia++;
                            const uint32_t w = ((sparse_bits >> j) & 1u) ? kRepeatSparse : kRepeatDense;
                            if(!KGMT_BOUND(idx < p.capacity && s < p.capacity))
                                {
                                    iw += w;
                                    continue;
                                }
                            // everything the sample needs is loaded before its
                            // first store (one round trip, not one per field)
                            const int32_t par = __ldg(p.up + s), r1 = (int32_t)(__ldg(p.ur1f + s) & 0x7FFFFFFFu);
                            const float dist = append_row(p, p.us + (size_t)s * D, p.tree + (size_t)idx * D, D);
                            p.parent[idx] = par;
                            p.cost[idx] = dist;
                            p.node_r1[idx] = r1;
                            for(uint32_t r = 0; r < w; ++r, ++iw)
                                if(iw < p.capacity) p.rep_new[iw] = idx;
                            if(dist < p.goal_radius) atomicMin(&st.goal_cand, (int)idx);
                        }
                }
            // ---- tile done; the last tile of the query finalises it ----
            __syncthreads();
            if(threadIdx.x == 0)
                {
                    const uint32_t n_tiles = cbase.base[q + 1] - cbase.base[q];
                    const uint32_t done = atomic_add_release(&st.tiles_done, 1u);
                    // the block is free now: its next ticket, in flight with the count
                    next = gridDim.x + atomicAdd(&sched->ticket_c, 1u);
                    if(done == n_tiles - 1) s_fin = 1;
                }
            __syncthreads();
            if(s_fin)
                {
                    // every tile of this query is done: thread 0 finalises it
                    // and counts it finalised while the other threads clear
                    // its look-back words for the next iteration (nothing in
                    // this kernel reads them again, and the next append
                    // launch sees the stores: no fence on the path)
                    if(threadIdx.x == 0)
                        {
                            __threadfence();
                            st.f_accept = s_fa;
                            finalize_query(p, st, sched);
                            const uint32_t running = sched->running;
                            if(running == 1u)
                                {
                                    // the only running query: its finaliser is
                                    // the last, and no other block's results
                                    // are left to acquire (2: no block fence)
                                    __threadfence();
                                    s_glob = 2;
                                }
                            else if(atomic_add_release(&sched->finalized, 1u) == running - 1u) s_glob = 1;
                        }
                    const uint32_t n_tiles = cbase.base[q + 1] - cbase.base[q];
                    for(uint32_t i = threadIdx.x; i < n_old; i += kAppendThreads) p.tiles_old[i] = 0ull;
                    for(uint32_t i = threadIdx.x; i < n_tiles - n_old; i += kAppendThreads) p.tiles_slot[i] = 0ull;
                    __syncthreads();
                }
            if(s_glob)
                {
                    if(s_glob == 1) __threadfence();
                    compute_schedule<kAppendThreads, true>(P, S, sched, tile_a_base, tile_c_base, tile_c_old);
                }
            __syncthreads();
        }
}

// ---------------------------------------------------------------------------
// goal -> root path walk for finished queries (KGMT.cu:344-360)
// ---------------------------------------------------------------------------
// One warp a query: lane 0 follows the parents (a chain of dependent loads,
// ~0.4 us a node, and the only serial part), then all lanes copy the rows
// together.  What the host reads goes straight to its pinned memory: the
// states, the error bits and, packed one path behind the other, the rows of
// every path found by this launch (paths longer than kPathChunk rows, or past
// the buffer, stay on the device only).  A thread that walked and copied node
// by node took ~1 us a node (22 us for 22 nodes; now 9).
constexpr uint32_t kPathChunk = 128;  // nodes walked before their rows are copied
constexpr int kPathWarps = 4;         // queries per block

__global__ void __launch_bounds__(32 * kPathWarps) k_paths(const QueryParams* __restrict__ P, QueryState* S, uint32_t n, Sched* sched,
                                                           const HostSink sink)
{
    __shared__ int32_t s_node[kPathWarps][kPathChunk];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, q = blockIdx.x * kPathWarps + warp;
    if(blockIdx.x == 0 && threadIdx.x == 0 && sink.error) *sink.error = sched->error;
    if(q >= n) return;
    QueryState& st = S[q];
    if(st.status == KGMT_QUERY_SUCCESS && st.path_len == 0)
        {
            const QueryParams& p = P[q];
            const uint32_t D = p.sample_dim, max_rows = p.max_iterations + 2;
            const float* tree = p.tree;
            const int32_t* parent = p.parent;
            const int32_t goal = st.goal_index;
            int32_t i = goal;
            uint32_t len = 0, at = kNoPath;
            while(i >= 0 && len < max_rows)
                {
                    uint32_t k = 0;
                    if(lane == 0)
                        for(; k < kPathChunk && i >= 0 && len + k < max_rows; ++k)
                            {
                                s_node[warp][k] = i;
                                i = __ldg(parent + i);
                            }
                    k = __shfl_sync(0xffffffffu, k, 0);
                    i = __shfl_sync(0xffffffffu, i, 0);
                    // the whole path is in hand: its place in the host buffer
                    const bool whole = len == 0 && (i < 0 || k >= max_rows);
                    if(whole && sink.paths)
                        {
                            if(lane == 0)
                                {
                                    at = atomicAdd(&sched->path_words, k * D);
                                    if(at > sink.path_words || k * D > sink.path_words - at) at = kNoPath;
                                }
                            at = __shfl_sync(0xffffffffu, at, 0);
                        }
                    float* dev = p.path + (size_t)len * D;
#pragma unroll 4
                    for(uint32_t e = lane; e < k * D; e += 32)
                        {
                            const float v = __ldg(tree + (size_t)s_node[warp][e / D] * D + e % D);
                            dev[e] = v;
                            if(at != kNoPath) sink.paths[at + e] = v;
                        }
                    len += k;
                    __syncwarp();
                }
            if(lane == 0)
                {
                    st.goal_cost = p.cost[goal];
                    st.path_at = at;
                    st.path_len = len;
                }
            __syncwarp();
        }
    if(sink.states)
        for(uint32_t j = lane; j < sizeof(QueryState) / 8; j += 32)
            ((unsigned long long*)(sink.states + q))[j] = ((const unsigned long long*)&st)[j];
}

// ---------------------------------------------------------------------------
// obstacles: [n][6] rows (min xyz, max xyz) -> [n][2] float4 in the arena
// ---------------------------------------------------------------------------
__global__ void k_stage_obstacles(const float* __restrict__ src, float4* dst, uint32_t n, int w)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    stage_box(src + (size_t)i * 2 * w, w, dst + 2 * i);
}

// ---------------------------------------------------------------------------
// function-level propagation with explicit uniforms: sample rows [n][D] and
// eight uniforms a sample in, end rows, verdicts and region ids out
// ---------------------------------------------------------------------------
// Each block stages the boxes, builds the culling grid over them in its own
// shared memory where that pays (no workspace, nothing shared between calls)
// and runs a contiguous share of the samples.  Four forms:
//   one sample a thread, blocks of 128 (four warps load the four schedulers of
//   an SM evenly), where a call's time is its slowest sample's: without the grid
//   (plain, and wide: more and leaner blocks), or with it (culled);
//   sorted, blocks of 256: each share is counting-sorted by step count, 1024
//   samples at a time, and the runs of 32 are taken longest first by whichever
//   warp is free, so a warp's lanes loop equally long.
// End rows leave through a per-warp stage, so that a warp's stores cover whole
// rows.  Bound by instruction issue (the model's step).  Against one kernel for
// all models that ran one unsorted sample a thread and tested every box at
// every step: 2^20 quadrotor samples in 200 boxes 352 us, 1631 before; 200,000
// Dubins samples in 50 boxes 26 us, 60 before; 1000 double-integrator samples
// in 5 boxes (latency) 4.1 us, 4.8 before.
constexpr uint32_t kSamplesChunk = 1024;  // samples sorted at a time
// dynamic shared memory of the largest call (boxes; the grid's starts and
// items); the static arrays stay below the 22 KB left of an SM's 227
constexpr size_t kSamplesSmemMax = 205 * 1024;
// grid entries a block holds (scenes with more test every box): 8 a box, which
// boxes of the workloads' sizes stay below, within the shared memory there is
static uint32_t samples_items(uint32_t n_obs)
{
    const size_t room = (kSamplesSmemMax - (size_t)n_obs * 32 - kGridBuildBytes) / 2;
    return (uint32_t)std::min<size_t>(std::max<size_t>(4096, (size_t)n_obs * 8), std::min<size_t>(room, kMaxGridItems));
}
static size_t samples_smem(uint32_t n_obs, uint32_t items) { return (size_t)n_obs * 32 + (items ? kGridBuildBytes + (size_t)items * 2 : 0); }
enum { kSamplesPlain, kSamplesWide, kSamplesCulled, kSamplesSorted };
constexpr int samples_threads(int form) { return form == kSamplesSorted ? 256 : 128; }
// Blocks per SM that the forms are compiled for.  Plain and culled: no spills
// before warps (1000 double-integrator samples in 5 boxes 4.1 us at 3 blocks, 4.4
// at 5).  Wide: a wave of 97,280 samples (77,000 double-integrator samples in 20
// boxes 9.5 us at 5 blocks, 10.5 in two waves of 3, 12.0 sorted, 9.7 by the one kernel
// for all; Dubins 14.9, 15.6, 17.6, 14.7).  The quadrotor has no wide form: sorted, it
// keeps its state in 128 registers (77,000 samples in 20 boxes 38 us, 42 at 5 blocks).
// The other models sorted trade a few spills for more warps (2^20 double-integrator
// samples in 20 boxes 66 us at 3 blocks, 76 at 2).
constexpr int samples_blocks(int model, int form)
{
    const bool quad = model == KGMT_MODEL_QUADROTOR;
    return form == kSamplesWide ? (quad ? 3 : 5) : form == kSamplesSorted && quad ? 2 : 3;
}

template <int MODEL, int FORM>
__global__ void __launch_bounds__(samples_threads(FORM), samples_blocks(MODEL, FORM))
  k_propagate_samples(const __grid_constant__ QueryParams p, const float* x0, const float* __restrict__ uni, const float* __restrict__ obs_rows,
                      uint32_t n_obs, uint32_t n, uint32_t share, uint32_t grid_items, float* x1, uint8_t* valid, int32_t* r1, int32_t* r2)
{
    constexpr int D = ModelDims<MODEL>::D, NC = ModelDims<MODEL>::NC;
    constexpr uint32_t NT = (uint32_t)samples_threads(FORM);
    constexpr bool SORTED = FORM == kSamplesSorted, GRID = FORM == kSamplesCulled || SORTED;
    // one run a warp: its rows are on their way while the boxes are staged (not
    // in the wide form, for the registers)
    constexpr bool AHEAD = FORM == kSamplesPlain || FORM == kSamplesCulled;
    extern __shared__ float4 s_dyn[];
    float4* s_obs = s_dyn;
    char* s_grid = (char*)(s_dyn + 2 * (size_t)n_obs);
    uint16_t* s_items = (uint16_t*)(s_grid + kGridBuildBytes);
    __shared__ float s_stage[NT * D];
    __shared__ uint32_t s_scan[34];
    __shared__ uint32_t s_hist[kSortBins];
    __shared__ uint16_t s_perm[SORTED ? kSamplesChunk : 1];
    __shared__ uint32_t s_next;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b0 = min(n, blockIdx.x * share), b1 = min(n, b0 + share);
    float a[D], u[8];
    auto load = [&](uint32_t s) {
#pragma unroll
        for(int j = 0; j < D; ++j) a[j] = x0[(size_t)s * D + j];
#pragma unroll
        for(int j = 0; j < NC + 1; ++j) u[j] = uni[(size_t)s * 8 + j];
    };
    if(AHEAD && b0 + threadIdx.x < b1) load(b0 + threadIdx.x);
    const int w = MODEL == KGMT_MODEL_UNICYCLE ? 2 : 3;
    for(uint32_t i = threadIdx.x; i < n_obs; i += NT) stage_box(obs_rows + (size_t)i * 2 * w, w, s_obs + 2 * i);
    __syncthreads();
    std::conditional_t<GRID, BlockGrid, NoGrid> grid;
    if constexpr(GRID)
        {
            uint32_t total;
            grid = BlockGrid{grid_items ? build_grid<false>(p, s_obs, n_obs, grid_items, s_grid, s_scan, s_items, &total) : nullptr, s_items};
        }
    const unsigned full = 0xffffffffu;
    float* stage = s_stage + warp * 32 * D;
    for(uint32_t c0 = b0; c0 < b1; c0 += kSamplesChunk)
        {
            const uint32_t cn = min(kSamplesChunk, b1 - c0);
            const uint32_t n_runs = (cn + 31u) / 32u;
            if(SORTED)
                {
                    constexpr int PER = (int)kSamplesChunk / NT;
                    uint32_t key[PER], rank[PER];
                    if(threadIdx.x < kSortBins) s_hist[threadIdx.x] = 0;
                    if(threadIdx.x == 0) s_next = 0;
                    __syncthreads();
#pragma unroll
                    for(int h = 0; h < PER; ++h)
                        {
                            const uint32_t i = (uint32_t)h * NT + threadIdx.x;
                            key[h] = kSortBins - 1;
                            if(i < cn)
                                {
                                    const int k = draw_steps(p, uni[(size_t)(c0 + i) * 8 + NC]);
                                    key[h] = k < kSortBins - 1 ? (k > 0 ? (uint32_t)k : 0u) : kSortBins - 2;
                                    rank[h] = atomicAdd(&s_hist[key[h]], 1u);
                                }
                        }
                    __syncthreads();
                    if(threadIdx.x < 32)
                        {
                            const uint32_t v = s_hist[threadIdx.x];
                            uint32_t x = v;
#pragma unroll
                            for(int o = 1; o < 32; o <<= 1)
                                {
                                    const uint32_t y = __shfl_up_sync(full, x, o);
                                    if(lane >= (uint32_t)o) x += y;
                                }
                            s_hist[threadIdx.x] = x - v;
                        }
                    __syncthreads();
#pragma unroll
                    for(int h = 0; h < PER; ++h)
                        {
                            const uint32_t i = (uint32_t)h * NT + threadIdx.x;
                            if(i < cn) s_perm[s_hist[key[h]] + rank[h]] = (uint16_t)i;
                        }
                    __syncthreads();
                }
            for(uint32_t run = warp;;)
                {
                    if(SORTED)
                        {
                            if(lane == 0) run = atomicAdd(&s_next, 1u);
                            run = __shfl_sync(full, run, 0);
                        }
                    if(run >= n_runs) break;
                    // longest runs first
                    const uint32_t slot = (SORTED ? n_runs - 1u - run : run) * 32u + lane;
                    const bool live = slot < cn;
                    const uint32_t s = c0 + (live ? (SORTED ? (uint32_t)s_perm[slot] : slot) : 0u);
                    if(live)
                        {
                            float b[D];
                            if(!AHEAD) load(s);
                            PropCount cnt;
                            const bool ok = propagate_model<MODEL>(p, grid, a, u, s_obs, n_obs, b, cnt);
                            valid[s] = ok ? 1 : 0;
                            const CellIds c = cell_ids(p, b);
                            if(r1) r1[s] = c.r1;
                            if(r2) r2[s] = c.r2;
#pragma unroll
                            for(int j = 0; j < D; ++j) stage[lane * D + j] = b[j];
                        }
                    __syncwarp();
                    const uint32_t rows = min(32u, cn - (slot - lane));
                    // element e of the stage is column e % D of row e / D
#pragma unroll
                    for(uint32_t i = 0; i < (uint32_t)D; ++i)
                        {
                            const uint32_t e = i * 32u + lane, row = e / D;
                            const uint32_t rs = __shfl_sync(full, s, row & 31u);
                            if(row < rows) x1[(size_t)rs * D + (e - row * D)] = stage[e];
                        }
                    __syncwarp();
                    if(!SORTED) break;  // one run a warp
                }
            __syncthreads();
        }
}

// ---------------------------------------------------------------------------
// host-side launch wrappers
// ---------------------------------------------------------------------------
// launch as a programmatic dependent of the kernel before it in the stream
// (the kernel body waits for that one with pdl_wait)
static cudaLaunchConfig_t dependent_config(int grid, int block, size_t smem, cudaStream_t s, cudaLaunchAttribute* attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3((unsigned)block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <int NT, int MODELS>
static cudaError_t launch_propagate_t(const LaunchArgs& a, int grid, uint32_t boxes, cudaStream_t s)
{
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = dependent_config(grid, NT, prop_smem_bytes(boxes), s, attr);
    return cudaLaunchKernelEx(&cfg, k_propagate<NT, MODELS>, a.params, a.states, a.sched, (const uint32_t*)a.tile_a_base, boxes);
}

template <int NT>
static cudaError_t launch_propagate_m(const LaunchArgs& a, int models, int grid, uint32_t boxes, cudaStream_t s)
{
    switch(models)
        {
            case kBitDI: return launch_propagate_t<NT, kBitDI>(a, grid, boxes, s);
            case kBitQuad: return launch_propagate_t<NT, kBitQuad>(a, grid, boxes, s);
            case kBitDubins: return launch_propagate_t<NT, kBitDubins>(a, grid, boxes, s);
            case kBitUnicycle: return launch_propagate_t<NT, kBitUnicycle>(a, grid, boxes, s);
            default: return launch_propagate_t<NT, kAllModels>(a, grid, boxes, s);
        }
}

cudaError_t launch_propagate(const LaunchArgs& a, int block, int models, int grid, uint32_t smem_boxes, cudaStream_t s)
{
    const uint32_t boxes = smem_boxes < kSmemBoxesMin ? kSmemBoxesMin : smem_boxes > (uint32_t)kSmemObstacles ? (uint32_t)kSmemObstacles : smem_boxes;
    switch(block)
        {
            case 128: return launch_propagate_m<128>(a, models, grid, boxes, s);
            case 512: return launch_propagate_m<512>(a, models, grid, boxes, s);
            default: return launch_propagate_m<256>(a, models, grid, boxes, s);
        }
}

// blocks of one variant per SM; also lets the variant take its dynamic
// shared memory on top of more than 48 KB in total (the launch wrappers run
// after this has been called for the variant)
template <int NT, int MODELS>
static int occupancy_t(uint32_t boxes)
{
    int n = 0;
    const size_t smem = prop_smem_bytes(boxes);
    if(cudaFuncSetAttribute(k_propagate<NT, MODELS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prop_smem_bytes(kSmemObstacles)) != cudaSuccess)
        {
            cudaGetLastError();
            return 0;
        }
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_propagate<NT, MODELS>, NT, smem);
    return n;
}

template <int NT>
static int occupancy_m(int models, uint32_t boxes)
{
    switch(models)
        {
            case kBitDI: return occupancy_t<NT, kBitDI>(boxes);
            case kBitQuad: return occupancy_t<NT, kBitQuad>(boxes);
            case kBitDubins: return occupancy_t<NT, kBitDubins>(boxes);
            case kBitUnicycle: return occupancy_t<NT, kBitUnicycle>(boxes);
            default: return occupancy_t<NT, kAllModels>(boxes);
        }
}

int propagate_blocks_per_sm(int block, int models, uint32_t boxes)
{
    int n = 0;
    switch(block)
        {
            case 128: n = occupancy_m<128>(models, boxes); break;
            case 512: n = occupancy_m<512>(models, boxes); break;
            default: n = occupancy_m<256>(models, boxes); break;
        }
    return n > 0 ? n : 1;
}

int append_blocks_per_sm()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_append, kAppendThreads, 0);
    return n > 0 ? n : 1;
}

cudaError_t launch_append(const LaunchArgs& a, int grid, cudaStream_t s)
{
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = dependent_config(grid, kAppendThreads, 0, s, attr);
    return cudaLaunchKernelEx(&cfg, k_append, a.params, a.states, a.sched, a.tile_a_base, a.tile_c_base, a.tile_c_old);
}

cudaError_t launch_score(const LaunchArgs& a, int sms, bool large, cudaStream_t s)
{
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg;
    if(large)
        {
            cfg = dependent_config(sms * kScoreBlocksPerSm, kScoreThreads, 0, s, attr);
            const cudaError_t e = cudaLaunchKernelEx(&cfg, k_score, a.params, (const QueryState*)a.states, (const Sched*)a.sched);
            if(e != cudaSuccess) return e;
        }
    cfg = dependent_config(sms * kSumBlocksPerSm, kSumThreads, 0, s, attr);
    return cudaLaunchKernelEx(&cfg, k_score_sum, a.params, a.states, (const Sched*)a.sched);
}

cudaError_t launch_admit(const LaunchArgs& a, uint32_t first, uint32_t count, cudaStream_t s, const uint32_t* slots)
{
    if(count == 0) return cudaSuccess;
    k_admit<<<count, 256, 0, s>>>(a.params, a.states, first, count, slots);
    cudaError_t e = cudaGetLastError();
    if(e != cudaSuccess) return e;
    k_build_grid<<<count, 256, 0, s>>>(a.params, first, count, slots);
    return cudaGetLastError();
}

cudaError_t launch_schedule(const LaunchArgs& a, cudaStream_t s)
{
    k_schedule<<<1, kAppendThreads, 0, s>>>(a.params, a.states, a.sched, a.tile_a_base, a.tile_c_base, a.tile_c_old);
    return cudaGetLastError();
}

cudaError_t launch_paths(const LaunchArgs& a, uint32_t n, const HostSink& sink, cudaStream_t s)
{
    if(n == 0) return cudaSuccess;
    k_paths<<<(n + kPathWarps - 1) / kPathWarps, 32 * kPathWarps, 0, s>>>(a.params, a.states, n, a.sched, sink);
    return cudaGetLastError();
}

cudaError_t launch_begin(const LaunchArgs& a, const QueryParams& p, cudaStream_t s)
{
    // four table entries a thread, up to four blocks' worth of threads per SM
    const uint32_t items = p.regions > p.tiles_per_chain ? p.regions : p.tiles_per_chain;
    const uint32_t clear = std::min<uint32_t>((items + 1023u) / 1024u, 608u);
    k_begin<<<1 + clear, 256, 0, s>>>(p, a);
    return cudaGetLastError();
}

cudaError_t launch_stage_obstacles(const float* src, float4* dst, uint32_t n, int ws_dims, cudaStream_t s)
{
    if(n == 0) return cudaSuccess;
    k_stage_obstacles<<<(n + 255) / 256, 256, 0, s>>>(src, dst, n, ws_dims == 2 ? 2 : 3);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// persistent tail launch
// ---------------------------------------------------------------------------
size_t tail_scratch_bytes() { return sizeof(TailScratch); }

template <int MODELS>
static int tail_occupancy_t()
{
    int n = 0;
    const size_t smem = tail_smem_bytes(kSmemObstacles, tail_row_dim<MODELS>());
    if(cudaFuncSetAttribute(k_tail<MODELS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        {
            cudaGetLastError();
            return 0;
        }
    if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_tail<MODELS>, kTailThreads, smem) != cudaSuccess)
        {
            cudaGetLastError();
            return 0;
        }
    return n;
}

int tail_blocks_per_sm(int models)
{
    switch(models)
        {
            case kBitDI: return tail_occupancy_t<kBitDI>();
            case kBitQuad: return tail_occupancy_t<kBitQuad>();
            case kBitDubins: return tail_occupancy_t<kBitDubins>();
            case kBitUnicycle: return tail_occupancy_t<kBitUnicycle>();
            default: return tail_occupancy_t<kAllModels>();
        }
}

template <int MODELS>
static cudaError_t launch_tail_t(const LaunchArgs& a, TailScratch* ts, int grid, uint32_t boxes, uint32_t max_samples, unsigned long long tag0,
                                 uint32_t limit, uint32_t* host_words, cudaStream_t s)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3((unsigned)kTailThreads, 1, 1);
    cfg.dynamicSmemBytes = tail_smem_bytes(boxes, tail_row_dim<MODELS>());
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_tail<MODELS>, a.params, a.states, a.sched, ts, a.tile_a_base, a.tile_c_base, a.tile_c_old, boxes,
                              max_samples, tag0, limit, host_words);
}

cudaError_t launch_tail(const LaunchArgs& a, TailScratch* ts, int models, int grid, uint32_t smem_boxes, uint32_t max_samples, unsigned long long tag0,
                        uint32_t limit, uint32_t* host_words, cudaStream_t s)
{
    if(grid < 2 * kTailQueries || grid > kTailMaxBlocks) return cudaErrorInvalidValue;
    const uint32_t boxes = smem_boxes < kSmemBoxesMin ? kSmemBoxesMin : smem_boxes > (uint32_t)kSmemObstacles ? (uint32_t)kSmemObstacles : smem_boxes;
    switch(models)
        {
            case kBitDI: return launch_tail_t<kBitDI>(a, ts, grid, boxes, max_samples, tag0, limit, host_words, s);
            case kBitQuad: return launch_tail_t<kBitQuad>(a, ts, grid, boxes, max_samples, tag0, limit, host_words, s);
            case kBitDubins: return launch_tail_t<kBitDubins>(a, ts, grid, boxes, max_samples, tag0, limit, host_words, s);
            case kBitUnicycle: return launch_tail_t<kBitUnicycle>(a, ts, grid, boxes, max_samples, tag0, limit, host_words, s);
            default: return launch_tail_t<kAllModels>(a, ts, grid, boxes, max_samples, tag0, limit, host_words, s);
        }
}

template <int MODEL, int FORM>
static cudaError_t launch_samples_t(const QueryParams& p, const float* x0, const float* u, const float* obs, uint32_t n_obs, uint32_t n,
                                    uint32_t share, uint32_t items, float* x1, uint8_t* valid, int32_t* r1, int32_t* r2, cudaStream_t s)
{
    const size_t smem = samples_smem(n_obs, items);
    if(smem > 26 * 1024)
        {
            // more than 48 KB with the static arrays (always the same limit,
            // so that calls from several threads agree)
            const cudaError_t e = cudaFuncSetAttribute(k_propagate_samples<MODEL, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)kSamplesSmemMax);
            if(e != cudaSuccess) return e;
        }
    k_propagate_samples<MODEL, FORM><<<(n + share - 1) / share, samples_threads(FORM), smem, s>>>(p, x0, u, obs, n_obs, n, share, items, x1,
                                                                                                 valid, r1, r2);
    return cudaGetLastError();
}

// SMs of the current device, asked for once per device (a property that does
// not change; two threads asking at once store the same number)
static cudaError_t current_sms(int* sms)
{
    static std::atomic<int> known[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if(e != cudaSuccess) return e;
    const bool kept = dev >= 0 && dev < 64;
    if(kept && (*sms = known[dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
    e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
    if(e == cudaSuccess && kept) known[dev].store(*sms, std::memory_order_relaxed);
    return e;
}

// Whether the blocks build the grid: when the box tests it saves take longer than
// it does.  A test takes about 18 cycles (15 in the plane), the cell walk as much as
// 8 tests, and the build 10,500 cycles and 30 a box.  The time is that of the longest
// run: a few samples are not likely to draw the most steps or to last (n / (n + 8) of
// the way there), and with more than one warp a scheduler each adds 0.7 of its own.  A scene with more
// boxes than the grid has room for entries has none.  Without / with the grid: 1000
// Dubins samples in 40 boxes 8.9 / 12.2 us, 640 boxes 81 / 31; 58,000 in 20 boxes 11.7
// / 15.3, 40 boxes 16.9 / 16.4; 20,000 quadrotor samples in 20 boxes 24.8 / 27.9, 40
// boxes 29.6 / 28.3; one sample of the double integrator in 500 boxes, which it meets
// in its first step, 13 / 24.
static bool samples_culled(const QueryParams& p, uint32_t n_obs, uint32_t n, int sms)
{
    if(n_obs <= 8u || samples_items(n_obs) < n_obs) return false;
    const double warps = std::max(1.0, n / (128.0 * sms)), steps = p.min_steps + (p.max_steps - p.min_steps) * (n / (n + 8.0));
    return (1.0 + 0.7 * (warps - 1.0)) * steps * (p.planar ? 15.0 : 18.0) * (n_obs - 8.0) > 10500.0 + 30.0 * n_obs;
}

template <int MODEL>
static cudaError_t launch_samples_m(const QueryParams& p, const float* x0, const float* u, const float* obs, uint32_t n_obs, uint32_t n, float* x1,
                                    uint8_t* valid, int32_t* r1, int32_t* r2, cudaStream_t s)
{
    int sms = 0;
    const cudaError_t e = current_sms(&sms);
    if(e != cudaSuccess) return e;
    const uint32_t items = samples_culled(p, n_obs, n, sms) ? samples_items(n_obs) : 0u;
    const size_t smem = samples_smem(n_obs, items);
    // blocks that are resident together
    auto resident = [&](int form) {
        const size_t each = smem + (size_t)samples_threads(form) * ModelDims<MODEL>::D * 4 + 4096;  // the stage, the small arrays
        const size_t fit = std::max<size_t>(1, 227 * 1024 / each);
        return (uint32_t)sms * (uint32_t)std::min<size_t>((size_t)samples_blocks(MODEL, form), fit);
    };
    // one sample a thread while the resident blocks have a thread for each, else
    // sorted shares (200,000 quadrotor samples in 50 boxes: 73 us sorted, 148 not)
    constexpr uint32_t nt = (uint32_t)samples_threads(kSamplesPlain);
    if(items)
        {
            if(n <= resident(kSamplesCulled) * nt)
                return launch_samples_t<MODEL, kSamplesCulled>(p, x0, u, obs, n_obs, n, nt, items, x1, valid, r1, r2, s);
        }
    else if(n <= resident(kSamplesPlain) * nt)
        return launch_samples_t<MODEL, kSamplesPlain>(p, x0, u, obs, n_obs, n, nt, 0u, x1, valid, r1, r2, s);
    else if constexpr(MODEL != KGMT_MODEL_QUADROTOR)
        {
            if(n <= resident(kSamplesWide) * nt)
                return launch_samples_t<MODEL, kSamplesWide>(p, x0, u, obs, n_obs, n, nt, 0u, x1, valid, r1, r2, s);
        }
    const uint32_t blocks = resident(kSamplesSorted);
    const uint32_t share = ((n + blocks - 1) / blocks + 31u) & ~31u;
    return launch_samples_t<MODEL, kSamplesSorted>(p, x0, u, obs, n_obs, n, share, items, x1, valid, r1, r2, s);
}

cudaError_t launch_propagate_samples(const QueryParams& p, const float* x0, const float* u, const float* obs, uint32_t n_obs, uint32_t n,
                                     float* x1, uint8_t* valid, int32_t* r1, int32_t* r2, cudaStream_t s)
{
    if(n == 0) return cudaSuccess;
    switch(p.model)
        {
            case KGMT_MODEL_QUADROTOR: return launch_samples_m<KGMT_MODEL_QUADROTOR>(p, x0, u, obs, n_obs, n, x1, valid, r1, r2, s);
            case KGMT_MODEL_DUBINS_AIRPLANE: return launch_samples_m<KGMT_MODEL_DUBINS_AIRPLANE>(p, x0, u, obs, n_obs, n, x1, valid, r1, r2, s);
            case KGMT_MODEL_UNICYCLE: return launch_samples_m<KGMT_MODEL_UNICYCLE>(p, x0, u, obs, n_obs, n, x1, valid, r1, r2, s);
            default: return launch_samples_m<KGMT_MODEL_DOUBLE_INTEGRATOR>(p, x0, u, obs, n_obs, n, x1, valid, r1, r2, s);
        }
}

}  // namespace kgmt
