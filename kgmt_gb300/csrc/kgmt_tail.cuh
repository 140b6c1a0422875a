// kgmt_tail.cuh -- whole planning iterations in one persistent launch for
// batches with few running queries and single plans.
//
// While at most kTailQueries queries run and an iteration is a few samples a
// resident thread, the time of the chain of launches is latency: launches, the
// schedule round trip, the look-back hand-overs of the ordered append.  k_tail
// runs those iterations back to back inside one cooperative launch of one block
// per SM.  Each iteration the running queries split the blocks twice, in
// proportion to their samples and to their old nodes, so a block has the
// samples of one query (its boxes stay staged while it keeps that query) and
// the old nodes of one:
//
//   propagate   the block's samples, one a thread, with the per-sample code of
//               k_propagate; accepted end rows stay in shared memory; the old
//               nodes' regions and draws are fetched ahead
//                                     -- meet: accepted samples of each block --
//   scores      one block a query (Graph.cu:207-358); the other blocks append
//               their accepted rows meanwhile (KGMT.cu:317-362): tree index =
//               the accepted samples of the blocks before + the rank inside
//   re-activate once the query's scores are flagged ready (no meeting point):
//               draws against the scores (KGMT.cu:364-377), counted
//                            -- meet: re-activated nodes and repeats of each --
//   frontier    both lists of the next frontier, in index order
//                                      -- meet: smallest goal index of each --
//   finalise    every block, every query, from the same payloads; block 0 writes
//               the state back.
//
// A meeting point is an exchange: each block writes one word -- the iteration's
// tag and a payload -- and reads every block's, so the counts that the prefix
// sums need arrive with the barrier itself.  The words need no reset: the host
// numbers the launches, and a tag is the launch's number and the iteration, 64 bits
// that no engine uses twice.  The mailboxes have room for 28 of them, which come
// round after 2048 launches; they may, because every iteration rewrites every
// mailbox, so what a launch finds there is of the launch before it.  The score
// flags are rewritten only by launches with as many queries, and hold whole tags.  Every wait is bounded (kErrBarrierTimeout, reported
// as KGMT_ERR_TIMEOUT: a launch that gives up leaves the iteration half done, and
// nothing may go on from its state).  The launch stops before an iteration that is too large
// and leaves the state exactly as the chain of launches expects it (it recomputes
// the schedule), so the host can go on with that chain.
//
// Bound by latency: the slowest sample's steps, then about ten dependent L2
// round trips (three meetings, the scores, the gathers) and, the code being
// straight-line and long, instruction fetches: loops are kept rolled and helpers
// out of line.  Measured an iteration (double integrator, 20,000-node trees):
// one query 16.5 us (17.4 with four grid-wide barriers and rows through global
// memory), 16 queries 22.6 (38 in the chain of launches, which took over above
// four).
#pragma once
#include <climits>
#include <cstdint>

#include "kgmt_iter.cuh"

namespace kgmt {

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// All blocks of the cooperative launch meet here, each with a payload (thread 0's
// value counts); pay[] (shared memory) gets every block's, and what a block wrote
// before the call is visible to every block after it.  Thread 0 publishes the
// block's writes and its word (one fence), adds the block's arrival and waits for
// all of them (an acquiring read, so every thread's after the barrier); then
// every thread reads one block's word.  The arrivals only
// grow: a launch starts from what the last one left.  The words are kept twice,
// used by turns: a block that is through may leave its word for the next meeting
// while a slower one still reads this meeting's (after the goal meeting nothing
// else holds it back), but it cannot get to the one after, which has this
// meeting's words, before every block has arrived at the next and so has read
// them.  False when the wait gave up, after limit x units polls.
struct Meeting {
    uint32_t target;  // arrivals that complete the last meeting
    uint32_t row;     // words of the next one
};

__device__ __noinline__ bool meet(TailScratch* ts, Meeting& m, uint32_t payload, unsigned long long* pay, uint32_t limit, uint32_t units,
                                  uint32_t* error)
{
    __shared__ int s_ok;
    __syncthreads();
    m.target += gridDim.x;
    uint32_t* word = ts->word[m.row];
    m.row ^= 1u;
    if(threadIdx.x == 0)
        {
            *(volatile uint32_t*)&word[blockIdx.x] = payload;
            __threadfence();
            atomicAdd(&ts->arrivals, 1u);
            int ok = 1;
            uint32_t spins = 0;
            while((int32_t)(ld_acquire_u32(&ts->arrivals) - m.target) < 0)
                {
                    if(++spins > limit)
                        {
                            spins = 0;
                            if(--units == 0u)
                                {
                                    atomicOr(error, kErrBarrierTimeout);
                                    ok = 0;
                                    break;
                                }
                        }
                    __nanosleep(32);
                }
            s_ok = ok;
        }
    __syncthreads();
    if(threadIdx.x < gridDim.x) pay[threadIdx.x] = ld_relaxed_u32(&word[threadIdx.x]);
    __syncthreads();
    return s_ok != 0;
}

// The blocks exchange payloads of kExchangeBits and nothing else: no fence, and no
// writes ordered by it.  Every block leaves a word with the meeting's tag in
// every block's own row of mailboxes and waits until its own row has it
// throughout: one store and one load on the path.  (All blocks polling one row of
// words took 5 us; a mailbox row is read by one block only.)
__device__ __noinline__ bool exchange(TailBox (*boxes)[kTailMaxBlocks], unsigned long long payload, unsigned long long tag, unsigned long long* pay,
                                      uint32_t limit, uint32_t* error)
{
    __shared__ int s_ok;
    __shared__ unsigned long long s_mine;
    const unsigned long long want = (tag << kExchangeBits) >> kExchangeBits;  // the tag's bits that fit beside the payload
    if(threadIdx.x == 0)
        {
            s_ok = 1;
            s_mine = (want << kExchangeBits) | payload;
        }
    __syncthreads();
    if(threadIdx.x < gridDim.x)
        {
            st_volatile_u64(&boxes[threadIdx.x][blockIdx.x], s_mine);
            const TailBox* from = &boxes[blockIdx.x][threadIdx.x];
            uint32_t spins = 0;
            unsigned long long w;
            while(((w = ld_relaxed_u64(from)) >> kExchangeBits) != want)
                if(++spins > limit)
                    {
                        atomicOr(error, kErrBarrierTimeout);
                        s_ok = 0;
                        break;
                    }
            pay[threadIdx.x] = w & ((1ull << kExchangeBits) - 1ull);
        }
    __syncthreads();
    return s_ok != 0;
}

// Exclusive prefix of one value a thread over the block, and the total; one
// barrier (each thread adds up the warps before its own).  scratch: 2 x 8 words,
// used in turn (`turn`: 0, 1, 0, ... between barriers).
__device__ __noinline__ uint32_t tail_scan(uint32_t v, uint32_t (*scratch)[kTailThreads / 32], uint32_t turn, uint32_t* total)
{
    constexpr int NW = kTailThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += y;
        }
    if(lane == 31) scratch[turn][warp] = x;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for(int w = 0; w < NW; ++w)
        {
            const uint32_t t = scratch[turn][w];
            before += w < warp ? t : 0u;
            sum += t;
        }
    *total = sum;
    return before + x - v;
}

// sums of the low `bits` and of the remaining bits of pay[lo .. hi); by a warp,
// every lane gets them
__device__ __forceinline__ uint2 range_sums(const unsigned long long* pay, uint32_t lo, uint32_t hi, int bits)
{
    uint32_t a = 0, b = 0;
#pragma unroll 1
    for(uint32_t j = lo + (threadIdx.x & 31u); j < hi; j += 32)
        {
            a += (uint32_t)pay[j] & ((1u << bits) - 1u);
            b += (uint32_t)(pay[j] >> bits);
        }
    return make_uint2(__reduce_add_sync(0xffffffffu, a), __reduce_add_sync(0xffffffffu, b));
}

// replicated per-query loop state (every block holds the same copy)
struct TailQuery {
    int slot;
    uint32_t status, itr, tree, n_react, w_new, spe, n_samples, drawn;
    uint32_t slices;  // of a large region table (0: scored by one block)
    uint32_t n_next;  // accepted samples of this iteration
    uint32_t units;   // of the wait for a sample
    float fa;
    // of the query's params
    uint32_t capacity, samples_per_node, max_iterations;
    float epsilon;
    uint64_t seed;
    const int32_t* node_r1;
    uint32_t* rep_old;
    ScoreParams sp;
    // this iteration's blocks: [sample0, sample0 + samples_nb) take its
    // samples, share_s each; [node0, node0 + nodes_nb) its old nodes
    uint32_t sample0, samples_nb, share_s, node0, nodes_nb, share_n;
};

// re-activation draw of old node i (KGMT.cu:371-373)
__device__ __forceinline__ float reactivation_draw(uint64_t seed, uint32_t i, uint32_t itr)
{
    return u01(philox4x32_10(i, itr, 1u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32)).x);
}

// exclusive prefix over the warp's lanes
__device__ __forceinline__ uint32_t warp_prefix(uint32_t v)
{
    uint32_t x = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if((threadIdx.x & 31u) >= (unsigned)o) x += y;
        }
    return x - v;
}

constexpr uint32_t kTailAhead = 8;      // old nodes a thread draws before the scores are known
constexpr uint32_t kTailBitWords = 16;  // words of re-activation bits a thread keeps between counting and scatter

// dynamic shared memory of a launch that stages `boxes` boxes and meets rows of
// at most `dim` floats
__host__ __device__ constexpr uint32_t tail_smem_bytes(uint32_t boxes, uint32_t dim)
{
    return staged_bytes(boxes) + kTailShare * dim * 4u + kTailBitWords * (uint32_t)kTailThreads * 4u;
}

template <int MODELS>
constexpr uint32_t tail_row_dim()
{
    return (MODELS & kBitQuad) ? 17u : (MODELS & (kBitDI | kBitDubins)) ? 10u : 7u;
}

// Re-activation bits of up to 16 old nodes from i (a multiple of 4: the tables
// start 256-byte aligned), below end: regions four at a time, then the draws,
// then the scores (acquired by the caller, so past L1 once and then from it).
__device__ __noinline__ uint32_t reactivated16(const TailQuery& Q, uint32_t i, uint32_t end)
{
    const int32_t* node_r1 = Q.node_r1;
    const float* score = Q.sp.score;
    const uint64_t seed = Q.seed;
    const uint32_t itr = Q.itr;
    const float fa = Q.fa;
    int32_t reg[16];
#pragma unroll
    for(int g = 0; g < 16; g += 4)
        {
            const uint32_t ib = i + g;
            if(ib + 3 < end)
                {
                    const int4 v = __ldcg((const int4*)(node_r1 + ib));
                    reg[g] = v.x, reg[g + 1] = v.y, reg[g + 2] = v.z, reg[g + 3] = v.w;
                }
            else
#pragma unroll
                for(int j = 0; j < 4; ++j) reg[g + j] = ib + j < end ? __ldcg(node_r1 + ib + j) : 0;
        }
    uint32_t bits = 0;
#pragma unroll
    for(int j = 0; j < 16; ++j)
        if(i + j < end && reactivation_draw(seed, i + j, itr) <= score[reg[j]] + fa) bits |= 1u << j;
    return bits;
}

// 32 of them
__device__ __forceinline__ uint32_t reactivated32(const TailQuery& Q, uint32_t i, uint32_t end)
{
    uint32_t m = 0;
#pragma unroll 1
    for(uint32_t h = 0; h < 32u && i + h < end; h += 16u) m |= reactivated16(Q, i + h, end) << h;
    return m;
}

template <int MODELS>
__global__ void __launch_bounds__(kTailThreads, 1) k_tail(const QueryParams* __restrict__ P, QueryState* S, Sched* sched, TailScratch* ts,
                                                         uint32_t* tile_a_base, uint32_t* tile_c_base, uint32_t* tile_c_old,
                                                         uint32_t smem_boxes, uint32_t max_samples, unsigned long long tag0, uint32_t limit,
                                                         uint32_t* host_words)
{
    constexpr int NT = kTailThreads;
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    extern __shared__ float4 s_dyn[];
    uint16_t* s_gstart = (uint16_t*)s_dyn;
    uint16_t* s_gitems = (uint16_t*)((char*)s_dyn + kSmemStartBytes);
    uint32_t* s_gmeta = (uint32_t*)((char*)s_dyn + kSmemStartBytes + kSmemGridItems * 2);
    float4* s_obs = (float4*)((char*)s_dyn + kSmemGridBytes);
    __shared__ uint32_t s_copy;
    __shared__ alignas(8) uint64_t mbar;
    __shared__ QueryParams s_p;
    __shared__ PropCtx s_c;
    __shared__ PropShared s_sh;
    __shared__ float s_lanes[kScoreLanes];
    __shared__ uint32_t s_scan[34];
    __shared__ uint32_t s_turn[2][NT / 32];
    __shared__ TailQuery tq[kTailQueries];
    __shared__ unsigned long long s_pay[kTailMaxBlocks];
    __shared__ uint32_t s_goal[kTailQueries], s_goal_min;
    __shared__ int s_score_q, s_qs, s_qn, s_nr, s_too_large, s_too_many;
    __shared__ uint32_t s_units;
    // the block's samples of this iteration: accepted end rows (dynamic, behind
    // the boxes), parents, and region words with the accept flag
    float* s_rows = (float*)((char*)s_dyn + staged_bytes(smem_boxes));
    uint32_t* s_bits = (uint32_t*)(s_rows + kTailShare * tail_row_dim<MODELS>());
    __shared__ int32_t s_par[kTailShare];
    __shared__ uint32_t s_word[kTailShare];
    const uint32_t G = gridDim.x, b = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;

    // ---- the running queries, in slot order (the same in every block) ----
    if(threadIdx.x == 0)
        {
            mbar_init(&mbar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    const uint32_t n_slots = __ldcg(&sched->n_slots);
    uint32_t count = 0;
    for(uint32_t base = 0; base < n_slots; base += NT)
        {
            const uint32_t i = base + threadIdx.x;
            const uint32_t run = (i < n_slots && __ldcg(&S[i].status) == KGMT_QUERY_RUNNING) ? 1u : 0u;
            uint32_t tot;
            const uint32_t pos = count + block_exclusive_scan<NT>(run, s_scan, &tot);
            if(run && pos < (uint32_t)kTailQueries) tq[pos].slot = (int)i;
            count += tot;
        }
    if(count == 0 || count > (uint32_t)kTailQueries)
        {
            // nothing for this launch: the chain's state is untouched
            if(b == 0 && threadIdx.x == 0)
                {
                    ts->iterations = 0;
                    ts->declined = count > 0 ? 1u : 0u;
                    if(host_words)
                        {
                            *(volatile uint32_t*)&host_words[0] = 0u;
                            *(volatile uint32_t*)&host_words[1] = count > 0 ? 1u : 0u;
                        }
                }
            return;
        }
    const int nq = (int)count;
    __syncthreads();
    if((int)threadIdx.x < nq)
        {
            TailQuery& Q = tq[threadIdx.x];
            const QueryState& st = S[Q.slot];
            Q.status = __ldcg(&st.status);
            Q.itr = __ldcg(&st.itr);
            Q.tree = __ldcg(&st.tree_size);
            Q.n_react = __ldcg(&st.n_react);
            Q.w_new = __ldcg(&st.w_new);
            Q.spe = __ldcg(&st.spe);
            Q.n_samples = __ldcg(&st.n_samples);
            Q.drawn = __ldcg(&st.samples_drawn);
            const QueryParams& gp = P[Q.slot];
            Q.capacity = gp.capacity, Q.samples_per_node = gp.samples_per_node, Q.max_iterations = gp.max_iterations;
            Q.epsilon = gp.epsilon, Q.seed = gp.seed;
            Q.node_r1 = gp.node_r1, Q.rep_old = gp.rep_old;
            Q.sp = score_params(gp);
            Q.units = wait_units(gp.max_steps, gp.n_obstacles);
            Q.slices = Q.sp.regions > kScoreSmall ? (Q.sp.regions + kTailSlice - 1) / kTailSlice : 0u;
        }
    __syncthreads();

    uint32_t iters = 0, declined = 0;
    unsigned long long tag = tag0;
    Meeting next{__ldcg(&ts->arrived), 0u};  // (arrived is rewritten by block 0 after every block's last meeting)
    int cur_slot = -1;
    uint32_t phase = 0;
    // thread 0: work of the current slot's samples, added to its state when the
    // block changes query or leaves
    unsigned long long run_steps = 0, run_tests = 0, run_samples = 0;
    auto flush = [&] {
        if(cur_slot < 0 || run_samples == 0) return;
        QueryState& st = S[cur_slot];
        atomicAdd(&st.steps, run_steps);
        atomicAdd(&st.tests, run_tests);
        const unsigned long long lookup = s_p.n_obstacles ? kOpsPerGridLookup : 0u;
        atomicAdd(&ts->fp32_ops, run_steps * (ops_per_step(s_p.model) + lookup) + run_tests * kOpsPerObstacleTest);
        atomicAdd(&ts->samples, run_samples);
        run_steps = run_tests = run_samples = 0;
    };
    for(;;)
        {
            // ---- the iteration's size and its division among the blocks, a
            // query a lane: warp 0 divides its samples, warp 1 its old nodes ----
            if(warp < 2)
                {
                    const unsigned full = 0xffffffffu;
                    const bool run = (int)lane < nq && tq[lane].status == KGMT_QUERY_RUNNING;
                    const unsigned running = __ballot_sync(full, run);
                    const uint32_t nr = (uint32_t)__popc(running);
                    const uint32_t n = !run ? 0u : warp == 0 ? tq[lane].n_samples : tq[lane].tree;
                    // at most 32 queries of at most 2^28 nodes: weights of 32
                    // nodes; samples past 2^24 are too many in any case
                    const uint32_t weight = warp == 0 ? min(n, 1u << 24) : (n + 31u) >> 5;
                    const uint32_t tot = __reduce_add_sync(full, weight);
                    uint32_t nb = n ? 1u : 0u;
                    if(nr == 1u) nb *= G;
                    else if(n) nb += (uint32_t)((float)(G - nr) * 0.99999f * ((float)weight * __frcp_rn((float)tot)));
                    // a share with share * nb >= n, whole warps or 16-byte words
                    uint32_t share = n ? (uint32_t)((float)n * 1.00001f * __frcp_rn((float)nb)) + 1u : 0u;
                    share = warp == 0 ? (share + 31u) & ~31u : (share + 3u) & ~3u;
                    const uint32_t first = warp_prefix(nb);
                    const unsigned at = __ballot_sync(full, b - first < nb);
                    const unsigned big = __ballot_sync(full, share > (warp == 0 ? kTailShare : kTailNodes));
                    // a block's samples take as many rounds of its threads
                    constexpr uint32_t kRounds = (kTailShare + NT - 1) / NT;
                    const uint32_t units = kRounds * min(__reduce_max_sync(full, run ? tq[lane].units : 1u), 0xFFFFFFFFu / kRounds);
                    const uint32_t order = (uint32_t)__popc(running & ((1u << lane) - 1u));
                    // a query's scores are finished by the order-th block from the end
                    const unsigned mine = __ballot_sync(full, run && order == G - 1u - b);
                    if(run)
                        {
                            TailQuery& Q = tq[lane];
                            if(warp == 0) Q.sample0 = first, Q.samples_nb = nb, Q.share_s = share;
                            else Q.node0 = first, Q.nodes_nb = nb, Q.share_n = share;
                        }
                    if(lane == 0)
                        {
                            const int here = at ? __ffs((int)at) - 1 : -1;
                            if(warp == 0)
                                {
                                    s_nr = (int)nr;
                                    s_too_large = tot > max_samples || big;
                                    s_qs = here;
                                    s_score_q = mine ? __ffs((int)mine) - 1 : -1;
                                    s_sh.acc = 0, s_sh.steps = 0, s_sh.tests = 0;
                                    s_goal_min = kNone;
                                    s_units = units;
                                }
                            else s_qn = here, s_too_many = big != 0u;
                        }
                    if(warp == 0) s_goal[lane] = kNone;
                }
            __syncthreads();
            if(s_nr == 0) break;
            if(s_too_large | s_too_many)
                {
                    declined = 1;
                    break;
                }
            tag += 1;
            const int qs = s_qs, qn = s_qn;

            // ---- the block's samples (KGMT.cu:218-299) ----
            uint32_t lo = 0, hi = 0;
            if(qs >= 0)
                {
                    const uint32_t ns = tq[qs].n_samples, share = tq[qs].share_s;
                    lo = min(ns, (b - tq[qs].sample0) * share), hi = min(ns, lo + share);
                }
            if(lo < hi)
                {
                    const int slot = tq[qs].slot;
                    bool wait_obs = false;
                    if(slot != cur_slot)
                        {
                            if(threadIdx.x == 0) flush();
                            __syncthreads();
                            const uint32_t* src = (const uint32_t*)&P[slot];
                            uint32_t* dst = (uint32_t*)&s_p;
                            for(int i = threadIdx.x; i < (int)(sizeof(QueryParams) / 4); i += NT) dst[i] = src[i];
                            if(threadIdx.x == 0)
                                {
                                    const QueryParams& gp = P[slot];
                                    const uint32_t n_obs = gp.n_obstacles;
                                    const bool obs_s = n_obs > 0 && n_obs <= smem_boxes;
                                    const bool grid = gp.grid_meta != nullptr;
                                    const uint32_t bytes = (obs_s ? n_obs * 32u : 0u) + (grid ? 16u + kSmemStartBytes + kSmemGridItems * 2 : 0u);
                                    s_copy = bytes;
                                    if(bytes)
                                        {
                                            fence_proxy_async_smem();
                                            mbar_expect_tx(&mbar, bytes);
                                            if(obs_s) bulk_copy_g2s(s_obs, gp.obstacles, n_obs * 32u, &mbar);
                                            if(grid)
                                                {
                                                    bulk_copy_g2s(s_gmeta, gp.grid_meta, 16u, &mbar);
                                                    bulk_copy_g2s(s_gstart, gp.grid_start, kSmemStartBytes, &mbar);
                                                    bulk_copy_g2s(s_gitems, gp.grid_items, kSmemGridItems * 2, &mbar);
                                                }
                                        }
                                }
                            cur_slot = slot;
                            __syncthreads();
                            wait_obs = s_copy != 0;
                        }
                    if(threadIdx.x == 0)
                        {
                            s_c.itr = tq[qs].itr;
                            s_c.spe = tq[qs].spe;
                            s_c.n_react = tq[qs].n_react;
                            s_c.n_samples = tq[qs].n_samples;
                        }
                    __syncthreads();
                    const size_t D = s_p.sample_dim;
                    for(uint32_t r0 = lo; r0 < hi; r0 += NT)
                        propagate_range<NT, MODELS>(s_p, s_c, r0, min((uint32_t)NT, hi - r0), smem_boxes, &s_sh, s_obs, s_gstart, s_gitems, s_gmeta,
                                                    s_rows + (r0 - lo) * D, s_par + (r0 - lo), s_word + (r0 - lo), [&] {
                                                        // the staged boxes: waited for once, before their first use
                                                        if(!wait_obs) return;
                                                        wait_obs = false;
                                                        uint32_t spins = 0;
                                                        while(!mbar_try_wait(&mbar, phase))
                                                            if(++spins > kSpinLimit)
                                                                {
                                                                    if(threadIdx.x == 0) atomicOr(&sched->error, kErrCopyTimeout);
                                                                    break;
                                                                }
                                                        phase ^= 1u;
                                                    });
                }
            // old nodes of the block: a thread has n1 - n0 consecutive ones, the
            // last thread the first (the first warps have the samples); a few a
            // thread are drawn, and their regions fetched, while slower warps
            // and blocks still propagate
            uint32_t n0 = 0, n1 = 0;
            if(qn >= 0)
                {
                    const TailQuery& Q = tq[qn];
                    const uint32_t c0 = min(Q.tree, (b - Q.node0) * Q.share_n), c1 = min(Q.tree, c0 + Q.share_n);
                    uint32_t k = (Q.share_n + NT - 1) / NT;
                    if(k > kTailAhead) k = (k + 3u) & ~3u;  // 16-byte loads
                    n0 = min(c1, c0 + (NT - 1u - threadIdx.x) * k), n1 = min(c1, n0 + k);
                    if(k <= kTailAhead)
                        // (two words a node of the thread's own in shared memory: a
                        // rolled loop, for the instruction cache's sake)
#pragma unroll 1
                        for(uint32_t j = 0; n0 + j < n1; ++j)
                            {
                                s_bits[2 * j * NT + threadIdx.x] = (uint32_t)__ldcg(Q.node_r1 + n0 + j);
                                s_bits[(2 * j + 1) * NT + threadIdx.x] = __float_as_uint(reactivation_draw(Q.seed, n0 + j, Q.itr));
                            }
                }
            __syncthreads();
            const uint32_t acc_block = s_sh.acc;
            if(threadIdx.x == 0 && lo < hi) run_steps += s_sh.steps, run_tests += s_sh.tests, run_samples += hi - lo;
            if(!meet(ts, next, acc_block, s_pay, limit, s_units, &sched->error)) return;

            // ---- region scores, first of all: every re-activation waits for them ----
            uint32_t large = 0;
            for(int q = 0; q < nq; ++q)
                if(tq[q].status == KGMT_QUERY_RUNNING) large += tq[q].slices;
            const int score_q = s_score_q;
            if(score_q >= 0 && !tq[score_q].slices) update_scores<NT>(tq[score_q].sp, S[tq[score_q].slot], s_lanes);
            if(large)
                {
                    // slices of large tables go round the blocks; once all are
                    // scored, one block a query sums and normalises
                    uint32_t before = 0;
#pragma unroll 1
                    for(int q = 0; q < nq; ++q)
                        if(tq[q].status == KGMT_QUERY_RUNNING && tq[q].slices)
                            {
                                for(uint32_t j = (b + G - before % G) % G; j < tq[q].slices; j += G) score_slice<NT, kTailSlice>(tq[q].sp, j);
                                before += tq[q].slices;
                            }
                    if(!meet(ts, next, acc_block, s_pay, limit, 1u, &sched->error)) return;  // (the same payload: it is read below)
                    if(score_q >= 0 && tq[score_q].slices) score_finish<NT>(tq[score_q].sp, S[tq[score_q].slot], s_lanes);
                }
            if(score_q >= 0)
                {
                    __syncthreads();
                    if(threadIdx.x == 0)
                        {
                            __threadfence();
                            st_volatile_u64(&ts->scored[score_q], tag);
                        }
                }

            // ---- accepted samples: of each query (by the last warps: the first
            // ones have the rows), and before the block's own ----
#pragma unroll 1
            for(int q = NT / 32 - 1 - (int)warp; q < nq; q += NT / 32)
                {
                    TailQuery& Q = tq[q];
                    const uint32_t n = range_sums(s_pay, Q.sample0, Q.sample0 + Q.samples_nb, 31).x;
                    if(lane == 0 && Q.status == KGMT_QUERY_RUNNING)
                        {
                            Q.n_next = n;
                            Q.fa = f_accept_vals(Q.capacity, Q.epsilon, Q.tree, n, Q.itr);
                        }
                }
            const uint32_t acc_before = qs >= 0 ? range_sums(s_pay, tq[qs].sample0, b, 31).x : 0u;

            // ---- accepted rows appended in slot order (KGMT.cu:317-362); a
            // thread has `per` consecutive samples ----
            const uint32_t n_own = hi - lo, per = (n_own + NT - 1) / NT;
            const uint32_t i0 = min(n_own, threadIdx.x * per), i1 = min(n_own, i0 + per);
            constexpr uint32_t kPer = (kTailShare + NT - 1) / NT;
            uint32_t ca = 0, cw = 0, sparse_bits = 0;
            if(i0 < i1)
                {
                    uint32_t word[kPer];
                    int32_t valid[kPer];
#pragma unroll
                    for(uint32_t j = 0; j < kPer; ++j)
                        {
                            word[j] = i0 + j < i1 ? s_word[i0 + j] : 0u;
                            valid[j] = word[j] >> 31 ? __ldcg(s_p.valid + (word[j] & 0x7FFFFFFFu)) : 0;
                        }
#pragma unroll
                    for(uint32_t j = 0; j < kPer; ++j)
                        if(word[j] >> 31)
                            {
                                const bool sparse = valid[j] < kSparseValidLimit;
                                sparse_bits |= sparse ? 1u << j : 0u;
                                ca += 1u;
                                cw += sparse ? kRepeatSparse : kRepeatDense;
                            }
                }
            static_assert(kTailShare * kRepeatSparse < (1u << kRepeatBits) && kTailShare < (1u << 18), "a block's repeats and rows share one word");
            uint32_t own;
            const uint32_t ex = tail_scan((ca << kRepeatBits) | cw, s_turn, 0, &own);
            // the rows appended are the samples counted as accepted, from which every
            // block has its first row (the chain's finaliser compares them too)
            if(threadIdx.x == 0 && (own >> kRepeatBits) != acc_block) atomicOr(&sched->error, kErrAppendMismatch);
            const uint32_t first = qs >= 0 ? tq[qs].tree + acc_before + (ex >> kRepeatBits) : 0u;
            if(ca)
                {
                    [[maybe_unused]] const uint32_t cap = s_p.capacity;
                    const int D = (int)s_p.sample_dim;
                    uint32_t idx = first;
                    for(uint32_t i = i0; i < i1; ++i)
                        {
                            if(!(s_word[i] >> 31)) continue;
                            if(KGMT_BOUND(idx < cap))
                                {
                                    const float* row = s_rows + (size_t)i * D;
                                    float* dst = s_p.tree + (size_t)idx * D;
                                    for(int c = 0; c < D; ++c) dst[c] = row[c];
                                    const float dist = goal_distance(s_p, row);
                                    s_p.parent[idx] = s_par[i];
                                    s_p.cost[idx] = dist;
                                    s_p.node_r1[idx] = (int32_t)(s_word[i] & 0x7FFFFFFFu);
                                    if(dist < s_p.goal_radius) atomicMin(&s_goal_min, idx);
                                }
                            ++idx;
                        }
                }

            // ---- old nodes re-activated (KGMT.cu:364-377), counted; the bits
            // are kept for the scatter (a thread of more than 32 kTailBitWords
            // nodes draws again there) ----
            uint32_t obits = 0, n_old = 0;
            if(qn >= 0)
                {
                    if(threadIdx.x == 0)
                        {
                            uint32_t spins = 0;
                            while(ld_relaxed_u64(&ts->scored[qn]) != tag)
                                if(++spins > limit)
                                    {
                                        atomicOr(&sched->error, kErrBarrierTimeout);
                                        break;
                                    }
                            (void)ld_acquire_u64(&ts->scored[qn]);
                        }
                    __syncthreads();
                    const TailQuery& Q = tq[qn];
                    if(Q.share_n <= kTailAhead * NT)
                        {
                            const float* score = Q.sp.score;
                            const float fa = Q.fa;
#pragma unroll 2
                            for(uint32_t j = 0; n0 + j < n1; ++j)
                                if(__uint_as_float(s_bits[(2 * j + 1) * NT + threadIdx.x]) <= score[s_bits[2 * j * NT + threadIdx.x]] + fa)
                                    obits |= 1u << j;
                            n_old = (uint32_t)__popc(obits);
                        }
                    else
                        for(uint32_t w = 0, i = n0; i < n1; ++w, i += 32u)
                            {
                                const uint32_t m = reactivated32(Q, i, n1);
                                n_old += (uint32_t)__popc(m);
                                if(w < kTailBitWords) s_bits[w * NT + threadIdx.x] = m;
                            }
                }
            uint32_t old_block;
            // (the last thread has the first nodes)
            const uint32_t old_ex = [&] {
                const uint32_t before = tail_scan(n_old, s_turn, 1, &old_block);
                return old_block - before - n_old;
            }();
            static_assert(2 * kTailAhead <= kTailBitWords, "the nodes drawn ahead use the bits' memory");
            const uint32_t w_block = own & ((1u << kRepeatBits) - 1u);
            if(!exchange(ts->box, ((unsigned long long)old_block << kRepeatBits) | w_block, tag, s_pay, limit, &sched->error)) return;

            // ---- the next frontier's lists ----
            const uint32_t old_before = qn >= 0 ? range_sums(s_pay, tq[qn].node0, b, kRepeatBits).y : 0u;
            const uint32_t w_before = qs >= 0 ? range_sums(s_pay, tq[qs].sample0, b, kRepeatBits).x : 0u;
#pragma unroll 1
            for(int q = NT / 32 - 1 - (int)warp; q < nq; q += NT / 32)
                {
                    TailQuery& Q = tq[q];
                    const uint32_t n = range_sums(s_pay, Q.node0, Q.node0 + Q.nodes_nb, kRepeatBits).y;
                    const uint32_t w = range_sums(s_pay, Q.sample0, Q.sample0 + Q.samples_nb, kRepeatBits).x;
                    if(lane == 0 && Q.status == KGMT_QUERY_RUNNING) Q.n_react = n, Q.w_new = w;
                }
            if(n_old)
                {
                    const TailQuery& Q = tq[qn];
                    uint32_t pos = old_before + old_ex;
                    for(uint32_t w = 0, i = n0; i < n1; ++w, i += 32u)
                        {
                            uint32_t m;
                            if(Q.share_n <= kTailAhead * NT) m = obits;
                            else if(w < kTailBitWords) m = s_bits[w * NT + threadIdx.x];
                            else m = reactivated32(Q, i, n1);
                            for(; m; m &= m - 1u)
                                {
                                    if(KGMT_BOUND(pos < Q.capacity)) Q.rep_old[pos] = i + (uint32_t)(__ffs((int)m) - 1);
                                    ++pos;
                                }
                        }
                }
            if(ca)
                {
                    const uint32_t cap = s_p.capacity;
                    uint32_t iw = w_before + (ex & ((1u << kRepeatBits) - 1u)), idx = first;
                    for(uint32_t i = i0; i < i1; ++i)
                        {
                            if(!(s_word[i] >> 31)) continue;
                            const uint32_t w = (sparse_bits >> (i - i0)) & 1u ? kRepeatSparse : kRepeatDense;
                            for(uint32_t r = 0; r < w; ++r, ++iw)
                                if(iw < cap) s_p.rep_new[iw] = idx;
                            ++idx;
                        }
                }
            __syncthreads();
            if(!meet(ts, next, s_goal_min, s_pay, limit, 1u, &sched->error)) return;

            // ---- finalise (KGMT.cu:88-95, 380-403); every block computes the
            // same state, block 0 writes it back ----
            if(threadIdx.x < G && (uint32_t)s_pay[threadIdx.x] != kNone)
                {
                    // the query whose samples that block had
                    for(int q = 0; q < nq; ++q)
                        if(tq[q].status == KGMT_QUERY_RUNNING && threadIdx.x - tq[q].sample0 < tq[q].samples_nb)
                            atomicMin(&s_goal[q], (uint32_t)s_pay[threadIdx.x]);
                }
            __syncthreads();
            if((int)threadIdx.x < nq)
                {
                    TailQuery& Q = tq[threadIdx.x];
                    if(Q.status == KGMT_QUERY_RUNNING)
                        {
                            const uint32_t goal = s_goal[threadIdx.x];
                            const uint32_t tree = Q.tree + Q.n_next;
                            uint32_t status = KGMT_QUERY_RUNNING;
                            if(goal != kNone) status = KGMT_QUERY_SUCCESS;
                            else if(Q.itr >= Q.max_iterations) status = KGMT_QUERY_ITER_LIMIT;
                            else if(tree >= Q.capacity) status = KGMT_QUERY_CAPACITY;
                            Q.drawn += Q.n_samples;
                            Q.tree = tree;
                            QueryState& st = S[Q.slot];
                            if(b == 0)
                                {
                                    st.tree_size = tree;
                                    st.samples_drawn = Q.drawn;
                                    st.n_react = Q.n_react;
                                    st.w_new = Q.w_new;
                                    st.f_accept = Q.fa;
                                }
                            if(status != KGMT_QUERY_RUNNING)
                                {
                                    Q.status = status;
                                    if(b == 0)
                                        {
                                            if(status == KGMT_QUERY_SUCCESS) st.goal_index = (int32_t)goal;
                                            st.t_end = globaltimer();
                                            st.status = status;
                                        }
                                }
                            else
                                {
                                    Q.itr += 1;
                                    plan_samples_vals(Q.capacity, Q.samples_per_node, tree, Q.n_react + Q.w_new, &Q.spe, &Q.n_samples);
                                    if(b == 0)
                                        {
                                            st.itr = Q.itr;
                                            st.spe = Q.spe;
                                            st.n_samples = Q.n_samples;
                                        }
                                }
                        }
                }
            __syncthreads();
            ++iters;
        }
    if(threadIdx.x == 0) flush();

    // ---- hand the state back: the chain's schedule of what is left ----
    if(b == 0)
        {
            if(threadIdx.x == 0)
                {
                    ts->iterations = iters;
                    ts->declined = declined;
                    ts->arrived = next.target;
                    atomicAdd(&sched->iterations, iters);
                    if(host_words)
                        {
                            *(volatile uint32_t*)&host_words[0] = iters;
                            *(volatile uint32_t*)&host_words[1] = declined;
                        }
                }
            __syncthreads();
            compute_schedule<NT, false>(P, S, sched, tile_a_base, tile_c_base, tile_c_old);
        }
}

}  // namespace kgmt
