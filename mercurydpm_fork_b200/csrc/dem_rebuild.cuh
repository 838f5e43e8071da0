// dem_rebuild.cuh -- the neighbour-list rebuild as one cooperative kernel.
//
// k_rebuild opens every time step (a cooperative launch: all its blocks are
// resident together). Every block decides from the same fields of the control record, which no thread of this launch writes unless it
// rebuilds, whether the skin budget is spent (the Verlet-skin test restating
// MercuryBase::hGridNeedsRebuilding, MercuryBase.cc:496-535); if not, it returns
// at once. One thread writes the step's view of the buffers (StepView). A
// control kernel of its own before it cost 2 to 3 us of a step, and 21 us with
// the 1,024 walls of a batch on its one block; deciding in k_sum's last block
// instead held every block of it at a fence (a step of the 1,000,000 drum 6 %
// slower). One launch that usually does nothing costs less than a graph
// conditional node around ten kernels. When the budget is spent, the blocks run
// the steps below in turn, separated by grid barriers:
//
//   1 cell keys per HGrid level and counts per cell         (keys_one)
//   2 total of the counts of one chunk of cells per block
//   3 exclusive scan of the chunk from the sum of the totals before it
//   4 counting-sort scatter                                 (scatter_one)
//   5 per-cell ordering by particle id, counters reset      (cell_sort_one)
//   6 permutation gather of the state                       (gather_one)
//   7 neighbour lists; each block takes the unit numbers of its
//     particles from one counter                            (build_one)
//   8 the units and, per list entry, its unit               (units_one)
//   9 contact history of the old units to the new ones      (carry_one)
//
// and block 0 makes the new state buffer and lists current. (The unit ranges
// of different blocks follow each other in any order: no result depends on
// a unit's number.) This replaces
// the HGrid buckets and the InteractionHandler lookup of the reference
// (Mercury3D.cc:224-416, InteractionHandler.cc:103-174).
//
// The barrier counter only grows: each rebuild adds gridDim.x arrivals per
// barrier, so a launch finds its base as the multiple of gridDim.x *
// RB_BARRIERS below the counter's value at its start (no block can pass the
// first barrier before every block has read it). Every wait is bounded: a
// block that polls RB_POLL_LIMIT times sets DEM_ERR_TIMEOUT and returns, and
// the host resets the counter when it sees that status.
#pragma once
#include "dem_pipeline.cuh"

namespace dem {

constexpr int RB_BLOCK = 256;
constexpr int RB_BARRIERS = 8;
constexpr long long RB_POLL_LIMIT = 1ll << 24;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

struct GridBarrier {
    unsigned long long* ctr;
    unsigned long long base;
    unsigned int passed;
};

// Thread 0 of the block waits until the counter reaches target, at most
// `limit` polls; false (and DEM_ERR_TIMEOUT in *status) if it gave up.
__device__ __forceinline__ bool wait_counter(const unsigned long long* ctr, unsigned long long target,
                                             unsigned int* status, long long limit)
{
    long long polls = 0;
    while (ld_acquire_u64(ctr) < target) {
        if (++polls > limit) {
            atomicOr(status, 1u << DEM_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(64);
    }
    return true;
}

// All blocks of the launch meet; false if this block gave up waiting.
__device__ __forceinline__ bool grid_barrier(GridBarrier& g, Control* ctl)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ++g.passed;
        __threadfence();
        atomicAdd(g.ctr, 1ull);
        const unsigned long long target = g.base + (unsigned long long)g.passed * gridDim.x;
        ok = wait_counter(g.ctr, target, &ctl->status, RB_POLL_LIMIT) ? 1 : 0;
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// Self-test of the bounded wait: every block arrives at a barrier whose
// target one block more than the grid would have to reach, so every wait
// runs out after `limit` polls, sets DEM_ERR_TIMEOUT in *status and returns.
// Its counter is its own (reset by the caller before the launch).
__global__ void __launch_bounds__(RB_BLOCK) k_barrier_expiry(unsigned long long* ctr, unsigned int* status,
                                                             long long limit)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(ctr, 1ull);
        wait_counter(ctr, (unsigned long long)gridDim.x + 1ull, status, limit);
    }
    __syncthreads();
}

// Sum of one int per thread over the block (RB_BLOCK threads).
__device__ __forceinline__ int block_sum(int v, int* warp_sums)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < RB_BLOCK / 32; ++w) total += warp_sums[w];
    __syncthreads();
    return total;
}

// step: 1 the launch opens a time step; 0 it only brings the lists up to date
// (before the initial evaluation). In most steps the launch is its first few
// loads alone: the pointers stay in the constant bank (__grid_constant__) and no
// load waits for another (a step of a box of 1,000: 17.4 -> 17.0 us).
__global__ void __launch_bounds__(RB_BLOCK, 3) k_rebuild(const __grid_constant__ DevPtrs d, unsigned long long* barrier_ctr, int step)
{
    Control* ctl = d.ctl;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
    // read by every block before the first barrier
    const int flip = ctl->pending_flip;
    const int hc = ctl->cur, lo = ctl->lbuf, hh = ctl->hcur ^ flip;
    const double spent = step ? spent_skin(ctl) : 0.0;
    const int age = ctl->list_age + step;
    // without short cuts: the fields arrive together
    const bool go = (ctl->force_rebuild != 0) | ((step != 0) & ((2.0 * spent >= ctl->skin) | (age >= d.wall_steps)));
    if (gt == 0) {
        StepView& v = ctl->view;
        v.pcur = ctl->pcur ^ flip;
        v.final_step = !step || ctl->steps_left <= 1;
        v.first_step = step && ctl->steps_done == 0;
        if (step && v.final_step) ctl->n_records = 0; // records describe the last evaluation only
        if (!go) {
            v.cur = hc;
            v.lbuf = lo;
            v.hcur = hh;
            ctl->next_disp_acc = spent;
            ctl->next_list_age = age;
        }
    }
    if (!go) return;
    __shared__ unsigned long long base_s;
    __shared__ int warp_sums[RB_BLOCK / 32];
    const int old_units = min(ctl->n_units, d.unit_cap);
    if (threadIdx.x == 0) {
        const unsigned long long per = (unsigned long long)gridDim.x * RB_BARRIERS;
        base_s = ld_acquire_u64(barrier_ctr) / per * per;
    }
    __syncthreads();
    GridBarrier g{barrier_ctr, base_s, 0u};

    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->n_units_next = 0;

    // 1 keys and counts
    for (int i = gt; i < d.n; i += gs) keys_one(d, i, hc);
    if (!grid_barrier(g, ctl)) return;

    // 2 total of this block's chunk of cells. A thread takes 16 cells of a tile in
    // 16-byte loads: a batch of 1,024 heaps has 22 million cells, mostly empty, and
    // a tile of one cell a thread made 195 dependent steps of 2 and 3.
    constexpr int PER = 16, TILE = PER * RB_BLOCK;
    const int tiles = (d.ncells + TILE - 1) / TILE;
    const int per_block = (tiles + gridDim.x - 1) / gridDim.x;
    const long long c0 = min((long long)d.ncells, (long long)blockIdx.x * per_block * TILE);
    const long long c1 = min((long long)d.ncells, c0 + (long long)per_block * TILE);
    auto load16 = [&](long long at, int (&v)[PER]) {
        if (at + PER <= c1) {
            const int4* p = reinterpret_cast<const int4*>(d.cell_count + at); // at: a multiple of 16
#pragma unroll
            for (int q = 0; q < PER / 4; ++q) {
                const int4 x = p[q];
                v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < PER; ++q) v[q] = at + q < c1 ? d.cell_count[at + q] : 0;
        }
    };
    int total = 0;
    for (long long t0 = c0; t0 < c1; t0 += TILE) {
        int v[PER];
        load16(t0 + (long long)threadIdx.x * PER, v);
#pragma unroll
        for (int q = 0; q < PER; ++q) total += v[q];
    }
    total = block_sum(total, warp_sums);
    if (threadIdx.x == 0) d.block_sums[blockIdx.x] = total;
    if (!grid_barrier(g, ctl)) return;

    // 3 scan from the totals of the chunks before
    int part = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += RB_BLOCK) part += d.block_sums[b];
    int before = block_sum(part, warp_sums);
    for (long long t0 = c0; t0 < c1; t0 += TILE) {
        const long long at = t0 + (long long)threadIdx.x * PER;
        int v[PER], mine = 0;
        load16(at, v);
#pragma unroll
        for (int q = 0; q < PER; ++q) mine += v[q];
        int tile_total;
        int run = before + block_exclusive_scan(mine, warp_sums, tile_total);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int x = v[q];
            v[q] = run;
            run += x;
        }
        if (at + PER <= c1) {
            int4* p = reinterpret_cast<int4*>(d.cell_start + at);
#pragma unroll
            for (int q = 0; q < PER / 4; ++q) p[q] = make_int4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else {
#pragma unroll
            for (int q = 0; q < PER; ++q)
                if (at + q < c1) d.cell_start[at + q] = v[q];
        }
        before += tile_total;
        __syncthreads(); // warp_sums is reused by the next tile
    }
    if (c0 < c1 && c1 == d.ncells && threadIdx.x == 0) d.cell_start[d.ncells] = before;
    if (!grid_barrier(g, ctl)) return;

    // 4 scatter
    for (int i = gt; i < d.n; i += gs) scatter_one(d, i);
    if (!grid_barrier(g, ctl)) return;

    // 5 id order inside each cell
    for (int i = gt; i < d.n; i += gs) cell_sort_one(d, i, hc);
    if (!grid_barrier(g, ctl)) return;

    // 6 gather
    for (int s = gt; s < d.n; s += gs) gather_one(d, s, hc);
    if (!grid_barrier(g, ctl)) return;

    // 7 lists, then the block's range of unit numbers
    __shared__ int unit_base;
    for (int s0 = blockIdx.x * RB_BLOCK; s0 < d.n; s0 += gs) {
        const int s = s0 + threadIdx.x;
        int pairs = 0, walls = 0;
        if (s < d.n) build_one(d, s, hc ^ 1, pairs, walls);
        int total;
        const int ex = block_exclusive_scan(pairs + walls, warp_sums, total);
        if (threadIdx.x == 0) unit_base = atomicAdd(&ctl->n_units_next, total);
        __syncthreads();
        if (s < d.n) d.ubase[s] = unit_base + ex;
    }
    if (!grid_barrier(g, ctl)) return;

    // 8 units of the new lists
    for (int s = gt; s < d.n; s += gs) {
        if (d.has_tri) carry_triangles(d, s, hh, hc);
        units_one(d, s, lo ^ 1, hh ^ 1, hc ^ 1);
    }
    if (!grid_barrier(g, ctl)) return;

    // 9 history
    for (int j = gt; j < old_units; j += gs) carry_one(d, j, lo, hh, hc);
    if (d.has_tri) // particles without a triangle unit have no history in the buffer written next either
        for (int s = gt; s < d.n; s += gs)
            if (!d.wact[hh ^ 1][s]) d.wact[hh][s] = 0u;

    if (blockIdx.x == 0 && threadIdx.x == 0) { // the gathered state and the new lists become current
        StepView& v = ctl->view;
        v.cur = ctl->cur = hc ^ 1;
        v.lbuf = ctl->lbuf = lo ^ 1;
        v.hcur = ctl->hcur = hh ^ 1;
        ctl->pcur = v.pcur;
        ctl->pending_flip = 0;
        ctl->n_units = min(ctl->n_units_next, d.unit_cap);
        ctl->disp_acc = ctl->next_disp_acc = 0.0;
        ctl->list_age = ctl->next_list_age = 0;
        ctl->force_rebuild = 0;
        ctl->n_rebuilds += 1;
    }
}

} // namespace dem
