// dem_pipeline.cuh -- one force evaluation as two kernels over the flat unit
// list of the last rebuild (pairs with the lower id first, particle-wall
// candidates), each contact's law evaluated once:
//
//   k_units    persistent blocks, a chunk of units at a time: the exact contact
//              predicate (BaseParticle::getInteractionWith,
//              BaseParticle.cc:688-710), one unit per thread with several in
//              flight; the block's contacts, compacted in shared memory, then
//              take the contact law with full warps (DPMBase::
//              computeInternalForce, DPMBase.cc:3113-3162; walls:
//              DPMBase.cc:3188-3215) with the spring of the unit's last
//              contact, and leave the force/torque shares of P and I at their
//              item. A pair that meets across a periodic boundary is two views,
//              each real particle against the other's ghost
//              (DPMBase.cc:3124-3139), evaluated by the same thread.
//   k_tri      (only with triangle walls) one thread per particle with
//              triangle-wall contacts in reach: the reference's wall loop for
//              them with group merging and overlap weighting, into one item.
//   k_sum      one thread per particle: the shares in neighbour-list order,
//              the body force (DPMBase.cc:3168-3179), then the wall shares --
//              the order the sequential code adds them -- then the
//              integration.
//
// Items are numbered by atomics; each particle adds its shares in its own
// list order, so results do not depend on them.
//
#pragma once
#include "dem_kernels.cuh"

namespace dem {

// One triangle contact of the initial evaluation (k_tri): wall, creation key,
// overlap, normal, force, torque, contact point, species, normal elastic
// energy, springs.
constexpr int TRI_REC = 26;
constexpr int SHARE = 12;            // doubles per item: P force, P torque, I force, I torque
// Launch shapes. k_units is compiled for 3 to 6 resident blocks per SM and
// k_sum for blocks of 64, 128 and 256 threads; the handle keeps the choice
// (dem_autotune measures the variants on the live state).
constexpr int UNIT_BLOCK = 128;
constexpr int UNIT_CHUNK_PER_TUNE = 4;   // units a block takes at a time: at most 4 x dem_tuning.detect_block
constexpr int UNIT_CHUNK_MAX = 256 * UNIT_CHUNK_PER_TUNE;
constexpr int DETECT_TUNE = 128;         // the default dem_tuning.detect_block
constexpr int SUM_BLOCK = 128;           // the default k_sum block
constexpr int SUM_THREADS_PER_SM = 640;  // k_sum's launch bounds: 640 / block resident blocks per SM

// Shared-memory copies of the instance record (when there is one instance)
// and of the species-pair table (when it has at most SP_STAGE_MAX entries),
// staged by k_units' blocks before their first contact: the contact law's
// parameters are then no dependent global loads.
constexpr int SP_STAGE_MAX = 16;
struct TableStage {
    __align__(16) unsigned char inst[sizeof(InstanceDev)];
    __align__(16) unsigned char sp[SP_STAGE_MAX * sizeof(dem_species_pair)];
};
static_assert(sizeof(InstanceDev) % 4 == 0 && sizeof(dem_species_pair) % 4 == 0, "staged as 32-bit words");

// Called by every thread of the block; the copies are there after the block's
// next barrier.
__device__ __forceinline__ void stage_tables(const DevPtrs& d, TableStage& st)
{
    if (d.single_instance) {
        const int* src = reinterpret_cast<const int*>(d.inst);
        int* dst = reinterpret_cast<int*>(st.inst);
        for (int k = threadIdx.x; k < (int)(sizeof(InstanceDev) / 4); k += blockDim.x) dst[k] = src[k];
    }
    if (d.n_species_table <= SP_STAGE_MAX) {
        const int* src = reinterpret_cast<const int*>(d.species);
        int* dst = reinterpret_cast<int*>(st.sp);
        const int words = d.n_species_table * (int)(sizeof(dem_species_pair) / 4);
        for (int k = threadIdx.x; k < words; k += blockDim.x) dst[k] = src[k];
    }
}

__device__ __forceinline__ const InstanceDev& staged_inst(const DevPtrs& d, const TableStage& st, int z)
{
    return d.single_instance ? *reinterpret_cast<const InstanceDev*>(st.inst) : d.inst[z];
}

__device__ __forceinline__ const dem_species_pair* staged_species(const DevPtrs& d, const TableStage& st)
{
    return d.n_species_table <= SP_STAGE_MAX ? reinterpret_cast<const dem_species_pair*>(st.sp) : d.species;
}

// Position of s in the particle-major row of t (the first 16 entries come
// from `head`, read ahead by the caller); -1 if absent.
__device__ __forceinline__ int find_in_row(const DevPtrs& d, int s, int t, int ct, const int4 (&head)[4])
{
    const int4* row = reinterpret_cast<const int4*>(d.rows + (size_t)t * d.cap); // cap is a multiple of 32
    for (int m0 = 0; m0 < ct; m0 += 16) {
        int4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = m0 == 0 ? head[j] : ((m0 + 4 * j < ct) ? row[(m0 >> 2) + j] : make_int4(-1, -1, -1, -1));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = m0 + 4 * j;
            if (q + 0 < ct && v[j].x == s) return q + 0;
            if (q + 1 < ct && v[j].y == s) return q + 1;
            if (q + 2 < ct && v[j].z == s) return q + 2;
            if (q + 3 < ct && v[j].w == s) return q + 3;
        }
    }
    return -1;
}

// Number of entries before k that particle s owns (the rank of entry k's pair
// among its units).
__device__ __forceinline__ int own_rank(const DevPtrs& d, int s, int k)
{
    int r = 0;
    for (int w = 0; w < (k >> 5); ++w) r += __popc(d.own[(size_t)w * d.ncap + s]);
    return r + __popc(d.own[(size_t)(k >> 5) * d.ncap + s] & ((1u << (k & 31)) - 1u));
}

// The units of particle s after a rebuild (list buffer l, uidx buffer h, state
// buffer nb): its own pairs, each filed in both particles' entries (the partner's row is
// searched for s; the lists are symmetric), two at a time with the first 16
// entries of both rows in flight together, then its walls. None has a
// history yet.
__device__ __forceinline__ void units_one(const DevPtrs& d, int s, int l, int h, int nb)
{
    const int cnt = min(d.cnt[s], d.cap);
    const int base = d.ubase[s];
    int u = base, pairs = 0;
    for (int w = 0; 32 * w < cnt; ++w) {
        const int left = cnt - 32 * w;
        unsigned int todo = d.own[(size_t)w * d.ncap + s] & (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
        pairs += __popc(todo);
        while (todo) {
            int t[2], ct[2], k[2];
            int4 head[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                t[j] = -1;
                if (todo) {
                    k[j] = 32 * w + __ffs(todo) - 1;
                    todo &= todo - 1;
                    t[j] = d.rows[(size_t)s * d.cap + k[j]];
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (t[j] >= 0) {
                    ct[j] = d.cnt[t[j]];
                    const int4* row = reinterpret_cast<const int4*>(d.rows + (size_t)t[j] * d.cap);
#pragma unroll
                    for (int q = 0; q < 4; ++q) head[j][q] = row[q]; // 16 <= cap entries: inside the row
                }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (t[j] < 0) continue;
                const int m = find_in_row(d, s, t[j], min(ct[j], d.cap), head[j]);
                // an asymmetric pair (the partner's row overflowed) or too many of them: no unit
                if (m < 0 || (unsigned)u >= (unsigned)d.unit_cap) {
                    atomicOr(&d.ctl->status, 1u << DEM_ERR_CAPACITY);
                    continue;
                }
                d.epair[nbr_at(d.ncap, t[j], m)] = u;
                d.epair[nbr_at(d.ncap, s, k[j])] = u;
                d.unit[l][u] = make_int2(s, t[j]);
                d.uidx[h][u] = UIDX_NONE;
                ++u;
            }
        }
    }
    for (; u < base + pairs; ++u) // units of pairs left out above
        if ((unsigned)u < (unsigned)d.unit_cap) {
            d.unit[l][u] = make_int2(-1, -1);
            d.uidx[h][u] = UIDX_NONE;
        }
    const unsigned int mask = d.wcand[s];
    d.wbase[s] = u;
    if (!mask) return;
    const unsigned int tri = d.has_tri ? d.inst[d.info[nb][s].z].tri_mask : 0u;
    const int n_walls = __popc(mask & ~tri) + ((mask & tri) ? 1 : 0);
    if ((unsigned)u + n_walls > (unsigned)d.unit_cap) {
        atomicOr(&d.ctl->status, 1u << DEM_ERR_CAPACITY);
        d.wcand[s] = 0u;
        return;
    }
    for (unsigned int b = mask & ~tri; b; b &= b - 1, ++u) {
        d.unit[l][u] = make_int2(s, ~(__ffs(b) - 1));
        d.uidx[h][u] = UIDX_NONE;
    }
    if (mask & tri) {
        d.unit[l][u] = make_int2(s, UNIT_TRI);
        d.uidx[h][u] = UIDX_NONE;
    }
}

// The history of old unit j (list buffer l, uidx buffer h, state buffer c)
// moves to the same pair or wall of the new list.
__device__ __forceinline__ void carry_one(const DevPtrs& d, int j, int l, int h, int c)
{
    const int v = d.uidx[h][j];
    if (v == UIDX_NONE) return;
    const int2 old = d.unit[l][j];
    if (old.x < 0 || old.y == UNIT_TRI) return; // a triangle history moves with the particle (carry_triangles)
    const int s = d.newidx[old.x];
    int u = -1;
    if (old.y >= 0) {
        const int t = d.newidx[old.y];
        const int ct = min(d.cnt[s], d.cap);
        const int4* row = reinterpret_cast<const int4*>(d.rows + (size_t)s * d.cap);
        int4 head[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) head[q] = row[q];
        const int m = find_in_row(d, t, s, ct, head);
        if (m >= 0) u = d.ubase[s] + own_rank(d, s, m);
        else atomicAdd(&d.ctl->lost_history, 1u); // out of reach, or deleted
    } else {
        const unsigned int bit = 1u << ~old.y, mask = d.wcand[s];
        const unsigned int tri = d.has_tri ? d.inst[d.info[c][old.x].z].tri_mask : 0u;
        if (mask & bit) u = d.wbase[s] + __popc(mask & ~tri & (bit - 1u));
    }
    // the spring stays where it is in the pool; the new unit points at it
    if (u >= 0 && (unsigned)u < (unsigned)d.unit_cap) d.uidx[h ^ 1][u] = v;
}

// Exclusive block scan of one int per thread (any block of whole warps); returns
// this thread's offset and the block total through `total`.
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        if (w < wid) before += warp_sums[w];
        total += warp_sums[w];
    }
    return before + x - v;
}

// What the first time step does with a unit that had a contact in the initial
// evaluation and has none now: the interaction outlives the step
// (InteractionHandler::eraseOldInteractions erases stamps <= 0 only), so its
// spring moves to the top of the next pool, below which the items of this
// evaluation stay (k_sum checks that they met no carry).
template <int NCOMP>
__device__ __forceinline__ int keep_spring(const DevPtrs& d, int pc, int from_idx)
{
    const int top = d.item_cap - 1 - (int)atomicAdd(&d.ctl->n_carry, 1u);
    if (top < 0) {
        atomicOr(&d.ctl->status, 1u << DEM_ERR_CAPACITY);
        return UIDX_NONE;
    }
    const double2* from = reinterpret_cast<const double2*>(d.pool[pc] + pool_at(NCOMP, from_idx));
    double2* to = reinterpret_cast<double2*>(d.pool[pc ^ 1] + pool_at(NCOMP, top));
#pragma unroll
    for (int q = 0; q < hist_stride(NCOMP) / 2; ++q) to[q] = from[q];
    return uidx_kept(top);
}

// The triangle walls (bits) particle s is near enough to for k_tri: the
// bounding box and face-plane tests, with the reach widened to the instance's
// largest interaction distance. The history rows of the others are carried
// over the first time step (whist, wact).
template <int NCOMP>
__device__ __forceinline__ unsigned int near_triangles(const DevPtrs& d, const InstanceDev& I, int s, V3 x, double r,
                                                       int hc, bool first)
{
    const double R = r + I.max_interaction_distance;
    unsigned int hit = 0u, kept = 0u;
    for (unsigned int b = d.wcand[s] & I.tri_mask; b; b &= b - 1) {
        const int w = __ffs(b) - 1;
        const WallGeom& tg = d.wgeom[I.wall_begin + w];
        if (triangle_near(tg, x, R) && triangle_plane_near(tg, x, R)) hit |= 1u << w;
    }
    if (first)
        for (unsigned int b = d.wact[hc][s] & I.tri_mask & ~hit; b; b &= b - 1) {
            const int w = __ffs(b) - 1;
            kept |= 1u << w;
            for (int q = 0; q < hist_stride(NCOMP); ++q) // with the creation key
                d.whist[hc ^ 1][whist_at(d.ncap, NCOMP, s, w) + q] = d.whist[hc][whist_at(d.ncap, NCOMP, s, w) + q];
        }
    d.wact[hc ^ 1][s] = kept; // k_tri adds the triangles it makes contacts with
    if (!hit) d.slott[s] = -1;
    return hit;
}

// The predicate of a wall or triangle unit (out of line: few units are walls,
// and their geometry would cost the pair path its registers): bit 0 it
// touches, bit 1 an old contact of it may outlive the first time step.
template <int NCOMP>
__device__ __noinline__ int wall_unit_touches(const DevPtrs& d, int j, int2 u, int c, int hc, bool first)
{
    const double4 ps = d.pr[c][u.x];
    const int4 is = d.info[c][u.x];
    const InstanceDev& I = d.inst[is.z];
    if (u.y == UNIT_TRI) {
        const unsigned int mask = near_triangles<NCOMP>(d, I, u.x, xyz(ps), ps.w, hc, first);
        d.uidx[hc ^ 1][j] = (int)mask; // for k_tri's item (k_units reads it back)
        return mask != 0u ? 1 : 0;
    }
    const int w = ~u.y, wg = I.wall_begin + w;
    if ((I.wall_off_mask >> w) & 1u) return 0;
    const dem_wall& wall = d.walls[wg];
    const dem_species_pair& sp = d.species[I.species_offset + is.y * I.n_species + wall.species];
    double dist;
    V3 nrm;
    return wall_distance(wall, d.wgeom + wg, xyz(ps), ps.w + sp.interaction_distance, dist, nrm) ? 3 : 2;
}

// Outward normal (x, y, z) of the wall unit (s, ~w) touches and the distance
// from it (w), out of line for the same reason, and called while little else is
// live (DPMBase::computeForcesDueToWalls / BaseWall::getInteractionWith,
// DPMBase.cc:3188-3215, BaseWall.cc:367-437).
__device__ __noinline__ double4 wall_normal_distance(const DevPtrs& d, int c, int s, int w)
{
    const double4 ps = d.pr[c][s];
    const int4 is = d.info[c][s];
    const InstanceDev& I = d.inst[is.z];
    const int wg = I.wall_begin + w;
    const dem_wall& wall = d.walls[wg];
    double dist;
    V3 nrm;
    wall_distance(wall, d.wgeom + wg, xyz(ps),
                  ps.w + d.species[I.species_offset + is.y * I.n_species + wall.species].interaction_distance, dist, nrm);
    return make_double4(nrm.x, nrm.y, nrm.z, dist);
}

// RECORD: this launch may be the last force evaluation of a dem_step call,
// which writes the contact records; the steps before it are launched with
// RECORD = false, a variant without the record path (fewer registers).
// MINB: resident blocks per SM the registers are budgeted for (4: 128
// registers a thread; 5: 102; 6: 85; 3: 168), i.e. warps in flight against
// spills; the time-step variant is compiled for 3 to 6 (dem_autotune).
//
// Bound by the latency of its gathers and of the laws' FP64 division and
// square-root chains, not by DRAM. One flat list of owned pairs and walls
// instead of a thread per particle walking its row: no divergence in the
// predicate, UNITS_IN_FLIGHT gathers per thread, and neither an item list nor
// per-entry marks pass through HBM between a detecting and an evaluating
// kernel. A launch takes equal chunks: with few units every block gets one of
// at least a warp, so a small system still spreads over all SMs. A time step with
// the three kernels that walked rows and passed an item list, against one with
// this kernel and k_sum (k_rebuild's launch included in both): box of 5,000 27.5
// and 18.5 us, drum of 30,011 38 and 23 us, 50,000 spheres on 32 triangles 74 and
// 23 us, drum of 1,000,000 0.41 and 0.37 ms.
template <int MODE, int NLAW, int FLAW, int NCOMP, bool RECORD, int MINB = 4>
__global__ void __launch_bounds__(UNIT_BLOCK, MINB) k_units(const __grid_constant__ DevPtrs d, int chunk_max)
{
    // more spills at these budgets (a step of the 1,000,000 drum: 290 us with 2, 301 us with 4)
    constexpr int UNITS_IN_FLIGHT = 2;
    __shared__ TableStage tables;
    __shared__ unsigned short hit_of[UNIT_CHUNK_MAX];
    __shared__ int n_hit, item0;
    Control* ctl = d.ctl;
    const StepView& view = ctl->view;
    const int c = view.cur, l = view.lbuf, hc = view.hcur, hn = hc ^ 1, pc = view.pcur;
    const bool record = RECORD && (MODE == 0 || view.final_step) && ctl->record;
    const bool first = (MODE == 1) && view.first_step;
    if (blockIdx.x == 0 && threadIdx.x == 0 && !ctl->spare) { // no kernel of this evaluation reads these
        ctl->hcur = hc;
        ctl->pcur = pc;
        ctl->pending_flip = 1; // this evaluation writes the other pool and uidx
        ctl->force_rebuild = 0;
        if (MODE == 1) {
            ctl->disp_acc = ctl->next_disp_acc;
            ctl->list_age = ctl->next_list_age;
            ctl->step_disp2_bits = 0ull;
            ctl->steps_left -= 1;
            ctl->steps_done += 1;
        }
    }
    const int n_units = min(ctl->n_units, d.unit_cap);
    const double dt = d.dt;
    stage_tables(d, tables);
    if (threadIdx.x == 0) n_hit = 0;
    const dem_species_pair* species = staged_species(d, tables);
    const bool need_info = !d.single_instance || d.n_species_table > 1; // else instance 0, species 0
    const double4* pr = d.pr[c];
    const int4* info = d.info[c];
    const int2* unit = d.unit[l];
    // equal chunks of at most chunk_max units, a multiple of a warp each
    const long long most = (long long)gridDim.x * chunk_max;
    const long long passes = (n_units + most - 1) / most;
    const int chunk = passes ? (int)(((n_units + passes * gridDim.x - 1) / (passes * gridDim.x) + 31) / 32) * 32 : 32;

    for (unsigned int c0u = blockIdx.x * (unsigned int)chunk; c0u < (unsigned int)n_units;
         c0u += gridDim.x * (unsigned int)chunk) {
        const int c0 = (int)c0u;
        const int m = min(chunk, n_units - c0);
        // ---- the predicate ----
        unsigned int hits = 0u, others = 0u; // bit i: unit c0 + threadIdx.x + i * UNIT_BLOCK touches / is no pair
#pragma unroll 1
        for (int i0 = 0; i0 * UNIT_BLOCK < m; i0 += UNITS_IN_FLIGHT) {
            int2 un[UNITS_IN_FLIGHT];
            double4 ps[UNITS_IN_FLIGHT], pt[UNITS_IN_FLIGHT];
#pragma unroll
            for (int i = 0; i < UNITS_IN_FLIGHT; ++i) {
                const int k = threadIdx.x + (i0 + i) * UNIT_BLOCK;
                un[i] = k < m ? unit[c0 + k] : make_int2(-1, -1);
            }
#pragma unroll
            for (int i = 0; i < UNITS_IN_FLIGHT; ++i)
                if (un[i].y >= 0) {
                    ps[i] = pr[un[i].x];
                    pt[i] = pr[un[i].y];
                }
#pragma unroll
            for (int i = 0; i < UNITS_IN_FLIGHT; ++i) {
                const int2 u = un[i];
                if (u.y < 0) {
                    if (u.x >= 0) others |= 1u << (i0 + i);
                    continue;
                }
                double idist = 0.0; // x + 0.0 == x: skipping the lookup keeps the predicate exact
                V3 xt = xyz(pt[i]);
                bool periodic = false;
                if (d.any_periodic || !d.zero_idist) {
                    const InstanceDev& I = d.inst[d.single_instance ? 0 : info[u.x].z];
                    if (!d.zero_idist)
                        idist = d.species[I.species_offset + info[u.x].y * I.n_species + info[u.y].y].interaction_distance;
                    xt = image_of(I, xyz(ps[i]), xt, periodic);
                }
                const double sum = pt[i].w + ps[i].w + idist; // rI + rP + distance (BaseParticle.cc:695-697)
                bool hit = !(len2(xyz(ps[i]) - xt) >= sum * sum);
                if (periodic && !hit) { // the partner's own view of a periodic pair
                    const V3 xs = image_of(d.inst[d.single_instance ? 0 : info[u.x].z], xyz(pt[i]), xyz(ps[i]), periodic);
                    hit = !(len2(xyz(pt[i]) - xs) >= sum * sum);
                }
                if (hit) {
                    hits |= 1u << (i0 + i);
                } else {
                    const int j = c0 + threadIdx.x + (i0 + i) * UNIT_BLOCK;
                    int v = UIDX_NONE;
                    if (first) {
                        const int from = uidx_spring(d.uidx[hc][j]);
                        if (from >= 0) v = keep_spring<NCOMP>(d, pc, from);
                    }
                    d.uidx[hn][j] = v;
                }
            }
        }
        for (unsigned int b = others; b; b &= b - 1) {
            const int i = __ffs(b) - 1, j = c0 + threadIdx.x + i * UNIT_BLOCK;
            const int2 u = unit[j];
            const int touch = wall_unit_touches<NCOMP>(d, j, u, c, hc, first);
            if (touch & 1) {
                hits |= 1u << i;
            } else if (u.y != UNIT_TRI) {
                int v = UIDX_NONE;
                if (first && touch) {
                    const int from = uidx_spring(d.uidx[hc][j]);
                    if (from >= 0) v = keep_spring<NCOMP>(d, pc, from);
                }
                d.uidx[hn][j] = v;
            }
        }
        // ---- the block's contacts ----
        __syncthreads(); // n_hit is 0, the tables are staged, the last chunk's hit_of is read
        for (unsigned int b = hits; b; b &= b - 1)
            hit_of[atomicAdd(&n_hit, 1)] = (unsigned short)(threadIdx.x + (__ffs(b) - 1) * UNIT_BLOCK);
        __syncthreads();
        const int n_here = n_hit;
        if (threadIdx.x == 0 && n_here) item0 = (int)atomicAdd(&ctl->n_items, (unsigned)n_here);
        __syncthreads();
        if (threadIdx.x == 0) n_hit = 0;
        if (n_here && item0 + n_here > d.item_cap) {
            if (threadIdx.x == 0) atomicOr(&ctl->status, 1u << DEM_ERR_CAPACITY);
            for (int h = threadIdx.x; h < n_here; h += UNIT_BLOCK) {
                const int j = c0 + hit_of[h];
                d.uidx[hn][j] = UIDX_NONE;
                if (unit[j].y == UNIT_TRI) d.slott[unit[j].x] = -1;
            }
            continue;
        }
        for (int h = threadIdx.x; h < n_here; h += UNIT_BLOCK) {
            const int j = c0 + hit_of[h];
            const int q = item0 + h;
            const int2 u = unit[j];
            if (d.has_tri && u.y == UNIT_TRI) { // its net share is summed after the other walls' shares
                d.slott[u.x] = q;
                d.tri_list[atomicAdd(&ctl->n_tri, 1u)] = make_int4(u.x, q, d.uidx[hn][j], 0);
                continue;
            }
            const int from = uidx_spring(d.uidx[hc][j]);
            d.uidx[hn][j] = q;
            const bool is_wall = u.y < 0;
            // view 0: P is u.x, the lower id (or a wall's particle); view 1, only of
            // a periodic pair: P is the other real particle, against u.x's ghost
#pragma unroll 1
            for (int view = 0;; ++view) {
                const int s = view ? u.y : u.x, t = view ? u.x : u.y;
                ContactGeom g;
                if (is_wall) {
                    const double4 nd = wall_normal_distance(d, c, s, ~t);
                    g.n = -xyz(nd);
                    g.distance = nd.w;
                }
                // the spring of the last evaluation (record 0 is read and not used when
                // there is none): read before anything else needs it
                Springs spr;
                load_springs(d.pool[pc], pool_at(NCOMP, max(from, 0)), NCOMP, spr);
                const double4 ps = pr[s];
                const double4 vs = d.vm[c][s];
                const double4 ws = d.wi[c][s];
                const int4 is = (need_info || record) ? info[s] : make_int4(0, 0, 0, 0);
                const InstanceDev& I = staged_inst(d, tables, is.z);
                const V3 xq = xyz(ps), vq = xyz(vs), wq = xyz(ws);
                const double rq = ps.w, mq = vs.w;
                const dem_species_pair* spp;
                bool periodic = false, touches = true;
                int pid_i = 0;
                V3 xt = zero3();
                if (is_wall) {
                    const int wg = I.wall_begin + ~t;
                    const dem_wall& wall = d.walls[wg];
                    spp = &species[I.species_offset + is.y * I.n_species + wall.species];
                    g.overlap = rq - g.distance;
                    g.c = xq - (rq - 0.5 * g.overlap) * g.n;
                    g.xp = xq; g.vp = vq; g.wp = wq; g.inv_mass_p = mq; g.curv_p = 1.0 / rq;
                    g.xi = v3(wall.position[0], wall.position[1], wall.position[2]);
                    g.vi = v3(wall.velocity[0], wall.velocity[1], wall.velocity[2]);
                    g.wi = v3(wall.angular_velocity[0], wall.angular_velocity[1], wall.angular_velocity[2]);
                    g.inv_mass_i = 0.0;
                    g.curv_i = 0.0;
                    g.i_is_wall = true;
                    pid_i = wg;
                } else {
                    const double4 pt = pr[t];
                    const double4 vt4 = d.vm[c][t];
                    const double4 wt4 = d.wi[c][t];
                    const int4 it = (need_info || record) ? info[t] : make_int4(0, 0, 0, 0);
                    xt = image_of(I, xq, xyz(pt), periodic);
                    const V3 branch = xq - xt;
                    const double d2 = len2(branch);
                    spp = &species[I.species_offset + is.y * I.n_species + it.y];
                    if (periodic) { // each view decides for itself
                        const double sum = pt.w + ps.w + spp->interaction_distance;
                        touches = !(d2 >= sum * sum);
                    }
                    g.distance = sqrt(d2);
                    g.n = branch / g.distance;
                    g.overlap = rq + pt.w - g.distance;
                    g.xp = xq; g.vp = vq; g.wp = wq; g.inv_mass_p = mq;
                    g.xi = xt; g.vi = xyz(vt4); g.wi = xyz(wt4); g.inv_mass_i = vt4.w;
                    g.c = g.xp - (rq - 0.5 * g.overlap) * g.n;
                    g.curv_p = 1.0 / rq;
                    g.curv_i = 1.0 / pt.w;
                    g.i_is_wall = false;
                    pid_i = it.x;
                }
                if (from < 0) {
                    spr.slide = zero3(); spr.roll = zero3(); spr.tors = zero3();
                } else if (view) {
                    // the higher-id side of a periodic pair restarts every step from the
                    // reversed spring of the lower-id side (InteractionHandler.cc:316-368,
                    // BaseInteraction::copySwitchPointer / reverseHistory)
                    spr.slide = -spr.slide; spr.roll = -spr.roll; spr.tors = -spr.tors;
                }
                ContactOut out;
                evaluate_contact<NLAW, FLAW>(*spp, g, spr, dt, out);
                // shares as 16-byte stores (96-byte items: every item and half is 16-byte aligned)
                double2* sh = reinterpret_cast<double2*>(d.shares + (size_t)q * SHARE) + 3 * view;
                V3 fp = out.force;
                V3 tp = out.torque - cross(xq - g.c, out.force);
                if (!touches) fp = tp = zero3();
                sh[0] = make_double2(fp.x, fp.y);
                sh[1] = make_double2(fp.z, tp.x);
                sh[2] = make_double2(tp.y, tp.z);
                if (view) break;
                // step 0 keeps the lower-id side's old spring of a periodic pair that
                // existed at the initial evaluation (equal stamps,
                // InteractionHandler.cc:339-352); read again here instead of kept in
                // registers. A view that does not touch keeps no spring, but for that step.
                if (periodic && ((first && from >= 0) || !touches)) {
                    spr.slide = zero3(); spr.roll = zero3(); spr.tors = zero3();
                    if (first && from >= 0) load_springs(d.pool[pc], pool_at(NCOMP, from), NCOMP, spr);
                }
                store_springs(d.pool[pc ^ 1], pool_at(NCOMP, q), NCOMP, spr);
                if (record && touches) {
                    const double meff = 1.0 / (g.inv_mass_p + g.inv_mass_i);
                    write_record(d, is.x, pid_i, is_wall ? 1 : 0, periodic ? 1 : 0, s, is_wall ? pid_i : t, g, out, spr,
                                 spring_energy(*spp, spr, meff));
                }
                if (is_wall) break;
                if (!periodic) { // I's share of an ordinary pair
                    const V3 fi = -out.force;
                    const V3 ti = -out.torque + cross(xt - g.c, out.force);
                    sh[3] = make_double2(fi.x, fi.y);
                    sh[4] = make_double2(fi.z, ti.x);
                    sh[5] = make_double2(ti.y, ti.z);
                    break;
                }
            }
        }
    }
}

// All triangle-wall contacts of one particle, in wall order, as the
// reference's sequential wall loop makes them with the triangle-wall
// correction on (its default build; DPMBase::computeForcesDueToWalls,
// DPMBase.cc:3188-3215):
//  * BaseWall::getInteractionWith (BaseWall.cc:375-409): a triangle of group
//    g > 0 meets every contact already made this step with a triangle of the
//    same group; unless both are face contacts, the larger overlap wins -- a
//    larger new overlap takes the earlier contact over (its force is taken
//    back, it moves to the new triangle with its spring), a smaller one drops
//    the new contact; otherwise the contact with this triangle from the last
//    step (InteractionHandler::getInteraction) or a new one is used.
//  * DPMBase::computeAllForces (DPMBase.cc:3443-3486): with two or more
//    triangle contacts, each force and torque is taken back and applied again
//    weighted by overlap / (sum of overlaps), at the contact point moved by
//    the same weight.
// The particle's net force and torque from these steps go into the item's P
// share; the springs of the contacts left go to their triangles' history rows.
// The contacts are visited in the particle's interaction-list order, which
// is creation order (BaseInteractable::addInteraction appends,
// removeInteraction erases in place): each triangle contact carries a
// creation key (the time step it was made x 16 + its rank within that
// step) in the pad word of its history row.
// The first time step shares its time stamp with the initial evaluation
// (both numberOfTimeSteps + 1 = 1), so there every contact of the initial
// evaluation counts as made this step: the group rule compares against all
// of them from the start, a triangle takes its own contact over from that
// list, and the weighting includes those not touched again. The initial
// evaluation keeps its contacts' state in tri_first for this.
constexpr int TRI_BLOCK = 64;
template <int MODE, int NLAW, int FLAW, int NCOMP>
__global__ void __launch_bounds__(TRI_BLOCK) k_tri(DevPtrs d)
{
    constexpr int MAXT = DEM_MAX_TRIANGLE_CONTACTS;
    static_assert(NCOMP % 2 == 1, "the pad word of a history row holds the creation key");
    Control* ctl = d.ctl;
    const int c = ctl->view.cur, hc = ctl->view.hcur, hn = hc ^ 1;
    const bool record = (MODE == 0 || ctl->view.final_step) && ctl->record;
    const bool first = (MODE == 1) && ctl->view.first_step;
    const int n_tri = min((int)ctl->n_tri, d.n);
    const double dt = d.dt;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_tri; t += gridDim.x * blockDim.x) {
        const int4 item = d.tri_list[t];
        const int s = item.x, q = item.y;
        const unsigned int mask = (unsigned int)item.z;
        const double4 ps = d.pr[c][s];
        const double4 vs = d.vm[c][s];
        const double4 ws = d.wi[c][s];
        const int4 is = d.info[c][s];
        const InstanceDev& I = d.inst[is.z];
        const int ns = I.n_species;
        const V3 xq = xyz(ps), vq = xyz(vs), wq = xyz(ws);
        const double rq = ps.w, mq = vs.w;
        const unsigned int was = d.wact[hc][s];
        int ew[MAXT], esw[MAXT], ord[MAXT]; // ord: entries in interaction-list order
        double eov[MAXT], eel[MAXT], ek[MAXT];
        const double step_key = 16.0 * (double)ctl->steps_done;
        int made = 0; // contacts made this step
        V3 en[MAXT], ec[MAXT], ef[MAXT], et[MAXT], etan[MAXT];
        Springs es[MAXT];
        int ne = 0;
        V3 F = zero3(), T = zero3();
        const int ci = d.caller[c][s];
        if (first) { // the initial evaluation's contacts, in list order
            const int n0 = min(d.tri_first_n[ci], MAXT);
            const double* rec = d.tri_first + (size_t)ci * MAXT * TRI_REC;
            for (int o = 0; o < n0; ++o, rec += TRI_REC) {
                ew[o] = (int)rec[0]; ek[o] = rec[1]; eov[o] = rec[2];
                en[o] = v3(rec[3], rec[4], rec[5]);
                ef[o] = v3(rec[6], rec[7], rec[8]);
                et[o] = v3(rec[9], rec[10], rec[11]);
                ec[o] = v3(rec[12], rec[13], rec[14]);
                esw[o] = (int)rec[15]; eel[o] = rec[16];
                es[o].slide = v3(rec[17], rec[18], rec[19]);
                es[o].roll = v3(rec[20], rec[21], rec[22]);
                es[o].tors = v3(rec[23], rec[24], rec[25]);
                etan[o] = zero3();
                ord[o] = o;
            }
            ne = n0;
        }
        for (unsigned int b = mask; b; b &= b - 1) {
            const int w = __ffs(b) - 1;
            const int wg = I.wall_begin + w;
            const dem_wall& wall = d.walls[wg];
            const dem_species_pair* spw = &d.species[I.species_offset + is.y * ns + wall.species];
            double dist;
            V3 nrm;
            if (!triangle_distance(d.wgeom[wg], xq, rq + spw->interaction_distance, dist, nrm)) continue;
            const double overlap = rq - dist;
            int k = -1;
            bool dropped = false;
            if (wall.group > 0) {
                const bool face = triangle_face_contact(d.wgeom[wg], nrm);
                for (int o = 0; o < ne; ++o) {
                    const int e = ord[o];
                    const int eg = I.wall_begin + ew[e];
                    if (d.walls[eg].group != wall.group) continue;
                    if (face && triangle_face_contact(d.wgeom[eg], en[e])) continue;
                    if (overlap > eov[e]) { // take e's force back; e moves to this triangle
                        F += -ef[e];
                        T += -et[e] + cross(xq - ec[e], ef[e]);
                        ew[e] = w;
                        k = e;
                    } else {
                        dropped = true;
                        break;
                    }
                }
            }
            if (dropped) continue;
            if (k < 0 && first) // InteractionHandler::getExistingInteraction: first in list order
                for (int o = 0; o < ne; ++o)
                    if (ew[ord[o]] == w) {
                        k = ord[o];
                        break;
                    }
            if (k < 0) {
                if (ne == MAXT) {
                    atomicOr(&ctl->status, 1u << DEM_ERR_CAPACITY);
                    continue;
                }
                k = ne;
                ew[k] = w;
                esw[k] = wall.species;
                es[k].slide = zero3(); es[k].roll = zero3(); es[k].tors = zero3();
                if (!first && ((was >> w) & 1u)) { // the contact with this triangle from the last step
                    const size_t hb = whist_at(d.ncap, NCOMP, s, w);
                    load_springs(d.whist[hc], hb, NCOMP, es[k]);
                    ek[k] = d.whist[hc][hb + NCOMP];
                } else {
                    ek[k] = step_key + (double)(made++);
                }
                int o = ne++; // insert by creation key
                while (o > 0 && ek[ord[o - 1]] > ek[k]) {
                    ord[o] = ord[o - 1];
                    --o;
                }
                ord[o] = k;
            }
            ContactGeom g;
            g.n = -nrm;
            g.distance = dist;
            g.overlap = overlap;
            g.c = xq - (rq - 0.5 * g.overlap) * g.n;
            g.xp = xq; g.vp = vq; g.wp = wq; g.inv_mass_p = mq; g.curv_p = 1.0 / rq;
            g.xi = v3(wall.position[0], wall.position[1], wall.position[2]);
            g.vi = v3(wall.velocity[0], wall.velocity[1], wall.velocity[2]);
            g.wi = v3(wall.angular_velocity[0], wall.angular_velocity[1], wall.angular_velocity[2]);
            g.inv_mass_i = 0.0;
            g.curv_i = 0.0;
            g.i_is_wall = true;
            ContactOut out;
            evaluate_contact<NLAW, FLAW>(d.species[I.species_offset + is.y * ns + esw[k]], g, es[k], dt, out);
            en[k] = g.n; eov[k] = g.overlap; ec[k] = g.c;
            ef[k] = out.force; et[k] = out.torque; etan[k] = out.tangential; eel[k] = out.normal_stiffness_energy;
            F += ef[k];
            T += et[k] - cross(xq - ec[k], ef[k]);
        }
        if (ne > 1) {
            double osum = 0.0;
            for (int o = 0; o < ne; ++o) osum += eov[ord[o]];
            for (int o = 0; o < ne; ++o) {
                const int e = ord[o];
                F += -ef[e];
                T += -et[e] + cross(xq - ec[e], ef[e]);
                const double wgt = eov[e] / osum;
                ec[e] = xq - (rq - 0.5 * eov[e]) * wgt * en[e];
                ef[e] = ef[e] * wgt;
                et[e] = et[e] * wgt;
                F += ef[e];
                T += et[e] - cross(xq - ec[e], ef[e]);
            }
        }
        double2* sh = reinterpret_cast<double2*>(d.shares + (size_t)q * SHARE);
        sh[0] = make_double2(F.x, F.y);
        sh[1] = make_double2(F.z, T.x);
        sh[2] = make_double2(T.y, T.z);
        // history: each triangle keeps the first contact (in order) now attached
        // to it; at the first step after the initial evaluation a contact of that
        // evaluation that no entry took outlives the step (as near_triangles carries them)
        unsigned int kept_bits = 0u;
        for (int o = 0; o < ne; ++o) {
            const int e = ord[o];
            const unsigned int bit = 1u << ew[e];
            if (kept_bits & bit) continue;
            kept_bits |= bit;
            const size_t hb = whist_at(d.ncap, NCOMP, s, ew[e]);
            store_springs(d.whist[hn], hb, NCOMP, es[e]);
            d.whist[hn][hb + NCOMP] = ek[e];
        }
        d.wact[hn][s] = (d.wact[hn][s] & ~mask) | kept_bits;
        if (MODE == 0) { // kept for the first time step
            double* rec = d.tri_first + (size_t)ci * MAXT * TRI_REC;
            for (int o = 0; o < ne; ++o, rec += TRI_REC) {
                const int e = ord[o];
                rec[0] = (double)ew[e]; rec[1] = ek[e]; rec[2] = eov[e];
                rec[3] = en[e].x; rec[4] = en[e].y; rec[5] = en[e].z;
                rec[6] = ef[e].x; rec[7] = ef[e].y; rec[8] = ef[e].z;
                rec[9] = et[e].x; rec[10] = et[e].y; rec[11] = et[e].z;
                rec[12] = ec[e].x; rec[13] = ec[e].y; rec[14] = ec[e].z;
                rec[15] = (double)esw[e]; rec[16] = eel[e];
                rec[17] = es[e].slide.x; rec[18] = es[e].slide.y; rec[19] = es[e].slide.z;
                rec[20] = es[e].roll.x; rec[21] = es[e].roll.y; rec[22] = es[e].roll.z;
                rec[23] = es[e].tors.x; rec[24] = es[e].tors.y; rec[25] = es[e].tors.z;
            }
            d.tri_first_n[ci] = ne;
        }
        if (record) {
            for (int e = 0; e < ne; ++e) {
                const int wg = I.wall_begin + ew[e];
                ContactGeom g;
                g.n = en[e]; g.overlap = eov[e]; g.c = ec[e]; g.xp = xq; g.xi = zero3();
                ContactOut out;
                out.force = ef[e]; out.torque = et[e]; out.tangential = etan[e];
                out.abs_normal_force = 0.0; out.normal_stiffness_energy = eel[e];
                const dem_species_pair& sp = d.species[I.species_offset + is.y * ns + esw[e]];
                write_record(d, is.x, wg, 1, 0, s, wg, g, out, es[e], spring_energy(sp, es[e], 1.0 / mq));
            }
        }
    }
}

template <int MODE, int BLOCK>
__global__ void __launch_bounds__(BLOCK, SUM_THREADS_PER_SM / BLOCK) k_sum(DevPtrs d)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    Control* ctl = d.ctl;
    const int c = ctl->view.cur, to = c ^ ctl->spare;
    const int* uidx = d.uidx[ctl->view.hcur ^ 1]; // of this evaluation
    const bool final_step = (MODE == 0) ? true : (ctl->view.final_step != 0);
    const double dt = d.dt;
    if ((int)blockIdx.x >= (d.n + BLOCK - 1) / BLOCK) { // the walls, for the next step
        if (!final_step && !ctl->spare) move_walls(d, s - (d.n + BLOCK - 1) / BLOCK * BLOCK);
        return;
    }
    if (s == 0) { // k_units and k_tri are done: the next evaluation starts new lists
        // the springs kept at the pool top in the first time step must not have
        // met this evaluation's items
        if (ctl->n_carry && (unsigned long long)ctl->n_items + ctl->n_carry > (unsigned long long)d.item_cap)
            atomicOr(&ctl->status, 1u << DEM_ERR_CAPACITY);
        ctl->n_carry = 0u;
        ctl->n_items = 0u;
        ctl->n_tri = 0u;
    }
    double disp2 = 0.0;
    if (s < d.n) {
        const double4 ps = d.pr[c][s];
        const double4 vs = d.vm[c][s];
        const double4 ws = d.wi[c][s];
        double4 qs = d.qo[c][s];
        const int4 is = d.info[c][s];
        const InstanceDev& I = d.inst[is.z];
        const int u0 = d.ubase[s], u1 = d.wbase[s]; // its own pairs' units
        const unsigned int walls = d.wcand[s];
        // ---- the shares in list order, the body force, the wall shares ----
        V3 F = zero3(), T = zero3();
        const int count = min(d.cnt[s], d.cap);
        constexpr int E = 8, B = 4; // entries whose units, then items are read together; shares read together
        for (int e0 = 0; e0 < count; e0 += E) {
            int q[E];
#pragma unroll
            for (int j = 0; j < E; ++j) q[j] = (e0 + j < count) ? d.epair[nbr_at(d.ncap, s, e0 + j)] : -1;
            // a pair's units are its lower id's: the particle's own half is P's
            // if the unit lies among its own units
            unsigned int half = 0u;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                if (q[j] < u0 || q[j] >= u1) half |= 1u << j;
                if (q[j] >= 0) q[j] = uidx[q[j]];
            }
#pragma unroll
            for (int k0 = 0; k0 < E; k0 += B) {
                double sh6[B][6];
#pragma unroll
                for (int j = 0; j < B; ++j)
                    if (q[k0 + j] >= 0) {
                        const double2* sh = reinterpret_cast<const double2*>(d.shares + (size_t)q[k0 + j] * SHARE) +
                                            3 * ((half >> (k0 + j)) & 1u);
                        const double2 a = sh[0], b = sh[1], e2 = sh[2];
                        sh6[j][0] = a.x; sh6[j][1] = a.y; sh6[j][2] = b.x;
                        sh6[j][3] = b.y; sh6[j][4] = e2.x; sh6[j][5] = e2.y;
                    }
#pragma unroll
                for (int j = 0; j < B; ++j) // in list order
                    if (q[k0 + j] >= 0) {
                        F += v3(sh6[j][0], sh6[j][1], sh6[j][2]);
                        T += v3(sh6[j][3], sh6[j][4], sh6[j][5]);
                    }
            }
        }
        if (!(is.w & FLAG_FIXED)) { // DPMBase::computeExternalForces (DPMBase.cc:3168-3179)
            const double m = 1.0 / vs.w;
            F += v3(I.gravity[0], I.gravity[1], I.gravity[2]) * m - d.drag * xyz(vs);
            int u = u1;
            for (unsigned int b = d.has_tri ? walls & ~I.tri_mask : walls; b; b &= b - 1, ++u) {
                const int q = uidx[u];
                if (q < 0) continue;
                const double2* sh = reinterpret_cast<const double2*>(d.shares + (size_t)q * SHARE);
                const double2 a = sh[0], b2 = sh[1], e2 = sh[2];
                F += v3(a.x, a.y, b2.x);
                T += v3(b2.y, e2.x, e2.y);
            }
            if (d.has_tri && (walls & I.tri_mask)) { // the net share of all triangle contacts (k_tri)
                const int q = d.slott[s];
                if (q >= 0) {
                    const double2* sh = reinterpret_cast<const double2*>(d.shares + (size_t)q * SHARE);
                    const double2 a = sh[0], b = sh[1], e2 = sh[2];
                    F += v3(a.x, a.y, b.x);
                    T += v3(b.y, e2.x, e2.y);
                }
            }
        }
        if (!(isfinite(F.x) && isfinite(F.y) && isfinite(F.z))) atomicOr(&ctl->status, 1u << DEM_ERR_NAN);

        // ---- integration ----
        double4 pn = ps, vn = vs, wn = ws;
        bool wrapped = false;
        if (final_step) {
            d.force[3 * (size_t)s + 0] = F.x;
            d.force[3 * (size_t)s + 1] = F.y;
            d.force[3 * (size_t)s + 2] = F.z;
            d.torque[3 * (size_t)s + 0] = T.x;
            d.torque[3 * (size_t)s + 1] = T.y;
            d.torque[3 * (size_t)s + 2] = T.z;
        }
        if (MODE == 1) {
            V3 x = xyz(ps), v = xyz(vs), w = xyz(ws);
            Q4 q{qs.x, qs.y, qs.z, qs.w};
            if (vs.w != 0.0) {
                const V3 a = ((F * vs.w) * 0.5) * dt;
                v += a; // BaseParticle::integrateAfterForceComputation
                V3 aw = zero3();
                if (d.rotation) {
                    const S33 Ib{ws.w, 0.0, 0.0, ws.w, 0.0, ws.w};
                    aw = ((rotate_inverse_inertia(q, Ib) * T) * 0.5) * dt;
                    w += aw;
                }
                if (!final_step) { // BaseParticle::integrateBeforeForceComputation of the next step
                    v += a;
                    const V3 disp = v * dt;
                    x += disp;
                    disp2 = len2(disp);
                    if (d.rotation) {
                        w += aw;
                        q = quat_rotate(q, w * dt);
                    }
                }
            } else if (!final_step) { // BaseInteractable::integrateBeforeForceComputation
                const V3 disp = v * dt;
                x += disp;
                disp2 = len2(disp);
                q = quat_rotate(q, w * dt);
            }
            if (!final_step && I.per_mask) { // PeriodicBoundary::checkBoundaryAfterParticlesMove
                double* xc = &x.x;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if ((I.per_mask >> k) & 1u) {
                        const double dl = xc[k] - I.per_lo[k], dr = I.per_hi[k] - xc[k];
                        if ((dl < dr ? dl : dr) < 0) {
                            wrapped = true;
                            if (I.per_hi[k] - xc[k] > xc[k] - I.per_lo[k])
                                xc[k] = xc[k] + I.per_L[k];
                            else
                                xc[k] = xc[k] - I.per_L[k];
                        }
                    }
                }
            }
            pn = make_double4(x.x, x.y, x.z, ps.w);
            vn = make_double4(v.x, v.y, v.z, vs.w);
            wn = make_double4(w.x, w.y, w.z, ws.w);
            qs = make_double4(q.q0, q.q1, q.q2, q.q3);
        }
        if (MODE == 1) { // the initial evaluation leaves the state as it is
            int4 isn = is;
            isn.w = wrapped ? (is.w | FLAG_WRAPPED) : (is.w & ~FLAG_WRAPPED);
            if (!final_step && I.n_del && !(is.w & FLAG_DELETED) && deletion_check(I, xyz(pn))) {
                park_deleted(ctl, pn, vn, wn, isn);
                disp2 = 0.0;
            }
            d.pr[to][s] = pn;
            d.vm[to][s] = vn;
            d.wi[to][s] = wn;
            d.qo[to][s] = qs;
            if (isn.w != is.w) d.info[to][s] = isn;
        }
    }
    if (MODE == 1) { // maximum displacement of this step (for the skin test)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) disp2 = fmax(disp2, __shfl_xor_sync(0xffffffffu, disp2, o));
        if ((threadIdx.x & 31) == 0 && disp2 > 0.0)
            atomicMax(&ctl->step_disp2_bits, (unsigned long long)__double_as_longlong(disp2));
    }
}

} // namespace dem
