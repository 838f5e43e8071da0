// dem_engine.cuh -- device data layout shared by the DEM kernels.
//
// Layout in HBM (all arrays indexed by the engine's sorted particle order,
// which is (instance, level, cell, id) after every neighbour-list rebuild):
//   pr[b][i]   double4 (x, y, z, radius)         b = state buffer 0/1
//   vm[b][i]   double4 (vx, vy, vz, invMass)
//   wi[b][i]   double4 (wx, wy, wz, invInertia)
//   qo[b][i]   double4 orientation quaternion (q0..q3)
//   info[b][i] int4    (id, species, instance, flags)
//   caller[b][i] int   index of the particle in the caller's upload order
// The 32-byte records let a neighbour's position+radius, velocity+mass and
// angular velocity+inertia each arrive in one 32-byte sector. A time step
// updates the state in place (k_sum touches only its own particle's records);
// the other buffer takes the permutation of a rebuild.
//
// Neighbour lists are fixed-capacity rows, one per particle: rows[i*cap + k]
// (k < cnt[i]). From them every rebuild makes a flat list of units, the work
// items of the force evaluation: unit[l][j] = (P, I) is a pair of sorted
// particle slots with the lower id first, (s, ~w) a particle and a wall w of
// its instance within reach, (s, UNIT_TRI) a particle near triangle walls. A
// particle's units are contiguous (from ubase[i]: its pairs in list order,
// then its walls in wall order), and epair[k*ncap + i] is the unit of its list
// entry k. Contact history is stored per contact: the springs of an
// evaluation's contacts sit in a pool indexed by the contact's item number in
// that evaluation, pool[p][q*stride + c] (3 or 9 components per spring,
// padded), and every unit keeps the item of its contact of the last
// evaluation, uidx[h][j] (uidx_kept below). Items also index the force shares
// that k_units leaves for k_sum. pool and uidx flip with every evaluation
// (p = Control::pcur, h = Control::hcur: read, write the other); a rebuild
// carries uidx to the new units (flipping h) and leaves the pool in place.
#pragma once
#include <cstdint>
#include "dem_math.cuh"
#include "dem_walls.cuh"
#include "../../include/dem_b200.h"

namespace dem {

constexpr int FLAG_FIXED = 1;
// deleted by a DeletionBoundary: also FLAG_FIXED, parked at DELETED_COORD,
// sorted into the graveyard cell (the last cell) at the next rebuild
constexpr int FLAG_DELETED = 2;
// a free row of an insertion boundary: parked like a deleted particle (also
// FLAG_DELETED and FLAG_FIXED) until a placement fills it
constexpr int FLAG_DORMANT = 4;
// the last drift moved the particle across a periodic boundary (set and
// cleared by every drift): the reference's HGrid still files it under its
// cell before the shift until the grid is next updated, which the insertion
// check reproduces
constexpr int FLAG_WRAPPED = 8;
constexpr double DELETED_COORD = 1e300;
constexpr int LEVEL_SHIFT = 8;

// I field of a unit for a particle near triangle walls (walls: ~w, w < 32)
constexpr int UNIT_TRI = INT32_MIN;
// uidx of a unit: >= 0 the item of its contact; UIDX_NONE no contact and no
// history; below that a spring kept without a contact (the first time step,
// k_units), at pool index uidx_kept(v).
constexpr int UIDX_NONE = -1;
__host__ __device__ __forceinline__ int uidx_kept(int v) { return -2 - v; }
// pool index of a unit's spring, -1 if it has none
__host__ __device__ __forceinline__ int uidx_spring(int v) { return v >= 0 ? v : (v == UIDX_NONE ? -1 : uidx_kept(v)); }

struct InstanceDev {
    double origin[3];
    double gravity[3];
    double per_lo[3];
    double per_hi[3];
    double per_L[3];
    double per_half[3];
    uint32_t per_mask;
    int species_offset;
    int n_species;
    int wall_begin;
    int wall_end;
    int n_levels;
    int cell_base[DEM_MAX_LEVELS];
    int dims[DEM_MAX_LEVELS][3];
    double inv_cell[DEM_MAX_LEVELS][3];
    double level_rmax[DEM_MAX_LEVELS];
    // the banding that assigned the levels (radius r: binary exponent of
    // r / level_rmin, clamped to level_bands - 1, through level_remap), for
    // particles placed by insertion boundaries
    double level_rmin;
    int level_bands;
    int level_remap[DEM_MAX_LEVELS];
    double max_interaction_distance;
    // DeletionBoundary planes: a particle is deleted when del_d - x . del_n < 0
    int n_del;
    uint32_t tri_mask;     // walls (bit w = wall_begin + w) that are triangle walls
    // walls (same bits) taken out during the run (WallHandler::removeObject):
    // no contacts with them from the next time step on
    uint32_t wall_off_mask;
    int tri_static;        // every triangle wall of the instance stands still
    double del_n[DEM_MAX_DELETION_PER_INSTANCE][3];
    double del_d[DEM_MAX_DELETION_PER_INSTANCE];
};

// Contact record written at the last force evaluation of a dem_step call:
// one row per contact (particle pairs once, from P's side; wall contacts).
struct ContactRecord {
    int id_p, id_i;
    int is_wall, periodic;
    int slot_p, slot_i;         // sorted indices (slot_i = wall index for walls)
    double overlap;
    double elastic_energy;
    double force[3];
    double contact_point[3];
    double branch[3];           // x_P - x_I (image position for periodic pairs); wall: 0
    double normal[3];           // unit normal of the contact (from I towards P)
    double tangential[3];       // the friction force (part of force)
    double springs[9];
};

// What the kernels of one force evaluation read: written by one thread of
// k_rebuild (or the host) before it, when all of that launch's blocks decide
// from the fields below, which k_units then advances.
struct StepView {
    int cur, lbuf, hcur, pcur; // state, unit-list, uidx and pool buffers to read
    int final_step;            // this step is the last of the dem_step call
    int first_step;            // this step is the first after the initial evaluation
};

struct Control {
    StepView view;
    double next_disp_acc;  // disp_acc and list_age once this step is under way
    int next_list_age;
    int pad0;
    int cur;               // state buffer holding the current state
    int lbuf;              // unit-list buffer in use
    int pending_flip;      // the last force evaluation wrote the other spring pool and uidx
    int force_rebuild;     // rebuild before the next evaluation regardless of displacement
    int record;            // record contacts at final/initial evaluations
    int spare;             // 1: k_sum writes the other state buffer (timing launches; the state stays)
    long long steps_left;
    long long n_rebuilds;
    long long steps_done;  // time steps since the upload
    int hcur;              // uidx (and triangle history) buffer of the last evaluation
    double disp_acc;       // sum of per-step maximum displacements since the last rebuild
    int list_age;          // time steps (moves of the walls) since the last rebuild
    int pad1;
    double skin;
    unsigned long long step_disp2_bits; // max |dx|^2 this step (bits of a non-negative double)
    unsigned int status;   // OR of (1u << DEM_ERR_*)
    unsigned int n_records;
    unsigned int record_capacity;
    unsigned int lost_history;
    unsigned int n_items;  // contact items of the current evaluation
    unsigned int n_tri;    // triangle-wall items of the current evaluation (tri_list)
    int pcur;              // spring pool holding the springs of the last evaluation
    unsigned int n_carry;  // first time step: springs kept without a contact (pool top)
    int n_units;           // units of the list in use
    int n_units_next;      // units of the list a rebuild is making
};

// Entry-major layouts: entry k of every particle is contiguous, so threads
// of consecutive particles touch consecutive words; the spring components of
// one entry are contiguous (one sector for a contact's history).
__host__ __device__ __forceinline__ size_t nbr_at(int ncap, int i, int k) { return (size_t)k * ncap + i; }
// A spring record holds ncomp doubles padded to an even count (3 -> 4,
// 9 -> 10), so every record starts on 16 bytes and moves as 16-byte vectors.
__host__ __device__ __forceinline__ int hist_stride(int ncomp) { return ncomp + (ncomp & 1); }
__host__ __device__ __forceinline__ size_t pool_at(int ncomp, int j) { return (size_t)j * hist_stride(ncomp); }
__host__ __device__ __forceinline__ size_t whist_at(int ncap, int ncomp, int i, int w)
{
    return ((size_t)w * ncap + i) * hist_stride(ncomp);
}

struct DevPtrs {
    // particle state, two buffers
    double4 *pr[2], *vm[2], *wi[2], *qo[2];
    int4 *info[2];
    int *caller[2];
    // forces of the last force evaluation (3 per particle, sorted order)
    double *force, *torque;
    // neighbour lists of the last rebuild, particle-major
    int *rows;
    int *cnt;
    // ownership bits: bit k%32 of word own[(k/32)*ncap + i] is set when
    // particle i has the lower id of its entry k's pair
    unsigned int *own;
    // walls (bit w = wall_begin + w) particle i has units for: those it can
    // touch before the next rebuild (build_one), and the triangle walls its one
    // triangle unit tests
    unsigned int *wcand;
    int2 *unit[2];
    int *uidx[2];
    int *ubase, *wbase;      // first unit / first wall unit of a particle
    int *epair;              // per entry: its pair's unit
    double *pool[2];         // springs per contact (item_cap records each)
    double *whist[2];        // triangle walls: springs and creation key per (particle, wall)
    unsigned int *wact[2];   // triangle walls: which of them hold a contact's history
    // broad phase scratch
    int *key, *perm, *newidx, *cell_count, *cell_start, *block_sums;
    unsigned long long *rb_barrier; // arrivals at the rebuild's grid barriers (only grows)
    float4 *pf;              // (x, y, z, r) in FP32 of the gathered state: the list build's prefilter
    int *row_slot;           // caller row -> slot of the current order (insertion boundaries only, else null)
    // tables
    const InstanceDev *inst;
    const dem_species_pair *species;
    dem_wall *walls;         // moved before every step's force evaluation (move_wall)
    WallGeom *wgeom;   // per wall; faces, edges and corners of intersection walls
    int n_walls;
    int n_instances;
    // triangle-wall items of one evaluation: (particle, item, wall bits, 0)
    int4 *tri_list;
    int *slott;              // per particle: its triangle-wall item or -1
    double *tri_first;       // triangle contacts of the initial evaluation, TRI_REC doubles each,
                             // DEM_MAX_TRIANGLE_CONTACTS per particle in caller order (k_tri)
    int *tri_first_n;        // their number per particle (caller order)
    double *shares;          // 12 doubles per item: P force, P torque, I force, I torque
    int item_cap;
    int unit_cap;
    Control *ctl;
    ContactRecord *records;
    // sizes
    int n;            // particles
    int ncap;         // allocated particle slots (ELL stride)
    int cap;          // neighbour capacity per particle (multiple of 32)
    int nwords;       // cap / 32
    int any_periodic; // some instance has a periodic direction
    int ncomp;        // history components per contact (3 or 9)
    int wmax;         // max walls per instance
    int ncells;
    int rotation;
    int single_instance;   // one instance: k_units stages its record in shared memory
    int n_species_table;   // entries of the species table
    int zero_idist;        // every species pair has interaction distance 0
    int has_tri;           // some wall is a triangle wall (k_tri runs)
    double dt;
    double drag;
    // time steps a list holds for the walls other than triangles that move (but
    // about their own axis); INT_MAX if none does
    int wall_steps;
};

} // namespace dem
