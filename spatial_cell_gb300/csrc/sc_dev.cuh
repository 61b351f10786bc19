// sc_dev.cuh -- device-side layout and helpers of the sm_103a step.
//
// State lives in HBM as structure-of-arrays (one float4 / int4 per item per
// field) instead of the reference's 256 / 304-byte structs (types.cuh:173-242),
// so every kernel moves only the fields it touches, 16 bytes at a time:
//
//   particles   pos      float4  x y z | radius
//               vel      float4  x y z | -        (ping-pong inside a step)
//               rot      float4  quaternion        (ping-pong in relax)
//               angvel   float4                    (ping-pong)
//               posnoise float4  x y z | -         (ping-pong in coordinateNoise)
//               angnoise float4                    (ping-pong in coordinateNoise)
//               info     int4    id | type | flags | state(8) hydrophobic(8)
//               dbg      float4  debugVector
//               lscs, spoly, nb  int               lastStateChangeStep,
//                                                  scheduledPolymerization,
//                                                  nActiveInteractions
//               bonds    int[24] interactions[8] {type, group, partnerId}
//   metabolic   pos vel rot angvel posnoise angnoise info dbg as above,
//               met float[SP] per item (S species padded to a multiple of 4),
//               orig int: load slot of the item, indexing the fields no step
//               kernel reads or writes (lscs, spoly, bonds), kept in load order.
//
// Every sort gathers all fields into the other buffer of each pair, so the
// sorted order of every array is the sorted order of the keys, as in the
// reference where CUB moves the whole struct (grid.cuh:91-103).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "scmath.h"
#include "spatialcell.h"

#define SC_THREADS 256
#define SC_ACTIVE SC_PARTICLE_FLAG_ACTIVE

// Pair lists.  Between a sort and applyVelocities no position, flag, type,
// radius or interaction changes, so the pairs that contribute to
// coordinateNoise / relax / relaxMetabolicParticles /
// relaxMetabolicParticlePartners are fixed for all of their sub-iterations
// (16 / 32 / 16 / 16 launches); likewise the diffusion pairs between
// applyVelocities and the next sort (8 launches).  Each list holds, per item
// and in the reference's visiting order, the candidate slots that pass every
// position-only test of the kernel, with the branch the pair takes.  Entries
// are tiled by warps of 32 items: entry k of item i is at
// ((i / 32) * K + k) * 32 + i % 32, so the 32 threads of a warp read one
// 128-byte line per k and all K entries of a warp sit in one K*128-byte block
// (one page, where a k-major layout would put each k of an item in a different
// page).  An item with more pairs than the list holds is marked by a count
// above the capacity and its kernels scan its neighbourhood instead.
#define SC_LIST_PP 128  // particle-particle: rule/chain/test bonds, polar pairs, collisions (dense
                        // lipid membranes list ~100)
#define SC_LIST_M 160   // metabolic: colliding metabolic particles and lipids (beside a dense
                        // membrane ~110)
#define SC_LIST_LM 48   // lipid <- metabolic collisions
#define SC_LIST_D 96    // metabolic diffusion partners
// The diffusion list's buffer holds the count-ordered diffusion list and,
// after it, the diffusion list's build scratch; the whole buffer is also the
// build scratch of the metabolic list (whose pool is sized by demand).
#define SC_LIST_DBUF (SC_LIST_M > 2 * SC_LIST_D ? SC_LIST_M : 2 * SC_LIST_D)
#define SC_PP_POLAR 0x80000000u
#define SC_PP_PARTNER 0x40000000u
#define SC_PP_COLLIDE 0x20000000u
#define SC_PP_INDEX 0x1FFFFFFFu
#define SC_M_FROM_P 0x80000000u
#define SC_M_INDEX 0x7FFFFFFFu

__host__ __device__ __forceinline__ size_t sc_list_at(int K, int i, int k) {
    return ((size_t)(i >> 5) * (size_t)K + (size_t)k) * 32 + (size_t)(i & 31);
}
__host__ __device__ __forceinline__ size_t sc_list_words(int K, int cap) { return (size_t)((cap + 31) / 32) * 32 * K; }

// Device-side error codes (sticky, first one wins).
#define SC_DERR_LOOKBACK_TIMEOUT 1
#define SC_DERR_POLY_OVERFLOW 2

struct ScCounters {
    int nActive;      // nActiveParticles (main.cu:244), bound of every particle kernel
    int lastActive;   // lastActiveParticle (main.cu:245)
    int nextId;       // nextParticleId (main.cu:246)
    int nActiveM;     // nActiveMetabolicParticles (main.cu:253)
    int error;        // first device-side error code
    int polyCount;    // scheduled polymerisations listed this step (k_poly_offsets)
    int polyCreates;  // of those, the ones whose rule creates a monomer
    int polyConflict; // 1: an item holds two bonds of its rule's group (k_poly_plan)
    int step;         // the step loop counter (main.cu:347)
    // what one builder resets lies together, so one memset resets it
    int tileCounter[8];   // k_onesweep, per item set and pass
    int farMove;          // a metabolic item moved more than a cell along an axis since its sort
    int ppClassCount[4];  // items per relax work class (k_build_pp); [3]: RelaxArgs::unsettled
    int ovfPP;            // items whose particle list overflowed (k_build_pp)
    int ovfD;             // items whose diffusion list overflowed (k_build_d)
    int ovfM;             // items whose metabolic list overflowed (k_build_m)
    unsigned long long poolOvfD;  // entries the overflowed diffusion lists asked of their pool (k_build_d_ovf)
    unsigned long long poolM;     // entries the metabolic list blocks asked of their pool (k_build_m)
    unsigned long long poolOvfM;  // the same for the overflowed metabolic items (k_build_m_ovf)
    unsigned long long poolLM;    // the same for the lipid-metabolic lists (k_build_lm)
    int workCount;                // items in the particle work list (k_complexify_select, k_lipid_select)
};

// Relax work classes: 0 bonded items, 1 items with polar (lipid) pairs and no
// bonds, 2 the rest (inactive items with the top bit of their index set).
// Each class has its own blocks, so a warp's items take the same branches.
#define SC_RELAX_CLASSES 3
#define SC_CLASS_INACTIVE 0x80000000u
// Particle list entries per item whose collision geometry is kept (k_build_pp).
#define SC_GEO_PP 8
// Bond match count of a bonded item (low bits) and its in-order flag (a
// test bond: relaxed by the in-order scan).
#define SC_MATCH_COUNT 0xff
#define SC_MATCH_INORDER 0x100

// The geometry of one replica of a batched sim (sc_create_batch): its box,
// its cells, where its cells start in the batch's key space, its noise key.
struct ScRep {
    float simSize, cell;
    int ngrid, bits, nUsed;
    uint32_t keyBase;
    uint64_t seed;
};

struct ScParams {
    float simSize, maxInt, maxDiff, cell;
    int ngrid, bits;
    uint32_t cells;           // cells of the key space (all replicas of a batch)
    uint32_t keyBase;         // first key of this item's replica (0 outside batches)
    int keyBits;              // key bits the sort orders (3 * bits + 1 outside batches)
    int nRep;                 // replicas of a batched sim (1 otherwise)
    const ScRep *reps;        // their geometry (batched sims)
    float moveNoise, rotNoise, metabNoise, velDecay, angDecay;
    int S, SP;
    int N, Nm;
    int coordSteps;
    uint64_t seed;
    const sc_rule *flat;      // id-indexed rules (flattenComplexificationInfo) + one zero rule
    int nFlat;
    const int *pidx;          // partner index [2 * type] -> [start, end)
    int nPidx;
    const sc_rule *prules;    // partner-mapped rules
    const sc_type_info *types;
    int nTypes;
    int listLimit;            // effective pair-list capacity (<= each list's size; smaller only in tests)
    int periodic;             // periodic box extension (sc_config.periodic)
    int walls;                // walled box: 0 clamp (reference), 1 reflect (sc_config.walls)
    int pairClaim;            // complexify by deterministic pair claim (sc_config.pair_claim)
    int metabLean;            // metabolic pair pool of 4-byte entries, geometry evaluated per sub-iteration
                              // (sc_config.metabolic_pairs 0); else 16-byte entries with it frozen (1, default)
    int nUsed;                // cells per axis the box spans, ceil(simSize / cell)
    int binned;               // SC_BINNED_*: sets whose positions are those their cells were sorted by
    int tileCapM, tileCapP;   // tile capacities (slots) of the metabolic sweeps; 0: tiles off
    // Candidate tests that need no record load: after a metabolic sort every
    // binned metabolic item is active (inactive ones sort past the cells)
    // until removeInterferingMetabolicParticles; after a particle sort
    // lipidP[slot] says "active lipid" (types and particle flags do not
    // change between sorts).
    int mAllActive;
    // 1: the metabolic items have moved once since their sort (apply
    // velocities); farMove then says whether one moved more than a cell along
    // an axis
    int movedOnce;
    const int *farMove;
    int lipidValid;
    const uint8_t *lipidP;
    // per set, the last sort's digit counts: SC_SORT_OUTSIDE in the first if it
    // found an active item outside its periodic box (loaded so, or moved by
    // more than a box in one step)
    const uint32_t *histP, *histM;
};
#define SC_SORT_OUTSIDE 0x80000000u
// Whether a position lies in the box [0, L]^3 (no NaN does).
__device__ __forceinline__ bool in_box(sc_f3 p, float L) {
    return p.x >= 0.0f && p.x <= L && p.y >= 0.0f && p.y <= L && p.z >= 0.0f && p.z <= L;
}

// Whether sorted particle j is an active lipid.
__device__ __forceinline__ bool active_lipid(const ScParams &P, const int4 *__restrict__ pinfo, int j) {
    if (P.lipidValid) return P.lipidP[j] != 0;
    const int4 tin = pinfo[j];
    return (tin.z & SC_ACTIVE) && tin.y == SC_PARTICLE_TYPE_LIPID;
}
// Whether sorted metabolic item j is active.
__device__ __forceinline__ bool active_m(const ScParams &P, const int4 *__restrict__ minfo, int j) {
    return P.mAllActive || (minfo[j].z & SC_ACTIVE);
}
#define SC_BINNED_P 1
#define SC_BINNED_M 2

// Cells per axis the cell index clamps to: the power-of-two grid of
// config.cuh:65-74, or in a periodic box the cells the box spans.
__host__ __device__ __forceinline__ int cell_limit(const ScParams &P) { return P.periodic ? P.nUsed : P.ngrid; }

// A neighbour's position as seen from an item at p: itself, or in a periodic
// box its nearest image.  When the neighbours' sets (need, SC_BINNED_*) still
// sit in the cells they were sorted into, neighbours from the 27 cells around
// p are less than 2.5 cells away per axis; if p's cell is not on a face of a
// periodic box at least 5 cells wide, that is less than half the box and
// every neighbour is its own nearest image, so the test is made once per item.
struct Imager {
    bool wrap;
    float L;
    sc_f3 p;
    __device__ __forceinline__ Imager(const ScParams &P, sc_f3 pos, int need) : wrap(false), L(P.simSize), p(pos) {
        if (P.periodic && (P.binned & need) != need) {
            wrap = true;
        } else if (P.periodic) {
            int n = P.nUsed;
            int cx = (int)sc_grid_idx(pos.x, P.cell, n), cy = (int)sc_grid_idx(pos.y, P.cell, n),
                cz = (int)sc_grid_idx(pos.z, P.cell, n);
            wrap = !(P.simSize >= 5.0f * P.cell) || cx == 0 || cy == 0 || cz == 0 || cx == n - 1 || cy == n - 1 ||
                   cz == n - 1;
        }
    }
    __device__ __forceinline__ sc_f3 operator()(sc_f3 t) const { return wrap ? sc_image3(t, p, L) : t; }
};

__device__ __forceinline__ sc_f4 ld4(const float4 *p, int i) {
    float4 v = p[i];
    return sc_make_f4(v.x, v.y, v.z, v.w);
}
__device__ __forceinline__ sc_f3 ld3(const float4 *p, int i) {
    float4 v = p[i];
    return sc_make_f3(v.x, v.y, v.z);
}
__device__ __forceinline__ void st4(float4 *p, int i, sc_f4 v) { p[i] = make_float4(v.x, v.y, v.z, v.w); }

// A 32-byte row (two float4, 32-byte aligned) in one 256-bit access
// (ld/st .v8 on the global space, sm_100 and later): a warp's scattered rows
// then cost one L1 wavefront per row instead of two.  The load is for
// buffers no thread writes during the kernel.
__device__ __forceinline__ void ld_row8(const float4 *p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}
__device__ __forceinline__ void st_row8(float4 *p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ void st3(float4 *p, int i, sc_f3 v, float w) { p[i] = make_float4(v.x, v.y, v.z, w); }

__device__ __forceinline__ int info_state(int w) { return (int)(int8_t)(w & 0xff); }
__device__ __forceinline__ int info_hydro(int w) { return (int)(int8_t)((w >> 8) & 0xff); }
__device__ __forceinline__ int info_pack(int state, int hydro) { return (state & 0xff) | ((hydro & 0xff) << 8); }

// flat[] holds nFlat id-indexed rules plus one zero rule at [nFlat]: ids
// without a rule read as all-zero, as the reference's memset table does.
__device__ __forceinline__ const sc_rule &rule_at(const ScParams &P, int id) {
    return P.flat[(id >= 0 && id < P.nFlat) ? id : P.nFlat];
}
__device__ __forceinline__ sc_f4 rule_ori(const sc_rule &r) {
    return sc_make_f4(r.relative_orientation[0], r.relative_orientation[1], r.relative_orientation[2],
                      r.relative_orientation[3]);
}
__device__ __forceinline__ sc_f3 rule_pos(const sc_rule &r) {
    return sc_make_f3(r.relative_position[0], r.relative_position[1], r.relative_position[2]);
}

__device__ __forceinline__ bool outside_cube(sc_f3 d, float lim) {
    return fabsf(d.x) > lim || fabsf(d.y) > lim || fabsf(d.z) > lim;
}

__device__ __forceinline__ uint32_t cell_key(const ScParams &P, uint32_t gx, uint32_t gy, uint32_t gz) {
    return P.keyBase + ((gx << (2 * P.bits)) | (gy << P.bits) | gz);
}

// Batched sims: every item carries its replica in the bits of its info
// record's w word above the hydrophobicity byte.  A kernel of a batch works
// on one item at a time with that replica's geometry (its neighbours are in
// the same replica's cells); outside batches P is used as given.
__device__ __forceinline__ int item_rep(int infoW) { return (int)((unsigned)infoW >> 8); }
template <bool BATCH>
__device__ __forceinline__ void rep_apply(ScParams &P, int infoW) {
    if (!BATCH) return;
    const int r = min(item_rep(infoW), P.nRep - 1);
    const ScRep g = P.reps[r];
    P.simSize = g.simSize;
    P.cell = g.cell;
    P.ngrid = g.ngrid;
    P.bits = g.bits;
    P.nUsed = g.nUsed;
    P.keyBase = g.keyBase;
    P.seed = g.seed;
}

// Visits the reference's 27-cell neighbourhood of pos (grid.cuh:13-25 and the
// loop of e.g. dynamics.cuh:445-451): cells clamped at the box edge, in gx, gy,
// gz order, slots ascending inside a cell.  Keys of the cells (gx, gy, z0..z1)
// are consecutive, so with the exclusive cell-start table (cellStart[c] =
// first sorted slot with key >= c) that run of cells is one slot range, and
// the visiting order is exactly the reference's.
// Offsets (-1..1 per axis) of the neighbour cells a scan visits.  All 27 by
// default; reach() drops a neighbour layer when no item in it can pass the
// interaction cube |delta| <= lim on that axis, which every caller tests
// before anything else, so the visits that remain are the reference's, in its
// order, and the results are unchanged.  The bound needs the neighbours to
// sit in the cells they were sorted into (P.binned covers `need`), lim at
// most the cell size, and a periodic box of at least 5 cells (no nearest image
// crosses back into the cube).  Candidates of cell c - 1 lie below c * cell
// and those of cell c + 1 at or above (c + 1) * cell (or at the box size
// past the top periodic cell), up to the rounding of the cell index; the
// margin covers that and the rounding of delta.
struct Reach {
    int xl = -1, xh = 1, yl = -1, yh = 1, zl = -1, zh = 1;
};
__device__ __forceinline__ void reach_axis(const ScParams &P, float p, int c, int n, float lim, int &lo, int &hi) {
    const float m = lim + 1e-3f + 4e-6f * (fabsf(p) + P.cell * (float)(c + 1));
    lo = (p - (float)c * P.cell > m) ? 0 : -1;
    const float upper = (P.periodic && c == n - 1) ? P.simSize : (float)(c + 1) * P.cell;
    hi = (upper - p > m) ? 0 : 1;
}
__device__ __forceinline__ Reach reach(const ScParams &P, sc_f3 pos, float lim, int need) {
    Reach r;
    if ((P.binned & need) != need || !(lim <= P.cell) || (P.periodic && !(P.simSize >= 5.0f * P.cell))) return r;
    const int n = cell_limit(P);
    reach_axis(P, pos.x, (int)sc_grid_idx(pos.x, P.cell, n), n, lim, r.xl, r.xh);
    reach_axis(P, pos.y, (int)sc_grid_idx(pos.y, P.cell, n), n, lim, r.yl, r.yh);
    reach_axis(P, pos.z, (int)sc_grid_idx(pos.z, P.cell, n), n, lim, r.zl, r.zh);
    return r;
}

// A neighbour cell index c + o (c in [0, n), o in -1..1) taken around the
// periodic box: ((c + o + n) mod n) without the integer division.
__device__ __forceinline__ uint32_t wrap_cell(int v, int n) {
    return (uint32_t)(v < 0 ? v + n : (v >= n ? v - n : v));
}

template <class F>
__device__ __forceinline__ void scan27(const ScParams &P, const uint32_t *__restrict__ cellStart, sc_f3 pos,
                                       const Reach &R, F &&f) {
    int n = cell_limit(P);
    int cx = (int)sc_grid_idx(pos.x, P.cell, n), cy = (int)sc_grid_idx(pos.y, P.cell, n),
        cz = (int)sc_grid_idx(pos.z, P.cell, n);
    if (P.periodic) {
        // the z run of a column is one slot range unless it wraps
        for (int ox = R.xl; ox <= R.xh; ox++) {
            for (int oy = R.yl; oy <= R.yh; oy++) {
                uint32_t base = cell_key(P, wrap_cell(cx + ox, n), wrap_cell(cy + oy, n), 0);
                if (cz + R.zl >= 0 && cz + R.zh <= n - 1) {
                    for (uint32_t j = cellStart[base + (uint32_t)(cz + R.zl)],
                                  e = cellStart[(base + (uint32_t)(cz + R.zh)) + 1];
                         j < e; j++)
                        f((int)j);
                } else {
                    for (int oz = R.zl; oz <= R.zh; oz++) {
                        uint32_t key = base + wrap_cell(cz + oz, n);
                        for (uint32_t j = cellStart[key], e = cellStart[key + 1]; j < e; j++) f((int)j);
                    }
                }
            }
        }
        return;
    }
    int x0 = max(cx + R.xl, 0), x1 = min(cx + R.xh, n - 1);
    int y0 = max(cy + R.yl, 0), y1 = min(cy + R.yh, n - 1);
    uint32_t z0 = (uint32_t)max(cz + R.zl, 0), z1 = (uint32_t)min(cz + R.zh, n - 1);
    for (int gx = x0; gx <= x1; gx++) {
        for (int gy = y0; gy <= y1; gy++) {
            uint32_t base = cell_key(P, (uint32_t)gx, (uint32_t)gy, 0);
            uint32_t s = cellStart[base + z0], e = cellStart[(base + z1) + 1];
            for (uint32_t j = s; j < e; j++) f((int)j);
        }
    }
}
template <class F>
__device__ __forceinline__ void scan27(const ScParams &P, const uint32_t *__restrict__ cellStart, sc_f3 pos, F &&f) {
    scan27(P, cellStart, pos, Reach(), f);
}

// Same neighbourhood, one cell at a time (for kernels that interleave two
// arrays cell by cell, metabolites.cuh:174-248).
template <class F>
__device__ __forceinline__ void cells27(const ScParams &P, sc_f3 pos, const Reach &R, F &&f) {
    int n = cell_limit(P);
    int cx = (int)sc_grid_idx(pos.x, P.cell, n), cy = (int)sc_grid_idx(pos.y, P.cell, n),
        cz = (int)sc_grid_idx(pos.z, P.cell, n);
    if (P.periodic) {
        for (int ox = R.xl; ox <= R.xh; ox++)
            for (int oy = R.yl; oy <= R.yh; oy++)
                for (int oz = R.zl; oz <= R.zh; oz++)
                    f(cell_key(P, wrap_cell(cx + ox, n), wrap_cell(cy + oy, n),
                               wrap_cell(cz + oz, n)));
        return;
    }
    for (int gx = max(cx + R.xl, 0); gx <= min(cx + R.xh, n - 1); gx++)
        for (int gy = max(cy + R.yl, 0); gy <= min(cy + R.yh, n - 1); gy++)
            for (int gz = max(cz + R.zl, 0); gz <= min(cz + R.zh, n - 1); gz++)
                f(cell_key(P, (uint32_t)gx, (uint32_t)gy, (uint32_t)gz));
}
template <class F>
__device__ __forceinline__ void cells27(const ScParams &P, sc_f3 pos, F &&f) {
    cells27(P, pos, Reach(), f);
}

// Whether an item's candidates of sets `need` may lie on either side of a
// periodic face whatever cell they are listed in (scan_words): the sets have
// moved since their sort, the box is under five cells, or a position lies
// outside the box, in the cell on the face that its index is clamped to and up
// to a box length from it.  An item that takes no images (Imager::wrap) has
// none to look for.
__device__ __forceinline__ bool scan_mixed(const ScParams &P, const Imager &IM, int need) {
    if (!IM.wrap) return false;
    if ((P.binned & need) != need || !(P.simSize >= 5.0f * P.cell) || !in_box(IM.p, P.simSize)) return true;
    return (((need & SC_BINNED_P) ? *P.histP : 0u) | ((need & SC_BINNED_M) ? *P.histM : 0u)) & SC_SORT_OUTSIDE;
}
// The same neighbourhood for the list builds, in two passes a thread takes
// word by word.  A builder's thread spends its time on candidates that leave
// at the cube test (three of four): visited one by one with the survivors
// handled in place, a third of a warp's lanes were busy.  Here the first pass
// tests up to 32 consecutive candidates without a branch and keeps the
// survivors as a bit mask; the second walks the masks' bits, so the costly
// part runs with a lane per survivor.  Candidates are visited in the
// reference's order: cells of a column's z run are consecutive in `cand`, a
// word's bits ascend, and when an item's words fill its slots they are walked
// before the scan goes on.
//
// cand holds positions in cell order, start(key) the first candidate of cell
// key (start(key + 1) the end of its run); up to seven records past a run's
// end are read and masked off, so cand has SC_CAND_PAD records more than
// candidates.  The first pass keeps a superset of what the cube |delta| <= lim
// holds.  In the box's interior that is the cube itself.  A run across a
// periodic face is tested against the item shifted by the box, with a margin:
// a coordinate difference and its image differ from the box length by the
// rounding of coordinates no larger than |pp| + 2 L + lim.  With `mixed`
// (scan_mixed) every candidate within that margin directly or across a face is
// kept.  f(k, cand[k]) makes the exact
// tests; without an image (Imager::wrap) the cube holds already.
//
// What bounds it is the latency of the candidates' loads at 32 warps per SM,
// so SC_SCAN_GROUP of them are in flight at a time and a survivor's record is
// loaded while the one before is handled.  524,288 + 2,097,152 items (a
// quarter of the large workload), per step: k_build_m 1136 -> 604 us (groups
// of four: 685; with the emission's four pairs in flight, which took 440 us
// one by one), k_build_d 598 -> 508 us, k_build_lm 211 -> 150 us; the columns
// advanced per lane instead of in step for the warp: 741 / 546 us.
#define SC_SCAN_GROUP 8
#define SC_CAND_PAD SC_SCAN_GROUP
#define SC_SCAN_WORDS 10
struct ScanWords {
    uint32_t base[SC_SCAN_WORDS][SC_THREADS], mask[SC_SCAN_WORDS][SC_THREADS];
};
template <class Start, class F>
__device__ __forceinline__ void scan_words(const ScParams &P, ScanWords &W, const float4 *__restrict__ cand,
                                           Start &&start, sc_f3 pp, const Reach &R, float lim, bool mixed, F &&f) {
    const int n = cell_limit(P), tid = threadIdx.x;
    const int cx = (int)sc_grid_idx(pp.x, P.cell, n), cy = (int)sc_grid_idx(pp.y, P.cell, n),
              cz = (int)sc_grid_idx(pp.z, P.cell, n);
    const float L = P.simSize;
    const float wide = lim + 1e-3f + 4e-6f * (L + fmaxf(fabsf(pp.x), fmaxf(fabsf(pp.y), fabsf(pp.z))));
    // a periodic column's z run that crosses the face is taken in two parts:
    // first the cells up to `cut`, then the rest
    const int za = cz + R.zl, zb = cz + R.zh;
    const bool split = P.periodic && (za < 0 || zb > n - 1);
    const int cut = za < 0 ? -1 : n - 1;
    int from = 0;             // where the scan goes on: the run, and its next candidate
    uint32_t fromB = 0;
    bool more;
    do {
        more = false;
        int nw = 0;
        // the columns in step for the whole warp (a lane without one idles), each in its two parts
        for (int r = 0; r < 18; r++) {
            const int ox = r / 6 - 1, oy = (r >> 1) % 3 - 1;
            if (more || r < from || ((r & 1) && !split) || ox < R.xl || ox > R.xh || oy < R.yl || oy > R.yh) continue;
            int gx = cx + ox, gy = cy + oy, z0 = za, z1 = zb;
            sc_f3 q = pp;       // the item as this run's candidates see it
            float far = lim;    // the first pass's cube
            if (P.periodic) {
                if (split) {
                    if (r & 1) z0 = cut + 1;
                    else z1 = cut;
                }
                if (gx < 0 || gx >= n || gy < 0 || gy >= n || z0 < 0 || z0 >= n) {
                    q.x = gx < 0 ? pp.x + L : (gx >= n ? pp.x - L : pp.x);
                    q.y = gy < 0 ? pp.y + L : (gy >= n ? pp.y - L : pp.y);
                    q.z = z0 < 0 ? pp.z + L : (z0 >= n ? pp.z - L : pp.z);
                    far = wide;
                    const int len = z1 - z0;
                    gx = (int)wrap_cell(gx, n);
                    gy = (int)wrap_cell(gy, n);
                    z0 = (int)wrap_cell(z0, n);
                    z1 = z0 + len;
                }
            } else {
                if (gx < 0 || gx >= n || gy < 0 || gy >= n) continue;
                z0 = max(z0, 0);
                z1 = min(z1, n - 1);
            }
            const uint32_t key = cell_key(P, (uint32_t)gx, (uint32_t)gy, 0);
            uint32_t b = start(key + (uint32_t)z0);
            const uint32_t e = start(key + (uint32_t)z1 + 1u);
            if (r == from && fromB) b = fromB;
            for (; b < e; b += 32u) {
                if (nw == SC_SCAN_WORDS) {
                    more = true;
                    from = r;
                    fromB = b;
                    break;
                }
                const uint32_t m = min(32u, e - b);
                const float4 *__restrict__ t = cand + b;
                uint32_t mask = 0;
                if (!mixed) {
                    for (uint32_t u = 0; u < m; u += SC_SCAN_GROUP) {
                        float4 c[SC_SCAN_GROUP];
#pragma unroll
                        for (int v = 0; v < SC_SCAN_GROUP; v++) c[v] = t[u + v];
                        uint32_t bits = 0;
#pragma unroll
                        for (int v = 0; v < SC_SCAN_GROUP; v++)
                            if (!(fmaxf(fabsf(c[v].x - q.x), fmaxf(fabsf(c[v].y - q.y), fabsf(c[v].z - q.z))) > far))
                                bits |= 1u << v;
                        mask |= bits << u;
                    }
                } else {
                    for (uint32_t u = 0; u < m; u++) {
                        const float4 c = t[u];
                        const float dx = fabsf(c.x - pp.x), dy = fabsf(c.y - pp.y), dz = fabsf(c.z - pp.z);
                        const float d = fmaxf(fminf(dx, fabsf(dx - L)),
                                              fmaxf(fminf(dy, fabsf(dy - L)), fminf(dz, fabsf(dz - L))));
                        if (!(d > wide)) mask |= 1u << u;
                    }
                }
                if (m < 32u) mask &= (1u << m) - 1u;
                if (mask) {
                    W.base[nw][tid] = b - 1u;
                    W.mask[nw][tid] = mask;
                    nw++;
                }
            }
        }
        // the survivors so far, the next one's record on its way
        uint32_t k = 0, base = 0, mask = 0;
        int w = 0;
        auto step = [&]() {
            if (!mask) {
                if (w == nw) return false;
                base = W.base[w][tid];
                mask = W.mask[w][tid];
                w++;
            }
            k = base + (uint32_t)__ffs((int)mask);
            mask &= mask - 1u;
            return true;
        };
        bool any = step();
        float4 c = cand[k];
        while (any) {
            const uint32_t kc = k;
            const float4 cc = c;
            any = step();
            c = cand[k];
            f((int)kc, cc);
        }
    } while (more);
}

__device__ __forceinline__ void set_error(ScCounters *c, int code) { atomicCAS(&c->error, 0, code); }
