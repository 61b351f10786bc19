// sc_step.cu -- the step's kernels on sm_103a, one per reference kernel.
//
// Each kernel computes, for every item it owns, exactly the floating-point
// expression sequence of the reference kernel named in its comment (same
// operand order, same implicit double-precision literals, no fused
// multiply-add: the file is built with -fmad=false), so its results are
// bit-identical to the reference's on the same input state.  What changes is
// where the data lives: structure-of-arrays fields read 16 bytes at a time,
// double buffering only for the fields a kernel's neighbours read, elementwise
// kernels updating in place, and no memset of a whole 256-byte-per-item
// buffer before each kernel (main.cu:326-638 does 92 of them per step).
//
// Launch shape: one thread per slot, 256 threads per CTA; the bound of every
// kernel is the device-side active counter, so no host round trip is needed
// between kernels (the reference reads nActiveParticles back three times per
// step, main.cu:369,399,616).
#include "sc_launch.h"
#include "sc_tile.cuh"

__device__ __forceinline__ bool p_order(int ta, int ia, int tb, int ib) { return ta < tb || (ta == tb && ia < ib); }

// ---- dynamics.cuh:19-215: move (its only live effect: debugVector.xyz = 0)
// fused with brownianMovementAndRotation, in place --------------------------------
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_move_brownian(const int *__restrict__ nActivePtr,
                                                              const int4 *__restrict__ info,
                                                              const float4 *__restrict__ pos, float4 *dbg,
                                                              float4 *posnoise, float4 *angnoise, ScParams P,
                                                              float scale, uint32_t su, uint32_t sn,
                                                              const int *__restrict__ stepPtr) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    const int step = *stepPtr;
    int4 in = info[i];
    if (!(in.z & SC_ACTIVE)) return;
    rep_apply<BATCH>(P, in.w);
    float4 d = dbg[i];
    d.x = 0.0f; d.y = 0.0f; d.z = 0.0f;
    dbg[i] = d;
    float radius = pos[i].w;
    uint32_t id = (uint32_t)in.x, st = (uint32_t)step;
    uint64_t seed = P.seed;
    sc_f4 r1 = sc_random_rotation(sc_uniform(seed, su, id, st, 0), sc_uniform(seed, su, id, st, 1),
                                  sc_uniform(seed, su, id, st, 2));
    float nrm = sc_normal(seed, sn, id, st, 0);
    float mag = sc_noise_mag(fabsf(nrm) * scale, radius);
    st3(posnoise, i, sc_rotate(sc_up(), r1) * mag, 0.0f);
    sc_f4 r2 = sc_random_rotation(sc_uniform(seed, su, id, st, 3), sc_uniform(seed, su, id, st, 4),
                                  sc_uniform(seed, su, id, st, 5));
    float t = sc_rot_noise(P.rotNoise, radius);
    st4(angnoise, i, sc_slerp(ld4(angnoise, i), r2, t));
}

// ---- dynamics.cuh:217-242 applyNoise, in place -------------------------------
__global__ void __launch_bounds__(SC_THREADS) k_apply_noise(const int *__restrict__ nActivePtr,
                                                            const int4 *__restrict__ info, float4 *vel,
                                                            float4 *posnoise, float4 *angvel, float4 *angnoise) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    if (!(info[i].z & SC_ACTIVE)) return;
    sc_f3 v = ld3(vel, i);
    v += ld3(posnoise, i);
    st3(vel, i, v, 0.0f);
    st3(posnoise, i, sc_zero3(), 0.0f);
    st4(angvel, i, sc_qmul(ld4(angnoise, i), ld4(angvel, i)));
    st4(angnoise, i, sc_qid());
}

// ---- dynamics.cuh:244-282 applyVelocities, in place ---------------------------
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_apply_velocities(const int *__restrict__ nActivePtr,
                                                                 const int4 *__restrict__ info, float4 *pos,
                                                                 float4 *vel, float4 *rot, float4 *angvel,
                                                                 ScParams P, float f, int *farMove) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    const int4 in = info[i];
    if (!(in.z & SC_ACTIVE)) return;
    rep_apply<BATCH>(P, in.w);
    float4 p4 = pos[i];
    sc_f3 p = sc_make_f3(p4.x, p4.y, p4.z);
    sc_f3 v = ld3(vel, i);
    if (farMove && !(fmaxf(fabsf(v.x), fmaxf(fabsf(v.y), fabsf(v.z))) * f < 0.999f * P.cell)) *farMove = 1;
    p = P.periodic ? sc_wrap3(p + v * f, P.simSize)
                   : (P.walls ? sc_reflect3(p + v * f, P.simSize) : clamp(p + v * f, 0.0f, P.simSize));
    v *= P.velDecay;
    sc_f4 av = ld4(angvel, i);
    sc_f4 r = sc_qmul(sc_slerp(sc_qid(), av, f), ld4(rot, i));
    r /= length(r);
    av = sc_slerp(av, sc_qid(), 1.0f - P.angDecay);
    pos[i] = make_float4(p.x, p.y, p.z, p4.w);
    st3(vel, i, v, 0.0f);
    st4(rot, i, r);
    st4(angvel, i, av);
}

// ---- pair lists ------------------------------------------------------------------
// The list of item i is read as entries list[k * cap + i], k < cnt[i]; cnt[i]
// above the list's capacity means "scan instead".
template <int K>
struct PairList {
    const uint32_t *__restrict__ list;
    const int *__restrict__ cnt;
    int cap;
    const int *__restrict__ perm;  // position -> item (count-ordered lists; null: identity)
};

// Packed 32-bit list entries: 4 consecutive entries of an item share one
// 16-byte chunk, chunks warp-tiled (chunk q of position g at
// ((g/32) * K/4 + q) * 32 + g%32), so one load brings 4 entries.
__host__ __device__ __forceinline__ size_t sc_list4_at(int K, int g, int k) {
    return (((size_t)(g >> 5) * (size_t)(K / 4) + (size_t)(k >> 2)) * 32 + (size_t)(g & 31)) * 4 + (size_t)(k & 3);
}
__device__ __forceinline__ const uint4 *sc_list4_chunks(const uint32_t *list, int K, int g) {
    return reinterpret_cast<const uint4 *>(list) + (size_t)(g >> 5) * (size_t)(K / 4) * 32 + (size_t)(g & 31);
}

// Count-ordered list layout.  A builder block first writes each item's list
// at the item's own position of `scratch`; this re-orders the block's items
// by descending list length and copies the lists to their new positions, so
// a consumer warp walks lists of similar lengths; the lists are written
// packed (sc_list4_at).  perm[g] is the item at
// position g (-1 past the last item), cnt[g] its list length.  Every thread
// of the block must call it.  `scratch` is written earlier in the same kernel
// by other threads of the block, so it is read through a plain (coherent)
// pointer after the barrier.
// The block's ranking by descending list length: thread t takes position
// b0 + t, whose item is b0 + *src (list length *cs, -1 past the last item).
template <int K>
__device__ __forceinline__ void count_rank(bool valid, int c, int *src, int *cs) {
    __shared__ int hist[K + 3];
    __shared__ int s_cnt[SC_THREADS], s_src[SC_THREADS];
    const int t = threadIdx.x;
    for (int b = t; b < K + 3; b += SC_THREADS) hist[b] = 0;
    s_cnt[t] = valid ? c : -1;
    __syncthreads();
    const int bin = valid ? 1 + min(c, K + 1) : 0;
    const int idx = atomicAdd(&hist[bin], 1);
    __syncthreads();
    if (t < 32) {  // exclusive prefix over bins, highest bin first
        int carry = 0;
        for (int top = K + 2; top >= 0; top -= 32) {
            const int b = top - t;
            const int v = b >= 0 ? hist[b] : 0;
            int x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, x, o);
                if (t >= o) x += y;
            }
            if (b >= 0) hist[b] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    s_src[hist[bin] + idx] = t;
    __syncthreads();
    *src = s_src[t];
    *cs = s_cnt[*src];
}

template <int K>
__device__ __forceinline__ void emit_count_ordered(bool valid, int c, int limit, int cap,
                                                   const uint32_t *scratch, uint32_t *__restrict__ list,
                                                   int *__restrict__ cnt, int *__restrict__ perm,
                                                   int *__restrict__ ovf = nullptr, int *__restrict__ ovfCount = nullptr) {
    const int b0 = blockIdx.x * SC_THREADS;
    int src, cs;
    count_rank<K>(valid, c, &src, &cs);
    const int g = b0 + threadIdx.x;
    if (g < cap) {
        perm[g] = cs >= 0 ? b0 + src : -1;
        cnt[g] = max(cs, 0);
    }
    const int n = min(max(cs, 0), min(K, limit));
    for (int k0 = 0; k0 < n; k0 += 8) {   // two chunks of four entries in flight together
        uint32_t e[8];
#pragma unroll
        for (int q = 0; q < 8; q++) e[q] = k0 + q < n ? scratch[sc_list_at(K, b0 + src, k0 + q)] : 0u;
        *reinterpret_cast<uint4 *>(list + sc_list4_at(K, g, k0)) = make_uint4(e[0], e[1], e[2], e[3]);
        if (k0 + 4 < n) *reinterpret_cast<uint4 *>(list + sc_list4_at(K, g, k0 + 4)) = make_uint4(e[4], e[5], e[6], e[7]);
    }
    if (ovf && cs > min(K, limit)) ovf[atomicAdd(ovfCount, 1)] = g;
}

// Bonds of one particle held in registers, with a one-word filter of the
// partner ids (bit id mod 32 set for each bond) that rules most candidates
// out before the slot-by-slot comparison.
struct BondRegs {
    int n;
    uint32_t filter;
    int t[SC_MAX_ACTIVE_INTERACTIONS], g[SC_MAX_ACTIVE_INTERACTIONS], p[SC_MAX_ACTIVE_INTERACTIONS];
    __device__ __forceinline__ void load(const int *__restrict__ nb, const int *__restrict__ bonds, int i) {
        n = min(max(nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
        filter = 0u;
#pragma unroll
        for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++) {
            const int *b = bonds + (size_t)i * 24 + 3 * k;
            t[k] = k < n ? b[0] : 0;
            g[k] = k < n ? b[1] : 0;
            p[k] = k < n ? b[2] : 0;
            if (k < n) filter |= 1u << (p[k] & 31);
        }
    }
    __device__ __forceinline__ bool has_partner(int id) const {
        if (!((filter >> (id & 31)) & 1u)) return false;
        bool r = false;
#pragma unroll
        for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++)
            if (k < n && p[k] == id) r = true;
        return r;
    }
};

// The tests of a candidate inside the interaction cube: returns the entry
// flags, 0 if the pair contributes nothing.
__device__ __forceinline__ uint32_t pp_flags_in_cube(sc_f3 delta, float trad, int j, float prad, int phydro,
                                                     const BondRegs &B, const int4 *__restrict__ info) {
    int4 tin = info[j];
    if (!(tin.z & SC_ACTIVE)) return 0;
    float dist = sc_norm3(delta);
    float s = prad + trad;
    int thydro = (int)(int8_t)(tin.w & 0xff);
    uint32_t f = 0;
    if ((phydro > 0 || thydro > 0) && sc_within_lipid_range(dist, s) && phydro == SC_POLAR && thydro == SC_POLAR)
        f |= SC_PP_POLAR;
    bool partner = B.has_partner(tin.x);
    if (partner) f |= SC_PP_PARTNER;
    if (!partner && dist < s) f |= SC_PP_COLLIDE;
    return f;
}

// The position-only tests of relax for candidate j of particle i
// (dynamics.cuh:452-478, 584-589, 775-777): returns the entry flags, 0 if
// the pair contributes nothing.
__device__ __forceinline__ uint32_t pp_flags(const ScParams &P, const Imager &IM, int i, int j, sc_f3 ppos, float prad,
                                             int phydro,
                                             const BondRegs &B, const float4 *__restrict__ pos,
                                             const int4 *__restrict__ info) {
    if (j == i) return 0;
    // the cube test first: most candidates fail it, and then need no record
    float4 t4 = pos[j];
    sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - ppos;
    if (outside_cube(delta, P.maxInt)) return 0;
    return pp_flags_in_cube(delta, t4.w, j, prad, phydro, B, info);
}

// Particle-particle list, built once after the sort; read by coordinateNoise
// and relax.
template <bool BATCH>
__device__ __forceinline__ void build_pp_block(
    ScParams P, ScanWords &W, int block, const uint32_t *__restrict__ cellStart, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ pos, const int4 *__restrict__ info, const int *__restrict__ nb,
    const int *__restrict__ bonds, uint32_t *__restrict__ list, int *__restrict__ cnt, int cap,
    int *__restrict__ classIdx, int *__restrict__ classCount, int *__restrict__ ovf, int *__restrict__ ovfCount,
    uint32_t *__restrict__ match, int *__restrict__ matchN, float4 *__restrict__ geo) {
    int i = block * SC_THREADS + threadIdx.x;
    if (i >= *nActivePtr) return;
    int4 in = info[i];
    int cls = 2;
    uint32_t inactive = 0;
    if (!(in.z & SC_ACTIVE)) {
        cnt[i] = 0;
        inactive = SC_CLASS_INACTIVE;
    } else {
        rep_apply<BATCH>(P, in.w);
        BondRegs B;
        B.load(nb, bonds, i);
        float4 p4 = pos[i];
        const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, ppos, SC_BINNED_P);
        const int phydro = (int)(int8_t)(in.w & 0xff);
        int c = 0, nm = 0;
        uint32_t any = 0;
        uint32_t *__restrict__ myMatch = match + (size_t)i * SC_MAX_ACTIVE_INTERACTIONS;
        const int K = min(SC_LIST_PP, P.listLimit);
        auto add = [&](int j, uint32_t f, sc_f3 delta, float4 t4) {
            if (c < K) list[sc_list_at(SC_LIST_PP, i, c)] = (uint32_t)j | f;
            // a colliding pair's position-only part of dynamics.cuh:775-786,
            // tpos - normalize(tpos - pos) * collisionDistance: the first
            // float3 its velocity term evaluates, the same in every
            // relaxation sub-iteration
            if ((f & SC_PP_COLLIDE) && c < SC_GEO_PP) {
                const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
                const sc_f3 a = tpos - normalize(delta) * (p4.w + t4.w);
                geo[sc_list_at(SC_GEO_PP, i, c)] = make_float4(a.x, a.y, a.z, t4.w);
            }
            c++;
            any |= f;
            if (f & SC_PP_PARTNER) {  // the bond slots naming this neighbour, in slot order
                const int tid_ = info[j].x;
#pragma unroll
                for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++)
                    if (k < B.n && B.p[k] == tid_ && nm < SC_MAX_ACTIVE_INTERACTIONS)
                        myMatch[nm++] = (uint32_t)j | ((uint32_t)k << 29);
            }
        };
        scan_words(P, W, pos, [&](uint32_t key) { return cellStart[key]; }, ppos, reach(P, ppos, P.maxInt, SC_BINNED_P),
                   P.maxInt, scan_mixed(P, IM, SC_BINNED_P), [&](int j, float4 t4) {
                       if (j == i) return;
                       const sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - ppos;
                       if (IM.wrap && outside_cube(delta, P.maxInt)) return;
                       const uint32_t f = pp_flags_in_cube(delta, t4.w, j, p4.w, phydro, B, info);
                       if (f) add(j, f, delta, t4);
                   });
        cnt[i] = c;
        // A test bond rotates the particle itself, which its later terms
        // read: its relaxation takes the in-order scan with the overflowed
        // items (its noise stays with the bonded class).
        bool testBond = false;
#pragma unroll
        for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++) testBond |= k < B.n && B.t[k] == 0;
        if (B.n >= 1) matchN[i] = nm | (testBond ? SC_MATCH_INORDER : 0);
        if (c > min(SC_LIST_PP, P.listLimit) || testBond) ovf[atomicAdd(ovfCount, 1)] = i;
        if (B.n >= 1) cls = 0;
        else if (c <= min(SC_LIST_PP, P.listLimit) && (any & SC_PP_POLAR)) cls = 1;
    }
    // append i to its class (warp-aggregated; order within a class is free)
    unsigned same = __match_any_sync(__activemask(), cls);
    int leader = __ffs(same) - 1, lane = threadIdx.x & 31;
    int base = 0;
    if (lane == leader) base = atomicAdd(&classCount[cls], __popc(same));
    base = __shfl_sync(same, base, leader);
    classIdx[(size_t)cls * cap + base + __popc(same & ((1u << lane) - 1u))] = i | (int)inactive;
}
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_build_pp(
    ScParams P, const uint32_t *__restrict__ cellStart, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ pos, const int4 *__restrict__ info, const int *__restrict__ nb,
    const int *__restrict__ bonds, uint32_t *__restrict__ list, int *__restrict__ cnt, int cap,
    int *__restrict__ classIdx, int *__restrict__ classCount, int *__restrict__ ovf, int *__restrict__ ovfCount,
    uint32_t *__restrict__ match, int *__restrict__ matchN, float4 *__restrict__ geo) {
    __shared__ ScanWords W;
    build_pp_block<BATCH>(P, W, blockIdx.x, cellStart, nActivePtr, pos, info, nb, bonds, list, cnt, cap, classIdx, classCount, ovf,
                          ovfCount, match, matchN, geo);
}

// Visits the contributing pairs of particle i in the reference's order: from
// the list, or (list overflow) by scanning.
template <class F>
__device__ __forceinline__ void for_pp(const ScParams &P, const uint32_t *__restrict__ cellStart,
                                       const PairList<SC_LIST_PP> &L, int i, sc_f3 ppos, float prad, int phydro,
                                       const int *__restrict__ nb, const int *__restrict__ bonds,
                                       const float4 *__restrict__ pos, const int4 *__restrict__ info, F &&f) {
    int c = L.cnt[i];
    if (c <= min(SC_LIST_PP, P.listLimit)) {
        for (int k = 0; k < c; k++) {
            uint32_t e = L.list[sc_list_at(SC_LIST_PP, i, k)];
            f((int)(e & SC_PP_INDEX), e);
        }
    } else {
        const Imager IM(P, ppos, SC_BINNED_P);
        BondRegs B;
        B.load(nb, bonds, i);
        scan27(P, cellStart, ppos, reach(P, ppos, P.maxInt, SC_BINNED_P), [&](int j) {
            uint32_t fl = pp_flags(P, IM, i, j, ppos, prad, phydro, B, pos, info);
            if (fl) f(j, fl);
        });
    }
}

// ---- dynamics.cuh:288-402 coordinateNoise -----------------------------------
// Only interaction partners change anything: for a listed item they are its
// bond matches (k_build_pp), in the reference's visiting order; an item
// whose list overflowed scans its neighbourhood.
// dynamics.cuh:288-402 for one particle; the new noise goes to pnOut / anOut.
template <bool BATCH>
__device__ __forceinline__ void coordinate_noise_item(
    const ScParams &P0, const uint32_t *__restrict__ cellStart, int i, const float4 *__restrict__ pos,
    const int4 *__restrict__ info, const int *__restrict__ nb, const int *__restrict__ bonds,
    const PairList<SC_LIST_PP> &L, const uint32_t *__restrict__ match, const int *__restrict__ matchN,
    const float4 *__restrict__ pnIn, const float4 *__restrict__ anIn, float4 *__restrict__ pnOut,
    float4 *__restrict__ anOut, float frac) {
    int4 in = info[i];
    float4 pn4 = pnIn[i], an4 = anIn[i];
    if (!(in.z & SC_ACTIVE) || nb[i] < 1) {
        *pnOut = pn4;
        *anOut = an4;
        return;
    }
    ScParams P = P0;
    rep_apply<BATCH>(P, in.w);
    const int nbi = min(max(nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
    const int *__restrict__ myBonds = bonds + (size_t)i * 24;
    float4 p4 = pos[i];
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const float prad = p4.w;
    sc_f3 ppn = sc_make_f3(pn4.x, pn4.y, pn4.z);
    sc_f4 pan = sc_make_f4(an4.x, an4.y, an4.z, an4.w);
    sc_f3 dPN = sc_zero3();
    sc_f4 dAN = sc_qid();
    float w = 0.0f;
    // one bond slot k naming neighbour j
    auto term = [&](int j, int k) {
        if (myBonds[3 * k] < 10 && frac > 0.25f) return;
        const float trad = pos[j].w;
        sc_f3 tpn = ld3(pnIn, j);
        sc_f4 tan_ = ld4(anIn, j);
        float pMag = length(ppn);
        dPN += (tpn - ppn) * 0.9f * trad / (prad + trad) * 1.0f;
        dPN *= fmaxf(length(dPN), pMag) / length(dPN);
        dAN = sc_slerp(dAN, sc_qmul(sc_qinv(pan), tan_), 0.9f * trad / (prad + trad) * 1.0f);
        w += 1.0f;
    };
    if (L.cnt[i] <= min(SC_LIST_PP, P.listLimit)) {
        const uint32_t *__restrict__ myMatch = match + (size_t)i * SC_MAX_ACTIVE_INTERACTIONS;
        const int nm = matchN[i] & SC_MATCH_COUNT;
        for (int m = 0; m < nm; m++) {
            const uint32_t e = myMatch[m];
            term((int)(e & SC_PP_INDEX), (int)(e >> 29));
        }
    } else {
        for_pp(P, cellStart, L, i, ppos, prad, (int)(int8_t)(in.w & 0xff), nb, bonds, pos, info,
               [&](int j, uint32_t fl) {
                   if (!(fl & SC_PP_PARTNER)) return;
                   const int tid_ = info[j].x;
#pragma unroll 1
                   for (int k = 0; k < nbi; k++)
                       if (myBonds[3 * k + 2] == tid_) term(j, k);
               });
    }
    ppn += dPN / fmaxf(w, 1.0f);
    pan = sc_qmul(sc_slerp(sc_qid(), dAN, 1.0f / fmaxf(w, 1.0f)), pan);
    st3(pnOut, 0, ppn, pn4.w);
    st4(anOut, 0, pan);
}


// Runs over the bonded work class (items with at least one bond), the new
// noise going to the fields' other buffers; every other item's noise is
// unchanged and copied there by the first launch of a run (age 0), after which
// both buffers hold it.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_coordinate_noise(
    ScParams P, const uint32_t *__restrict__ cellStart, const int *__restrict__ nActivePtr,
    const int *__restrict__ classIdx, const int *__restrict__ classCount, const float4 *__restrict__ pos,
    const int4 *__restrict__ info, const int *__restrict__ nb, const int *__restrict__ bonds, PairList<SC_LIST_PP> L,
    const uint32_t *__restrict__ match, const int *__restrict__ matchN, const float4 *__restrict__ pnIn,
    const float4 *__restrict__ anIn, float4 *__restrict__ pnOut, float4 *__restrict__ anOut, float frac, int age) {
    const int n0 = classCount[0], first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (int t = first; t < n0; t += stride) {
        const int i = classIdx[t];
        coordinate_noise_item<BATCH>(P, cellStart, i, pos, info, nb, bonds, L, match, matchN, pnIn, anIn, pnOut + i,
                                     anOut + i, frac);
    }
    if (age > 0) return;
    for (int i = first, n = *nActivePtr; i < n; i += stride) {
        if ((info[i].z & SC_ACTIVE) && nb[i] >= 1) continue;
        pnOut[i] = pnIn[i];
        anOut[i] = anIn[i];
    }
}

// ---- dynamics.cuh:405-822 relax ------------------------------------------------
struct RelaxArgs {
    const uint32_t *__restrict__ cellStart;
    const float4 *__restrict__ pos;
    const int4 *__restrict__ info;
    const int *__restrict__ nb;
    const int *__restrict__ bonds;
    PairList<SC_LIST_PP> L;
    const float4 *__restrict__ velIn, *__restrict__ rotIn, *__restrict__ avIn;
    float4 *__restrict__ velOut, *__restrict__ rotOut, *__restrict__ avOut, *__restrict__ dbg;
    const int *__restrict__ classIdx;    // items by work class (k_build_pp)
    const int *__restrict__ classCount;
    const uint32_t *__restrict__ match;  // bond matches of the list (k_build_pp)
    const int *__restrict__ matchN;
    const float4 *__restrict__ geo;      // colliding pairs' geometry (k_build_pp)
    const uint4 *__restrict__ bondRec;   // bonded class, a record per item (k_bond_plan)
    const int *__restrict__ ovf, *__restrict__ ovfCount;   // items left to the in-order scan
    int *__restrict__ unsettled;  // set when an unturned angular velocity is not a fixed point (relax_still)
    // sub-iterations since the input and output buffers of rot / angvel were
    // last out of step (0, 1, 2 and more): what does not change in a
    // sub-iteration is written until both buffers hold it
    int age;
};

// The relaxation of a particle that holds a test bond, pair by pair, or whose
// list overflowed: then its 27 cells are visited and the list's tests applied
// to each candidate.  The bond loop reads the particle's bonds from memory one at a
// time, so its body is emitted once; out of line, so that the lists' code
// does not carry its registers.
__device__ __noinline__ void relax_scan_item(const ScParams &P, const RelaxArgs &A, int i, int4 in, float4 v4, float4 r4,
                                           float4 a4) {
    float4 p4 = A.pos[i];
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, ppos, SC_BINNED_P);
    const float prad = p4.w;
    const sc_f3 pvel = sc_make_f3(v4.x, v4.y, v4.z);
    sc_f4 prot = sc_make_f4(r4.x, r4.y, r4.z, r4.w);
    sc_f4 pav = sc_make_f4(a4.x, a4.y, a4.z, a4.w);
    const int pid = in.x, ptype = in.y, phydro = (int)(int8_t)(in.w & 0xff);
    const int nbi = min(max(A.nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
    const int *__restrict__ myBonds = A.bonds + (size_t)i * 24;
    sc_f4 pdbg = sc_make_f4(0, 0, 0, 0);
    bool dbgTouched = false;
    sc_f3 dV = sc_zero3();
    sc_f4 dAV = sc_qid();
    sc_f3 phobPos = sc_zero3();
    float phobSum = 0.0f;
    float w = 0.0f;
    const sc_f3 up = sc_rotate(sc_up(), prot);
    const sc_f3 nextUp = sc_rotate(up, pav);
    const float flex = SC_PI_REF / 8;
    auto body = [&](int j, uint32_t fl) {
        float4 t4 = A.pos[j];
        const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
        const float trad = t4.w;
        const float idist = prad + trad;
        if (fl & SC_PP_POLAR) {
            // dynamics.cuh:478-582: polar (lipid) head / tail attraction
            sc_f3 tvel = ld3(A.velIn, j);
            sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), ld4(A.rotIn, j)), pav);
            sc_f3 pPV = -nextUp * prad + ppos + pvel;
            sc_f3 tpPV = -nextTup * trad + tpos + tvel;
            float Lr = length(tpPV - pPV) / (prad + trad);
            float attr = sc_polar_attr(Lr);
            w += 1.0f;
            dV += (tpPV - pPV) * 0.05f * attr * 1.0f;
            float pap = sc_powf(fminf(1.0f / fmaxf(Lr, 1e-6f), 10.0f) / 10.0f, 0.2f);
            phobSum += pap;
            phobPos += tpPV * pap;
        }
        if (fl & SC_PP_PARTNER) {
            // dynamics.cuh:584-771: interaction partners, in bond-slot order
            int4 tin = A.info[j];
            const int tid_ = tin.x, ttype = tin.y;
#pragma unroll 1
            for (int k = 0; k < nbi; k++) {
                if (myBonds[3 * k + 2] != tid_) continue;
                const int it = myBonds[3 * k];
                if (it >= 10) {
                    const sc_rule &pii = rule_at(P, it);
                    sc_f4 ro = rule_ori(pii);
                    sc_f3 rp = rule_pos(pii);
                    sc_f4 trot = ld4(A.rotIn, j), tav = ld4(A.avIn, j);
                    sc_f3 tvel = ld3(A.velIn, j);
                    bool o1 = p_order(ptype, pid, ttype, tid_), o2 = p_order(ttype, tid_, ptype, pid);
                    sc_f4 tro_p = o1 ? sc_qmul(trot, sc_qinv(ro)) : sc_qmul(trot, ro);
                    sc_f4 tro_t = o2 ? sc_qmul(prot, sc_qinv(ro)) : sc_qmul(prot, ro);
                    sc_f4 rro = sc_qmul(sc_qinv(sc_qmul(pav, prot)), sc_qmul(tav, tro_p));
                    sc_f4 orro = sc_qmul(sc_qinv(sc_qmul(tav, trot)), sc_qmul(pav, tro_t));
                    dAV = sc_slerp(dAV, sc_qmul(sc_slerp(rro, orro, 0.5f), rro), 0.9f * trad / (prad + trad));
                    sc_f3 rrp = o1 ? sc_rotate(-rp, sc_qmul(sc_qinv(ro), sc_qmul(tav, trot)))
                                   : sc_rotate(rp, sc_qmul(tav, trot));
                    rrp += tpos;
                    sc_f3 orrp = o2 ? sc_rotate(-rp, sc_qmul(sc_qinv(ro), sc_qmul(pav, prot)))
                                    : sc_rotate(rp, sc_qmul(pav, prot));
                    orrp += ppos;
                    w += 1.0f;
                    sc_f3 pDV = (rrp + tvel - (ppos + pvel)) * 0.9f * trad / (prad + trad) * 1.0f;
                    sc_f3 tpDV = (orrp + pvel - (tpos + tvel)) * 0.9f * prad / (prad + trad) * 1.0f;
                    dV += (pDV - (pDV + tpDV) / 2.0f) * 0.9f * prad / (prad + trad) * 1.0f;
                }
                if (it == 0) {
                    if (!dbgTouched) { pdbg = ld4(A.dbg, i); dbgTouched = true; }
                    sc_f4 trot = ld4(A.rotIn, j);
                    bool o1 = p_order(ptype, pid, ttype, tid_);
                    sc_f4 trod = sc_qmul(sc_quat(sc_up(), -SC_PI_REF / 6), sc_quat(sc_right(), SC_PI_REF / 6));
                    prot = sc_slerp(prot, o1 ? sc_qmul(trot, sc_qinv(trod)) : sc_qmul(trot, trod), 0.2f);
                    sc_f4 trpr = sc_quat(sc_forward(), -SC_PI_REF / 6);
                    sc_f3 rrp = o1 ? -sc_rotate(sc_up(), sc_qmul(trot, sc_qmul(sc_qinv(trod), trpr)))
                                   : sc_rotate(sc_up(), sc_qmul(trot, trpr));
                    rrp *= idist;
                    rrp += tpos;
                    pdbg.x = (float)((double)pdbg.x + (double)(rrp.x - ppos.x) * (1.0 - (double)0.2f));
                    pdbg.y = (float)((double)pdbg.y + (double)(rrp.y - ppos.y) * (1.0 - (double)0.2f));
                    pdbg.z = (float)((double)pdbg.z + (double)(rrp.z - ppos.z) * (1.0 - (double)0.2f));
                } else if (it == SC_INTERACTION_TYPE_CHAIN) {
                    if (!dbgTouched) { pdbg = ld4(A.dbg, i); dbgTouched = true; }
                    sc_f3 tvel = ld3(A.velIn, j);
                    sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), ld4(A.rotIn, j)), pav);
                    sc_f3 nnd = normalize(tpos + tvel - (ppos + pvel));
                    bool fwd = myBonds[3 * k + 1] == SC_INTERACTION_GROUP_FORWARD;
                    dAV = sc_slerp(dAV, sc_quat_from_to(nextUp, (fwd ? -1.0f : 1.0f) * nnd),
                                   0.9f * trad / (prad + trad));
                    sc_f3 relUp = (fwd ? 1.0f : -1.0f) * nextTup;
                    sc_f3 axis = sc_safe_cross(relUp, -nnd);
                    float ang = sc_angle3(relUp, -nnd);
                    sc_f3 rrp = sc_rotate(relUp, sc_quat(axis, fminf(fmaxf(ang, -flex), flex)));
                    rrp *= idist;
                    rrp += tpos;
                    sc_f3 oUp = (fwd ? -1.0f : 1.0f) * nextUp;
                    sc_f3 oaxis = sc_safe_cross(oUp, nnd);
                    float oang = sc_angle3(oUp, nnd);
                    sc_f3 orrp = sc_rotate(oUp, sc_quat(oaxis, fminf(fmaxf(oang, -flex), flex)));
                    orrp *= idist;
                    orrp += ppos;
                    w += 1.0f;
                    sc_f3 pDV = (rrp + tvel - (ppos + pvel)) * 0.9f * trad / (prad + trad) * 1.0f;
                    sc_f3 tpDV = (orrp + pvel - (tpos + tvel)) * 0.9f * prad / (prad + trad) * 1.0f;
                    dV += (pDV - (pDV + tpDV) / 2.0f) * 0.9f * prad / (prad + trad) * 1.0f;
                    pdbg.x = (float)((double)pdbg.x + (double)(rrp.x - ppos.x) * (1.0 - (double)0.9f));
                    pdbg.y = (float)((double)pdbg.y + (double)(rrp.y - ppos.y) * (1.0 - (double)0.9f));
                    pdbg.z = (float)((double)pdbg.z + (double)(rrp.z - ppos.z) * (1.0 - (double)0.9f));
                }
            }
        }
        if (fl & SC_PP_COLLIDE) {
            // dynamics.cuh:775-786: soft collision with a non-partner
            sc_f3 nd = normalize(tpos - ppos);
            float cd = prad + trad;
            sc_f3 tvel = ld3(A.velIn, j);
            w += 1.0f;
            dV += (tpos - nd * cd + tvel - (ppos + pvel)) * 0.9f * trad / (prad + trad) * 1.0f;
        }
    };
    // the pairs in the reference's order, from the list where there is one
    // (a test bond's item: its list holds what the scan would find)
    const int c = A.L.cnt[i];
    if (c <= min(SC_LIST_PP, P.listLimit)) {
        for (int k = 0; k < c; k++) {
            const uint32_t e = A.L.list[sc_list_at(SC_LIST_PP, i, k)];
            body((int)(e & SC_PP_INDEX), e);
        }
    } else {
        BondRegs B;
        B.load(A.nb, A.bonds, i);
        scan27(P, A.cellStart, ppos, reach(P, ppos, P.maxInt, SC_BINNED_P), [&](int j) {
            uint32_t fl = pp_flags(P, IM, i, j, ppos, prad, phydro, B, A.pos, A.info);
            if (fl) body(j, fl);
        });
    }
    sc_f3 nv = pvel + dV / fmaxf(w, 1.0f);
    pav = sc_qmul(sc_slerp(sc_qid(), dAV, 1.0f / fmaxf(w, 1.0f)), pav);
    if (phobSum > 0.0f) {
        sc_f3 dir = normalize(phobPos / phobSum - (ppos + nv));
        pav = sc_slerp(pav, sc_quat_from_to(-up, dir), 0.2f);
    }
    st3(A.velOut, i, nv, v4.w);
    st4(A.rotOut, i, prot);
    st4(A.avOut, i, pav);
    if (dbgTouched) st4(A.dbg, i, pdbg);
}

// The geometry of colliding entry k of item i with neighbour j, as k_build_pp
// stores it for the first SC_GEO_PP entries ({A.x, A.y, A.z, radius}).
__device__ __forceinline__ float4 collide_geo(const Imager &IM, sc_f3 ppos, float prad, float4 t4) {
    const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
    const sc_f3 a = tpos - normalize(tpos - ppos) * (prad + t4.w);
    return make_float4(a.x, a.y, a.z, t4.w);
}
// dynamics.cuh:775-786, the velocity term of a colliding pair (ppv the item's
// position plus its velocity).
__device__ __forceinline__ sc_f3 collide_term(float4 g, float4 tv, sc_f3 ppv, float prad) {
    return (sc_make_f3(g.x, g.y, g.z) + sc_make_f3(tv.x, tv.y, tv.z) - ppv) * 0.9f * g.w / (prad + g.w) * 1.0f;
}

// The angular velocity of an item no bond or polar pair turns.  The
// reference multiplies it by slerp(1, 1, t), t = 1 / max(w, 1) with w a count:
// fl(1 - t) + t rounds to 1 for every such t, so the factor is exactly the
// identity quaternion (0, 0, 0, 1), and the product changes nothing but the
// sign of a zero component or non-finite values.  The product is formed until
// both buffers hold it; when the second sub-iteration still changes a bit of
// some item (A.unsettled), every later one forms it too.
__device__ __forceinline__ void relax_still(const RelaxArgs &A, int i) {
    if (A.age >= 2 && *A.unsettled == 0) return;
    const float4 a4 = A.avIn[i];
    const sc_f4 o = sc_qmul(sc_qid(), sc_make_f4(a4.x, a4.y, a4.z, a4.w));
    A.avOut[i] = make_float4(o.x, o.y, o.z, o.w);
    if (A.age == 1 && (sc_f2u(o.x) != sc_f2u(a4.x) || sc_f2u(o.y) != sc_f2u(a4.y) || sc_f2u(o.z) != sc_f2u(a4.z) ||
                       sc_f2u(o.w) != sc_f2u(a4.w)))
        *A.unsettled = 1;
}

// A plain particle's relaxation (work class 2: collisions only): its records,
// its list count and its first SC_PLAIN_GROUP entries with their geometry lie
// at places known from its index, so the item waits one memory latency for
// them and one more for its neighbours' velocities.  Neither rot nor angvel
// turns (relax_still), so from the third sub-iteration on only velocities
// move: 56 bytes an item instead of 156, beside its pairs.
#define SC_PLAIN_GROUP 4
template <bool BATCH>
__device__ __forceinline__ void relax_plain(const ScParams &P0, const RelaxArgs &A, int e) {
    const int i = (int)((uint32_t)e & ~SC_CLASS_INACTIVE);
    if ((uint32_t)e & SC_CLASS_INACTIVE) {
        if (A.age == 0) {   // both buffers hold its records from then on
            A.velOut[i] = A.velIn[i];
            A.rotOut[i] = A.rotIn[i];
            A.avOut[i] = A.avIn[i];
        }
        return;
    }
    const int c = A.L.cnt[i];
    const float4 v4 = A.velIn[i], p4 = A.pos[i];
    uint32_t en[SC_PLAIN_GROUP];
    float4 g[SC_PLAIN_GROUP];
#pragma unroll
    for (int q = 0; q < SC_PLAIN_GROUP; q++) en[q] = A.L.list[sc_list_at(SC_LIST_PP, i, q)];
    if (c > min(SC_LIST_PP, P0.listLimit)) return;   // left to the scan
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const float prad = p4.w;
    const sc_f3 pvel = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = ppos + pvel;
    sc_f3 dV = sc_zero3();
    for (int k0 = 0; k0 < c; k0 += SC_PLAIN_GROUP) {
        if (k0 > 0) {
#pragma unroll
            for (int q = 0; q < SC_PLAIN_GROUP; q++)
                en[q] = k0 + q < c ? A.L.list[sc_list_at(SC_LIST_PP, i, k0 + q)] : 0u;
        }
        float4 tv[SC_PLAIN_GROUP];
        const bool kept = k0 < SC_GEO_PP;
#pragma unroll
        for (int q = 0; q < SC_PLAIN_GROUP; q++) {
            g[q] = make_float4(0, 0, 0, 0);
            tv[q] = g[q];
            if (k0 + q < c) {
                const int j = (int)(en[q] & SC_PP_INDEX);
                g[q] = kept ? A.geo[sc_list_at(SC_GEO_PP, i, k0 + q)] : A.pos[j];
                tv[q] = A.velIn[j];
            }
        }
        if (!kept) {
            ScParams P = P0;
            if (BATCH) rep_apply<BATCH>(P, A.info[i].w);
            const Imager IM(P, ppos, SC_BINNED_P);
#pragma unroll
            for (int q = 0; q < SC_PLAIN_GROUP; q++)
                if (k0 + q < c) g[q] = collide_geo(IM, ppos, prad, g[q]);
        }
#pragma unroll
        for (int q = 0; q < SC_PLAIN_GROUP; q++)
            if (k0 + q < c) dV += collide_term(g[q], tv[q], ppv, prad);
    }
    st3(A.velOut, i, pvel + dV / fmaxf((float)c, 1.0f), v4.w);
    if (A.age == 0) A.rotOut[i] = A.rotIn[i];
    relax_still(A, i);
}

// A polar particle's relaxation (work class 1: polar and collision pairs):
// the terms in list order, with the entries of SC_POLAR_GROUP pairs, then
// their neighbours' records, loaded together.
#define SC_POLAR_GROUP 2
template <bool BATCH>
__device__ __forceinline__ void relax_polar(const ScParams &P0, const RelaxArgs &A, int i) {
    const int c = A.L.cnt[i];
    const float4 v4 = A.velIn[i], r4 = A.rotIn[i], a4 = A.avIn[i], p4 = A.pos[i];
    if (c > min(SC_LIST_PP, P0.listLimit)) return;   // left to the scan
    ScParams P = P0;
    if (BATCH) rep_apply<BATCH>(P, A.info[i].w);
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, ppos, SC_BINNED_P);
    const float prad = p4.w;
    const sc_f3 pvel = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = ppos + pvel;
    const sc_f4 prot = sc_make_f4(r4.x, r4.y, r4.z, r4.w);
    sc_f4 pav = sc_make_f4(a4.x, a4.y, a4.z, a4.w);
    sc_f3 dV = sc_zero3();
    const sc_f4 dAV = sc_qid();
    sc_f3 phobPos = sc_zero3();
    float phobSum = 0.0f;
    float w = 0.0f;
    const sc_f3 up = sc_rotate(sc_up(), prot);
    const sc_f3 nextUp = sc_rotate(up, pav);
    for (int k0 = 0; k0 < c; k0 += SC_POLAR_GROUP) {
        uint32_t e[SC_POLAR_GROUP];
#pragma unroll
        for (int q = 0; q < SC_POLAR_GROUP; q++) e[q] = k0 + q < c ? A.L.list[sc_list_at(SC_LIST_PP, i, k0 + q)] : 0u;
        float4 t4[SC_POLAR_GROUP], tv[SC_POLAR_GROUP], tr[SC_POLAR_GROUP];
#pragma unroll
        for (int q = 0; q < SC_POLAR_GROUP; q++) {
            t4[q] = make_float4(0, 0, 0, 0);
            tv[q] = t4[q];
            tr[q] = t4[q];
            if (k0 + q < c) {
                const int j = (int)(e[q] & SC_PP_INDEX);
                t4[q] = A.pos[j];
                if (e[q] & (SC_PP_POLAR | SC_PP_COLLIDE)) tv[q] = A.velIn[j];
                if (e[q] & SC_PP_POLAR) tr[q] = A.rotIn[j];
            }
        }
#pragma unroll
        for (int q = 0; q < SC_POLAR_GROUP; q++) {
            if (k0 + q >= c) break;
            const uint32_t fl = e[q];
            const float trad = t4[q].w;
            if (fl & SC_PP_POLAR) {
                // dynamics.cuh:478-582: polar (lipid) head / tail attraction
                const sc_f3 tpos = IM(sc_make_f3(t4[q].x, t4[q].y, t4[q].z));
                const sc_f3 tvel = sc_make_f3(tv[q].x, tv[q].y, tv[q].z);
                sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), sc_make_f4(tr[q].x, tr[q].y, tr[q].z, tr[q].w)), pav);
                sc_f3 pPV = -nextUp * prad + ppos + pvel;
                sc_f3 tpPV = -nextTup * trad + tpos + tvel;
                float Lr = length(tpPV - pPV) / (prad + trad);
                float attr = sc_polar_attr(Lr);
                w += 1.0f;
                dV += (tpPV - pPV) * 0.05f * attr * 1.0f;
                float pap = sc_powf(fminf(1.0f / fmaxf(Lr, 1e-6f), 10.0f) / 10.0f, 0.2f);
                phobSum += pap;
                phobPos += tpPV * pap;
            }
            if (fl & SC_PP_COLLIDE) {
                w += 1.0f;
                dV += collide_term(collide_geo(IM, ppos, prad, t4[q]), tv[q], ppv, prad);
            }
        }
    }
    sc_f3 nv = pvel + dV / fmaxf(w, 1.0f);
    pav = sc_qmul(sc_slerp(sc_qid(), dAV, 1.0f / fmaxf(w, 1.0f)), pav);
    if (phobSum > 0.0f) {
        sc_f3 dir = normalize(phobPos / phobSum - (ppos + nv));
        pav = sc_slerp(pav, sc_quat_from_to(-up, dir), 0.2f);
    }
    st3(A.velOut, i, nv, v4.w);
    if (A.age == 0) A.rotOut[i] = r4;
    st4(A.avOut, i, pav);
}

// The same by SC_POLAR_LANES threads per item, for sims that do not fill the
// device: each thread forms the terms of every SC_POLAR_LANES-th pair, and
// the group's threads add them all in list order (so each holds the sums).
// One thread per item was the longest chain of a small sim's launch (the
// powf, roots and divisions of some eight entries one after another).
#define SC_POLAR_LANES 4
template <bool BATCH>
__device__ __forceinline__ void relax_polar_lanes(const ScParams &P0, const RelaxArgs &A, int i) {
    const int lane = threadIdx.x & 31, sub = lane & (SC_POLAR_LANES - 1), first = lane & ~(SC_POLAR_LANES - 1);
    const unsigned group = ((1u << SC_POLAR_LANES) - 1u) << first;
    const int c = A.L.cnt[i];
    const float4 v4 = A.velIn[i], r4 = A.rotIn[i], a4 = A.avIn[i], p4 = A.pos[i];
    uint32_t e = A.L.list[sc_list_at(SC_LIST_PP, i, sub)];
    if (c > min(SC_LIST_PP, P0.listLimit)) return;   // left to the scan
    ScParams P = P0;
    if (BATCH) rep_apply<BATCH>(P, A.info[i].w);
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, ppos, SC_BINNED_P);
    const float prad = p4.w;
    const sc_f3 pvel = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = ppos + pvel;
    const sc_f4 prot = sc_make_f4(r4.x, r4.y, r4.z, r4.w);
    sc_f4 pav = sc_make_f4(a4.x, a4.y, a4.z, a4.w);
    sc_f3 dV = sc_zero3();
    const sc_f4 dAV = sc_qid();
    sc_f3 phobPos = sc_zero3();
    float phobSum = 0.0f;
    float w = 0.0f;
    const sc_f3 up = sc_rotate(sc_up(), prot);
    const sc_f3 nextUp = sc_rotate(up, pav);
    for (int k0 = 0; k0 < c; k0 += SC_POLAR_LANES) {
        if (k0 > 0) e = k0 + sub < c ? A.L.list[sc_list_at(SC_LIST_PP, i, k0 + sub)] : 0u;
        const uint32_t fl = k0 + sub < c ? e : 0u;
        sc_f3 polar = sc_zero3(), pull = sc_zero3(), push = sc_zero3();
        float pap = 0.0f;
        if (fl) {
            const int j = (int)(fl & SC_PP_INDEX);
            const float4 t4 = A.pos[j], tv = A.velIn[j];
            if (fl & SC_PP_POLAR) {
                // dynamics.cuh:478-582: polar (lipid) head / tail attraction
                const float4 tr = A.rotIn[j];
                const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
                const float trad = t4.w;
                const sc_f3 tvel = sc_make_f3(tv.x, tv.y, tv.z);
                sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), sc_make_f4(tr.x, tr.y, tr.z, tr.w)), pav);
                sc_f3 pPV = -nextUp * prad + ppos + pvel;
                sc_f3 tpPV = -nextTup * trad + tpos + tvel;
                float Lr = length(tpPV - pPV) / (prad + trad);
                float attr = sc_polar_attr(Lr);
                polar = (tpPV - pPV) * 0.05f * attr * 1.0f;
                pap = sc_powf(fminf(1.0f / fmaxf(Lr, 1e-6f), 10.0f) / 10.0f, 0.2f);
                pull = tpPV * pap;
            }
            if (fl & SC_PP_COLLIDE) push = collide_term(collide_geo(IM, ppos, prad, t4), tv, ppv, prad);
        }
        __syncwarp(group);
#pragma unroll
        for (int u = 0; u < SC_POLAR_LANES; u++) {
            const uint32_t f = __shfl_sync(group, fl, first + u);
            const sc_f3 a = sc_make_f3(__shfl_sync(group, polar.x, first + u), __shfl_sync(group, polar.y, first + u),
                                       __shfl_sync(group, polar.z, first + u));
            const sc_f3 b = sc_make_f3(__shfl_sync(group, pull.x, first + u), __shfl_sync(group, pull.y, first + u),
                                       __shfl_sync(group, pull.z, first + u));
            const sc_f3 d = sc_make_f3(__shfl_sync(group, push.x, first + u), __shfl_sync(group, push.y, first + u),
                                       __shfl_sync(group, push.z, first + u));
            const float q = __shfl_sync(group, pap, first + u);
            if (f & SC_PP_POLAR) {
                w += 1.0f;
                dV += a;
                phobSum += q;
                phobPos += b;
            }
            if (f & SC_PP_COLLIDE) {
                w += 1.0f;
                dV += d;
            }
        }
    }
    sc_f3 nv = pvel + dV / fmaxf(w, 1.0f);
    pav = sc_qmul(sc_slerp(sc_qid(), dAV, 1.0f / fmaxf(w, 1.0f)), pav);
    if (phobSum > 0.0f) {
        sc_f3 dir = normalize(phobPos / phobSum - (ppos + nv));
        pav = sc_slerp(pav, sc_quat_from_to(-up, dir), 0.2f);
    }
    if (sub) return;
    st3(A.velOut, i, nv, v4.w);
    if (A.age == 0) A.rotOut[i] = r4;
    st4(A.avOut, i, pav);
}

// The bonded class's items in the order they are relaxed: each block of
// SC_THREADS ranked by bond-match count, chain-bonded items apart from
// rule-bonded ones (their pose terms are different code), so that a warp's
// lanes walk about as many bond terms of the same kind, with what an item's
// first loads depend on beside its index:
//   x  the item (-1: left to the scan)
//   y  its first bond match (k_build_pp; ~0: none)
//   z  that bond's interaction type
//   w  match count (bits 0-3) | first bond forward (4) | has polar pairs (5) |
//      list count (8-15) | terms in all (16-31)
__global__ void __launch_bounds__(SC_THREADS) k_bond_plan(ScParams P, PairList<SC_LIST_PP> L,
                                                          const int *__restrict__ classIdx,
                                                          const int *__restrict__ classCount,
                                                          const int *__restrict__ bonds,
                                                          const uint32_t *__restrict__ match,
                                                          const int *__restrict__ matchN, uint4 *__restrict__ rec) {
    __shared__ uint4 s_rec[SC_THREADS];
    const int n = classCount[0];
    for (int base = blockIdx.x * SC_THREADS; base < n; base += gridDim.x * SC_THREADS) {
        const int t = base + threadIdx.x;
        int key = 0;
        if (t < n) {
            const int i = classIdx[t];
            const int c = L.cnt[i];
            uint4 r = make_uint4(0xffffffffu, 0xffffffffu, 0u, 0u);
            if (c <= min(SC_LIST_PP, P.listLimit) && !(matchN[i] & SC_MATCH_INORDER)) {
                const int nm = min(matchN[i] & SC_MATCH_COUNT, SC_MAX_ACTIVE_INTERACTIONS);
                const int *__restrict__ b = bonds + (size_t)i * 24;
                int terms = 0;
                uint32_t any = 0;
                for (int k = 0; k < c; k++) {
                    const uint32_t e = L.list[sc_list_at(SC_LIST_PP, i, k)];
                    any |= e;
                    terms += ((e & SC_PP_POLAR) != 0) + ((e & SC_PP_COLLIDE) != 0);
                }
                const uint32_t *__restrict__ m = match + (size_t)i * SC_MAX_ACTIVE_INTERACTIONS;
                for (int k = 0; k < nm; k++) {
                    const int it = b[3 * (int)(m[k] >> 29)];
                    terms += it >= 10 || it == SC_INTERACTION_TYPE_CHAIN;
                }
                r.x = (uint32_t)i;
                uint32_t fwd = 0;
                if (nm > 0) {
                    const int k = (int)(m[0] >> 29);
                    r.y = m[0];
                    r.z = (uint32_t)b[3 * k];
                    fwd = b[3 * k + 1] == SC_INTERACTION_GROUP_FORWARD;
                }
                r.w = (uint32_t)nm | (fwd << 4) | ((any & SC_PP_POLAR) ? 1u << 5 : 0u) | ((uint32_t)c << 8) |
                      ((uint32_t)terms << 16);
            }
            key = (matchN[i] & SC_MATCH_COUNT) +
                  (bonds[(size_t)i * 24] == SC_INTERACTION_TYPE_CHAIN ? SC_MAX_ACTIVE_INTERACTIONS + 1 : 0);
            s_rec[threadIdx.x] = r;
        }
        int src, cs;
        count_rank<2 * SC_MAX_ACTIVE_INTERACTIONS + 1>(t < n, key, &src, &cs);
        if (cs >= 0) rec[t] = s_rec[src];
        __syncthreads();  // the shared arrays are reused by the next round
    }
}

// One bond of a bonded particle: what its pose terms read of the neighbour.
struct BondPair {
    int it;          // interaction type
    bool fwd;        // chain bonds: this particle's side
    bool o1, o2;     // rule bonds: p_order both ways
    sc_f3 tpos, tvel;
    float trad;
    sc_f4 trot, tav;
};
struct BondSelf {
    sc_f3 ppos, pvel, nextUp;
    float prad;
    sc_f4 prot, pav;
};
__device__ __forceinline__ bool bond_turns(int it) { return it >= 10 || it == SC_INTERACTION_TYPE_CHAIN; }

// The slerp target of dAV (dynamics.cuh:591-622, 700-712).
__device__ __forceinline__ sc_f4 bond_target(const ScParams &P, const BondSelf &S, const BondPair &b) {
    if (b.it >= 10) {
        const sc_f4 ro = rule_ori(rule_at(P, b.it));
        sc_f4 tro_p = b.o1 ? sc_qmul(b.trot, sc_qinv(ro)) : sc_qmul(b.trot, ro);
        sc_f4 tro_t = b.o2 ? sc_qmul(S.prot, sc_qinv(ro)) : sc_qmul(S.prot, ro);
        sc_f4 rro = sc_qmul(sc_qinv(sc_qmul(S.pav, S.prot)), sc_qmul(b.tav, tro_p));
        sc_f4 orro = sc_qmul(sc_qinv(sc_qmul(b.tav, b.trot)), sc_qmul(S.pav, tro_t));
        return sc_qmul(sc_slerp(rro, orro, 0.5f), rro);
    }
    sc_f3 nnd = normalize(b.tpos + b.tvel - (S.ppos + S.pvel));
    return sc_quat_from_to(S.nextUp, (b.fwd ? -1.0f : 1.0f) * nnd);
}

// The velocity term (dynamics.cuh:623-655, 713-769); chain bonds also give
// rrp - ppos for the debug vector.
__device__ __forceinline__ sc_f3 bond_velocity(const ScParams &P, const BondSelf &S, const BondPair &b, sc_f3 *dd) {
    const float prad = S.prad, trad = b.trad, idist = prad + trad;
    const sc_f3 ppos = S.ppos, pvel = S.pvel;
    sc_f3 rrp, orrp;
    if (b.it >= 10) {
        const sc_rule &pii = rule_at(P, b.it);
        const sc_f4 ro = rule_ori(pii);
        const sc_f3 rp = rule_pos(pii);
        rrp = b.o1 ? sc_rotate(-rp, sc_qmul(sc_qinv(ro), sc_qmul(b.tav, b.trot))) : sc_rotate(rp, sc_qmul(b.tav, b.trot));
        rrp += b.tpos;
        orrp = b.o2 ? sc_rotate(-rp, sc_qmul(sc_qinv(ro), sc_qmul(S.pav, S.prot))) : sc_rotate(rp, sc_qmul(S.pav, S.prot));
        orrp += ppos;
    } else {
        const float flex = SC_PI_REF / 8;
        sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), b.trot), S.pav);
        sc_f3 nnd = normalize(b.tpos + b.tvel - (ppos + pvel));
        sc_f3 relUp = (b.fwd ? 1.0f : -1.0f) * nextTup;
        sc_f3 axis = sc_safe_cross(relUp, -nnd);
        float ang = sc_angle3(relUp, -nnd);
        rrp = sc_rotate(relUp, sc_quat(axis, fminf(fmaxf(ang, -flex), flex)));
        rrp *= idist;
        rrp += b.tpos;
        sc_f3 oUp = (b.fwd ? -1.0f : 1.0f) * S.nextUp;
        sc_f3 oaxis = sc_safe_cross(oUp, nnd);
        float oang = sc_angle3(oUp, nnd);
        orrp = sc_rotate(oUp, sc_quat(oaxis, fminf(fmaxf(oang, -flex), flex)));
        orrp *= idist;
        orrp += ppos;
        *dd = rrp - ppos;
    }
    sc_f3 pDV = (rrp + b.tvel - (ppos + pvel)) * 0.9f * trad / (prad + trad) * 1.0f;
    sc_f3 tpDV = (orrp + pvel - (b.tpos + b.tvel)) * 0.9f * prad / (prad + trad) * 1.0f;
    return (pDV - (pDV + tpDV) / 2.0f) * 0.9f * prad / (prad + trad) * 1.0f;
}

// A block of bonded particles (work class 0), each relaxed by two threads in
// different warps.  Only bond terms turn dAV, and the velocity needs none of
// it, so one warp of a pair carries the orientation -- the slerp targets of the
// items' bond matches and dAV's chain over them -- and the other the velocity: the matches' velocity
// terms, then the list walked once to add every term in the reference's order
// (a test bond rotates the particle itself, which later terms read: such
// particles take the in-order scan).  The divisor of dAV's last slerp is a
// count the plan knows.  An item with polar pairs turns once more, towards
// its neighbours, when its velocity is known: its second thread finishes it
// with the first one's quaternion.
//
// Bound: the latency of one item's instruction chain, at a few warps per
// scheduler; two threads per item cut the chain in two, and the record takes
// two dependent loads out of it.  The class alone, 524,288 + 2,097,152 items
// (a quarter of the large workload): 37 -> 22 us a launch.
//
// List entries are loaded two together; with EARLY (sims that do not fill the
// device) four, the first of them while the bonds' terms are formed, which
// costs registers the larger sims want.
template <bool BATCH, bool EARLY, int T>
__device__ __forceinline__ void relax_bonded_block(const ScParams &P0, const RelaxArgs &A, int b, int n,
                                                   float4 *s_av) {
    constexpr int G = EARLY ? 4 : 2;
    // warps in pairs: one turns, the other moves the pair's 32 items (the
    // first half of a block's warps turns, so its schedulers hold both kinds)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pair = warp % (T / 64);
    const bool turner = warp < T / 64;
    const int slot = pair * 32 + lane;
    // The plan ranks every 256 items by their bonds, so its 32-item groups
    // come as eight weights: one-pair blocks take all the heaviest groups
    // first, and no launch ends on one (vesicle at 1/16: 134 us a launch in
    // plan order, 114 us so).
    const int ranked = (n + SC_THREADS - 1) / SC_THREADS;
    const int t = T == 64 ? (b % ranked * 8 + b / ranked) * 32 + lane : b * (T / 2) + slot;
    const uint4 r = t < n ? A.bondRec[t] : make_uint4(0xffffffffu, 0, 0, 0);
    const int i = (int)r.x;
    const bool polar = (r.w >> 5) & 1u;
    sc_f3 up = sc_zero3(), towards = sc_zero3(), newPos = sc_zero3();
    float phobSum = 0.0f;
    if (i >= 0) {
        const int nm = (int)(r.w & 15u), c = (int)((r.w >> 8) & 0xffu);
        const float4 p4 = A.pos[i], v4 = A.velIn[i], r4 = A.rotIn[i], a4 = A.avIn[i];
        const int4 in = A.info[i];
        ScParams P = P0;
        rep_apply<BATCH>(P, in.w);
        BondSelf S;
        S.ppos = sc_make_f3(p4.x, p4.y, p4.z);
        S.prad = p4.w;
        S.pvel = sc_make_f3(v4.x, v4.y, v4.z);
        S.prot = sc_make_f4(r4.x, r4.y, r4.z, r4.w);
        S.pav = sc_make_f4(a4.x, a4.y, a4.z, a4.w);
        const Imager IM(P, S.ppos, SC_BINNED_P);
        const uint32_t *__restrict__ myMatch = A.match + (size_t)i * SC_MAX_ACTIVE_INTERACTIONS;
        const int *__restrict__ myBonds = A.bonds + (size_t)i * 24;
        auto pair_of = [&](int m, BondPair &b) {
            const uint32_t me = m == 0 ? r.y : myMatch[m];
            const int j = (int)(me & SC_PP_INDEX), k = (int)(me >> 29);
            b.it = m == 0 ? (int)r.z : myBonds[3 * k];
            if (!bond_turns(b.it)) return false;
            b.fwd = m == 0 ? (r.w >> 4) & 1u : myBonds[3 * k + 1] == SC_INTERACTION_GROUP_FORWARD;
            const int4 tin = A.info[j];
            const float4 t4 = A.pos[j];
            b.tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
            b.trad = t4.w;
            b.trot = ld4(A.rotIn, j);
            b.tav = ld4(A.avIn, j);
            b.tvel = ld3(A.velIn, j);
            b.o1 = p_order(in.y, in.x, tin.y, tin.x);
            b.o2 = p_order(tin.y, tin.x, in.y, in.x);
            return true;
        };
        up = sc_rotate(sc_up(), S.prot);
        S.nextUp = sc_rotate(up, S.pav);
        if (turner) {
            sc_f4 dAV = sc_qid();
            for (int m = 0; m < nm; m++) {
                BondPair b;
                if (!pair_of(m, b)) continue;
                dAV = sc_slerp(dAV, bond_target(P, S, b), 0.9f * b.trad / (S.prad + b.trad));
            }
            const sc_f4 pav = sc_qmul(sc_slerp(sc_qid(), dAV, 1.0f / fmaxf((float)(r.w >> 16), 1.0f)), S.pav);
            if (polar) s_av[slot] = make_float4(pav.x, pav.y, pav.z, pav.w);
            else st4(A.avOut, i, pav);
        } else {
            const sc_f3 ppv = S.ppos + S.pvel;
            auto load = [&](int k0, uint32_t (&e)[G], float4 (&g)[G], float4 (&tv)[G]) {
                const bool kept = k0 < SC_GEO_PP;
#pragma unroll
                for (int q = 0; q < G; q++)
                    e[q] = k0 + q < c ? A.L.list[sc_list_at(SC_LIST_PP, i, k0 + q)] : 0u;
#pragma unroll
                for (int q = 0; q < G; q++) {
                    g[q] = make_float4(0, 0, 0, 0);
                    tv[q] = g[q];
                    if (e[q] & SC_PP_COLLIDE)
                        g[q] = kept ? A.geo[sc_list_at(SC_GEO_PP, i, k0 + q)] : A.pos[(int)(e[q] & SC_PP_INDEX)];
                    if (e[q] & (SC_PP_COLLIDE | SC_PP_POLAR)) tv[q] = A.velIn[(int)(e[q] & SC_PP_INDEX)];
                }
            };
            uint32_t e0[G];
            float4 g0[G], tv0[G];
            if (EARLY) load(0, e0, g0, tv0);
            // 1. the bonds' velocity terms: the first stays in registers (most
            // bonded items have one), the rest go to a per-thread array
            sc_f3 V0 = sc_zero3(), V[SC_MAX_ACTIVE_INTERACTIONS - 1];
            sc_f4 pdbg = sc_make_f4(0, 0, 0, 0);
            bool dbgTouched = false;
            int nt = 0;
            for (int m = 0; m < nm; m++) {
                BondPair b;
                if (!pair_of(m, b)) continue;
                sc_f3 dd = sc_zero3();
                const sc_f3 dv = bond_velocity(P, S, b, &dd);
                if (b.it == SC_INTERACTION_TYPE_CHAIN) {
                    if (!dbgTouched) {
                        pdbg = ld4(A.dbg, i);
                        dbgTouched = true;
                    }
                    pdbg.x = (float)((double)pdbg.x + (double)dd.x * (1.0 - (double)0.9f));
                    pdbg.y = (float)((double)pdbg.y + (double)dd.y * (1.0 - (double)0.9f));
                    pdbg.z = (float)((double)pdbg.z + (double)dd.z * (1.0 - (double)0.9f));
                }
                if (nt == 0) V0 = dv;
                else V[nt - 1] = dv;
                nt++;
            }
            if (dbgTouched) st4(A.dbg, i, pdbg);
            // 2. every velocity term in the reference's order
            sc_f3 dV = sc_zero3(), phobPos = sc_zero3();
            int ut = 0, mi = 0;
            auto walk = [&](int k0, const uint32_t (&e)[G], const float4 (&g)[G], const float4 (&tv)[G]) {
                const bool kept = k0 < SC_GEO_PP;
#pragma unroll
                for (int q = 0; q < G; q++) {
                    const uint32_t fl = e[q];
                    const int j = (int)(fl & SC_PP_INDEX);
                    if (fl & SC_PP_POLAR) {
                        // dynamics.cuh:478-582
                        const float4 t4 = A.pos[j];
                        const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
                        const float trad = t4.w;
                        const sc_f3 tvel = sc_make_f3(tv[q].x, tv[q].y, tv[q].z);
                        sc_f3 nextTup = sc_rotate(sc_rotate(sc_up(), ld4(A.rotIn, j)), S.pav);
                        sc_f3 pPV = -S.nextUp * S.prad + S.ppos + S.pvel;
                        sc_f3 tpPV = -nextTup * trad + tpos + tvel;
                        float Lr = length(tpPV - pPV) / (S.prad + trad);
                        float attr = sc_polar_attr(Lr);
                        dV += (tpPV - pPV) * 0.05f * attr * 1.0f;
                        float pap = sc_powf(fminf(1.0f / fmaxf(Lr, 1e-6f), 10.0f) / 10.0f, 0.2f);
                        phobSum += pap;
                        phobPos += tpPV * pap;
                    }
                    if (fl & SC_PP_PARTNER) {
                        // this neighbour's bond matches are the next ones in order
                        for (; mi < nm; mi++) {
                            const uint32_t me = mi == 0 ? r.y : myMatch[mi];
                            if ((int)(me & SC_PP_INDEX) != j) break;
                            const int it = mi == 0 ? (int)r.z : myBonds[3 * (int)(me >> 29)];
                            if (bond_turns(it)) {
                                dV += ut == 0 ? V0 : V[ut - 1];
                                ut++;
                            }
                        }
                    }
                    if (fl & SC_PP_COLLIDE)
                        dV += collide_term(kept ? g[q] : collide_geo(IM, S.ppos, S.prad, g[q]), tv[q], ppv, S.prad);
                }
            };
            for (int k0 = 0; k0 < c; k0 += G) {
                if (EARLY) {
                    if (k0 > 0) load(k0, e0, g0, tv0);
                    walk(k0, e0, g0, tv0);
                } else {
                    uint32_t e[G];
                    float4 g[G], tv[G];
                    load(k0, e, g, tv);
                    walk(k0, e, g, tv);
                }
            }
            const sc_f3 nv = S.pvel + dV / fmaxf((float)(r.w >> 16), 1.0f);
            st3(A.velOut, i, nv, v4.w);
            if (A.age == 0) A.rotOut[i] = r4;
            if (phobSum > 0.0f) {
                newPos = S.ppos + nv;
                towards = normalize(phobPos / phobSum - newPos);
            }
        }
    }
    __syncthreads();
    if (!turner && i >= 0 && polar) {
        const float4 q = s_av[slot];
        sc_f4 pav = sc_make_f4(q.x, q.y, q.z, q.w);
        if (phobSum > 0.0f) pav = sc_slerp(pav, sc_quat_from_to(-up, towards), 0.2f);
        st4(A.avOut, i, pav);
    }
    __syncthreads();  // s_av is reused by the block's next items
}

// ---- dynamics.cuh:405-822 relax ------------------------------------------------
// The classes write disjoint items and read only the input buffers, so they
// run side by side.  CLS = SC_RELAX_ALL: one grid over all of them, its blocks
// taking the bonded class first (the longest chains), then the polar and plain
// classes and the items left to the scan, so the short classes run while the
// long one does.  CLS = 0, 1, 2: one class (0 with the scan's items), at the
// occupancy its registers allow.
//
// The line between them is whether the particles fill the device
// (forkClasses in sc_sim.cu): 4,096 + 8,192 items take 1.95 ms a step with a
// launch per class in turn and 1.2 ms with one launch; 2,097,152 + 8,388,608
// take 27.5 ms with a kernel per class and 30.7 ms with one launch, whose two
// blocks per SM starve the plain and polar items.
#define SC_RELAX_ALL 3
#define SC_RELAX_ALL_LANES 4   // the same with SC_POLAR_LANES threads per polar item
//
// The bonded kernel's blocks are one pair of warps: an item's time goes with
// its bonds (a lattice complex's particles hold up to seven), and in blocks of
// four pairs the others' registers waited for the longest (vesicle at 1/16:
// 141 us a launch so, 134 us in pairs).  Ten pairs, three and four blocks per SM:
// batch of 24 replicas, two steps 11.3 ms at 2 / 4 / 5 blocks of 256, 11.0 ms
// so; sub-iteration of the large workload 170 us at 3 / 3 / 3, 181 us at
// 2 / 5 / 6.
__host__ __device__ constexpr int relax_threads(int cls) { return cls == 0 ? 64 : SC_THREADS; }
template <int CLS, bool BATCH>
__global__ void __launch_bounds__(relax_threads(CLS), CLS == 0 ? 10 : CLS == 1 ? 3 : CLS == 2 ? 4 : 2)
    k_relax(ScParams P, RelaxArgs A) {
    constexpr bool ALL = CLS >= SC_RELAX_ALL, B0 = CLS == 0 || ALL, B1 = CLS == 1 || ALL, B2 = CLS == 2 || ALL;
    constexpr int T = relax_threads(CLS);
    __shared__ float4 s_av[B0 ? T / 2 : 1];
    const int n0 = B0 ? A.classCount[0] : 0, n1 = B1 ? A.classCount[1] : 0, n2 = B2 ? A.classCount[2] : 0,
              nv = B0 ? *A.ovfCount : 0;
    constexpr int PL = CLS == SC_RELAX_ALL_LANES ? SC_POLAR_LANES : 1;   // threads per polar item
    const int b0 = T == 64 ? (n0 + SC_THREADS - 1) / SC_THREADS * 8 : (n0 + T / 2 - 1) / (T / 2),
              b1 = b0 + (n1 * PL + T - 1) / T, b2 = b1 + (n2 + T - 1) / T, b3 = b2 + (nv + T - 1) / T;
    for (int b = blockIdx.x; b < b3; b += gridDim.x) {
        if (B0 && b < b0) {
            relax_bonded_block<BATCH, CLS == SC_RELAX_ALL_LANES, T>(P, A, b, n0, s_av);
        } else if (B1 && b < b1) {
            const int t = (b - b0) * T + threadIdx.x;
            if (PL > 1) {
                if (t < n1 * PL) relax_polar_lanes<BATCH>(P, A, A.classIdx[(size_t)A.L.cap + t / PL]);
            } else if (t < n1) {
                relax_polar<BATCH>(P, A, A.classIdx[(size_t)A.L.cap + t]);
            }
        } else if (B2 && b < b2) {
            const int t = (b - b1) * T + threadIdx.x;
            if (t < n2) relax_plain<BATCH>(P, A, A.classIdx[2 * (size_t)A.L.cap + t]);
        } else if (B0) {
            const int t = (b - b2) * T + threadIdx.x;
            if (t < nv) {
                const int i = A.ovf[t];
                const int4 in = A.info[i];
                ScParams Q = P;
                rep_apply<BATCH>(Q, in.w);
                if (in.z & SC_ACTIVE) relax_scan_item(Q, A, i, in, A.velIn[i], A.rotIn[i], A.avIn[i]);
            }
        }
    }
}

// (float)((double)(rp + rt) + 0.8 * (double)rp) (metabolites.cuh:198,237,324),
// recomputed only when the partner radius changes.
struct CollisionDistCache {
    float rt = 0.0f, cd = 0.0f;
    sc_sqrt_le le;
    bool valid = false;
    __device__ __forceinline__ float get(float rp, float r) {
        if (!valid || !(r == rt)) {
            rt = r;
            valid = true;
            cd = sc_coll_dist(rp, r);
            le = sc_sqrt_le_make(cd);
        }
        return cd;
    }
    // sc_norm3(delta) <= the collision distance of (rp, r), the reference's
    // test (metabolites.cuh:193-203), mostly without the square root
    __device__ __forceinline__ bool collides(float rp, float r, sc_f3 delta) {
        get(rp, r);
        return sc_sqrt_le_test(le, sc_normsq3(delta));
    }
};

// ---- metabolites.cuh:140-264 relaxMetabolicParticles ----------------------
// List: per metabolic item, cell by cell, the colliding metabolic items then
// the colliding lipids (SC_M_FROM_P), as the reference's loops visit them.
// The M list of metabolic item i, written at position i of `list`.
// The colliding metabolic items, then lipids, of each neighbour cell of
// metabolic item i in visiting order, each handed to sink(j, fromP, t4) (j
// the neighbour's slot, t4 its position and radius; the collision distance is
// then cached in cm / cp).
template <class Sink>
__device__ __forceinline__ void scan_m_item(const ScParams &P, const uint32_t *__restrict__ cellStartM,
                                            const uint32_t *__restrict__ cellStartP, int i,
                                            const float4 *__restrict__ mpos, const int4 *__restrict__ minfo,
                                            const float4 *__restrict__ ppos_, const int4 *__restrict__ pinfo,
                                            const Imager &IM, sc_f3 pp, float prad, CollisionDistCache &cm,
                                            CollisionDistCache &cp, Sink &&sink) {
    const float lim = P.maxInt;
    cells27(P, pp, reach(P, pp, lim, SC_BINNED_M | SC_BINNED_P), [&](uint32_t key) {
        for (uint32_t j = cellStartM[key], e = cellStartM[key + 1]; j < e; j++) {
            if ((int)j == i || !active_m(P, minfo, (int)j)) continue;
            float4 t4 = mpos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) continue;
            if (cm.collides(prad, t4.w, delta)) sink(j, false, t4);
        }
        for (uint32_t j = cellStartP[key], e = cellStartP[key + 1]; j < e; j++) {
            if (!active_lipid(P, pinfo, (int)j)) continue;
            float4 t4 = ppos_[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) continue;
            if (cp.collides(prad, t4.w, delta)) sink(j, true, t4);
        }
    });
}

// The M list's candidates in one array: cell by cell, the metabolic items'
// positions, then the particles' (comb_start gives a cell's first), so that the
// reference's visiting order -- per cell, metabolic items then lipids -- is one
// run per column.  w holds the slot (SC_M_FROM_P for particles); what is no
// candidate (particles other than active lipids, inactive items) lies at
// infinity, which no cube reaches.  A radius other than its type's sets
// SC_M_ODD: the tests of all others need no radius.
#define SC_M_ODD 0x40000000u
#define SC_M_SLOT 0x3FFFFFFFu
__device__ __forceinline__ float type_radius(const ScParams &P, int type) {
    return type < P.nTypes ? P.types[type].radius : 0.0f;
}
struct CombStart {
    const uint32_t *__restrict__ m, *__restrict__ p;
    __device__ __forceinline__ uint32_t operator()(uint32_t key) const { return m[key] + p[key]; }
};
__global__ void __launch_bounds__(SC_THREADS) k_combine(ScParams P, const uint32_t *__restrict__ keysM,
                                                        const uint32_t *__restrict__ keysP, CombStart cs,
                                                        const float4 *__restrict__ mpos, const int4 *__restrict__ minfo,
                                                        const float4 *__restrict__ ppos_, const int4 *__restrict__ pinfo,
                                                        float4 *__restrict__ comb) {
    const long long total = (long long)P.N + P.Nm;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const bool m = t < P.Nm;
        const int j = (int)(m ? t : t - P.Nm);
        const uint32_t key = m ? keysM[j] : keysP[j];
        if (key >= P.cells) continue;   // in no cell
        const size_t at = m ? (size_t)j + cs.p[key] : (size_t)j + cs.m[key + 1];
        if (at >= (size_t)total) continue;
        float4 q = m ? mpos[j] : ppos_[j];
        if (!(m ? active_m(P, minfo, j) : active_lipid(P, pinfo, j))) q.x = q.y = q.z = INFINITY;
        const bool odd = !(q.w == type_radius(P, m ? SC_PARTICLE_TYPE_METABOLIC : SC_PARTICLE_TYPE_LIPID));
        q.w = __uint_as_float((uint32_t)j | (m ? 0u : SC_M_FROM_P) | (odd ? SC_M_ODD : 0u));
        comb[at] = q;
    }
}

__device__ __forceinline__ void build_m_item(const ScParams &P, ScanWords &W, CombStart cs,
                                             const float4 *__restrict__ comb, int i,
                                             const float4 *__restrict__ mpos, const float4 *__restrict__ ppos_,
                                             uint32_t *list, int &c) {
    const float4 p4 = mpos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
    // the collision distances (metabolites.cuh:193-203, 230-240) to the two kinds of candidates
    const sc_sqrt_le leM = sc_sqrt_le_make(sc_coll_dist(p4.w, type_radius(P, SC_PARTICLE_TYPE_METABOLIC))),
                     leP = sc_sqrt_le_make(sc_coll_dist(p4.w, type_radius(P, SC_PARTICLE_TYPE_LIPID)));
    const int limit = min(SC_LIST_M, P.listLimit);
    const float lim = P.maxInt;
    const bool wrap = IM.wrap;
    uint32_t *out = list + sc_list_at(SC_LIST_M, i, 0);
    scan_words(P, W, comb, cs, pp, reach(P, pp, lim, SC_BINNED_M | SC_BINNED_P), lim,
               scan_mixed(P, IM, SC_BINNED_M | SC_BINNED_P), [&](int, float4 t) {
        const uint32_t e = __float_as_uint(t.w);
        if ((e & ~SC_M_ODD) == (uint32_t)i) return;
        sc_f3 delta;
        if (wrap) {
            delta = IM(sc_make_f3(t.x, t.y, t.z)) - pp;
            if (outside_cube(delta, lim)) return;
        } else {
            delta = sc_make_f3(t.x, t.y, t.z) - pp;
        }
        const bool fromP = (e & SC_M_FROM_P) != 0;
        const float x = sc_normsq3(delta);
        bool hit;
        if (e & SC_M_ODD) {
            hit = sqrtf(x) <= sc_coll_dist(p4.w, (fromP ? ppos_ : mpos)[e & SC_M_SLOT].w);
        } else {
            sc_sqrt_le le;
            le.d = fromP ? leP.d : leM.d;
            le.lo = fromP ? leP.lo : leM.lo;
            le.hi = fromP ? leP.hi : leM.hi;
            hit = sc_sqrt_le_test(le, x);
        }
        if (hit) {
            if (c < limit) *out = e & ~SC_M_ODD;
            out += 32;
            c++;
        }
    });
}

// The full pair lists of the metabolic items whose list overflowed (listed
// by k_build_m with their pair counts): each takes a contiguous region of
// the overflow pool by atomicAdd and writes its pairs there in visiting order,
// 16-byte entries with the frozen geometry as the main pool's; an item the
// pool has no room for keeps offset -1 (it scans its neighbourhood).  The
// demand is counted in full for the pool's growth at the next synchronisation.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_build_m_ovf(
    ScParams P0, const uint32_t *__restrict__ cellStartM, const uint32_t *__restrict__ cellStartP,
    const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, const float4 *__restrict__ ppos_,
    const int4 *__restrict__ pinfo, const int *__restrict__ ovf, const int *__restrict__ ovfCount,
    const int *__restrict__ ovfN, long long *__restrict__ ovfOff, uint4 *__restrict__ pool, long long cap,
    unsigned long long *__restrict__ demand) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < *ovfCount; t += gridDim.x * blockDim.x) {
        const int i = ovf[t], n = ovfN[t];
        const unsigned long long base = n > 0 ? atomicAdd(demand, (unsigned long long)n) : 0ull;
        if (n <= 0 || base + (unsigned long long)n > (unsigned long long)cap) {
            ovfOff[t] = -1;
            continue;
        }
        ovfOff[t] = (long long)base;
        ScParams P = P0;
        rep_apply<BATCH>(P, minfo[i].w);
        const float4 p4 = mpos[i];
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
        const float prad = p4.w;
        CollisionDistCache cm, cp;
        uint4 *out = pool + base;
        int k = 0;
        scan_m_item(P, cellStartM, cellStartP, i, mpos, minfo, ppos_, pinfo, IM, pp, prad, cm, cp,
                    [&](uint32_t j, bool fromP, float4 t4) {
                        if (k >= n) return;
                        const sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
                        const sc_f3 nd = normalize(tpos - pp);
                        const float cd = fromP ? cp.get(prad, t4.w) : cm.get(prad, t4.w);
                        const sc_f3 a = tpos - nd * cd;
                        out[k++] = make_uint4(fromP ? (j | SC_M_FROM_P) : j, __float_as_uint(a.x),
                                              __float_as_uint(a.y), __float_as_uint(a.z));
                    });
    }
}

// A pool position for the pairs of one count-ordered list position: the
// block's items are ranked by count, each warp takes a region of
// (its longest list) x 32 entries of the pool, and a list that does not fit
// its capacity, or every list of a block the pool has no room for, is marked
// overflowed (cnt = INT_MAX; listed in `ovf` when given).  Returns the item,
// how many pairs to write and where its first one goes (entry k at
// out[32 k]).  With `items`, thread t of the block stands for item
// items[b0 + t] (a compacted list) and perm holds those items.
template <class T>
struct PoolSlot {
    int i, n;
    T *out;
};
template <int K, class T>
__device__ __forceinline__ PoolSlot<T> pool_take(const ScParams &P, int block, bool valid, int c, T *__restrict__ pool,
                                              long long poolCap, unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff,
                                              int *__restrict__ cnt, int *__restrict__ perm, int cap,
                                              int *__restrict__ ovf, int *__restrict__ ovfCount,
                                              const int *__restrict__ items = nullptr, int *__restrict__ ovfN = nullptr) {
    __shared__ int s_n[SC_THREADS / 32];
    __shared__ long long s_base;
    const int b0 = block * SC_THREADS, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int src, cs;
    count_rank<K>(valid, c, &src, &cs);
    const int limit = min(K, P.listLimit);
    bool ovfl = cs > limit;
    int n = ovfl ? 0 : max(cs, 0);
    // the warp's longest stored list (overflowed lists rank first but store nothing)
    const int wmax = __reduce_max_sync(0xffffffffu, n);
    if (lane == 0) s_n[warp] = wmax;
    __syncthreads();
    if (t == 0) {
        int total = 0;
        for (int w = 0; w < SC_THREADS / 32; w++) total += s_n[w] * 32;
        // 64-bit demand: it keeps counting what blocks ask for past the pool
        const unsigned long long base = total ? atomicAdd(poolUsed, (unsigned long long)total) : 0ull;
        s_base = base + (unsigned long long)total <= (unsigned long long)poolCap ? (long long)base : -1ll;
    }
    __syncthreads();
    if (s_base < 0 && cs > 0) {
        ovfl = true;
        n = 0;
    }
    long long off = s_base;
    for (int w = 0; w < warp; w++) off += s_n[w] * 32;
    const int g = b0 + t;
    if (g < cap) {
        perm[g] = cs >= 0 ? (items ? items[b0 + src] : b0 + src) : -1;
        cnt[g] = ovfl ? INT_MAX : max(cs, 0);
        if (lane == 0) warpOff[g >> 5] = s_base < 0 ? 0 : off;
    }
    if (ovfl && ovf) {
        const int t = atomicAdd(ovfCount, 1);
        ovf[t] = b0 + src;
        if (ovfN) ovfN[t] = max(cs, 0);  // its full pair count
    }
    PoolSlot<T> r;
    r.i = cs >= 0 && items ? items[b0 + src] : b0 + src;
    r.n = n;
    r.out = pool + (n ? off : 0) + lane;
    return r;
}

// M pairs with their frozen geometry.  Positions do not change between the
// sort and applyVelocities, so for every listed pair the part of the
// reference's velocity term that depends on positions only,
// A = tpos - normalize(tpos - pos) * collisionDistance (metabolites.cuh:
// 196-203, 235-242), is the same in every relaxation sub-iteration.  It is
// evaluated here, once per step, and each sub-iteration adds
// ((A + tvel) - (pos + vel)) * 0.9 * weight: A is exactly the float3 the
// reference's expression evaluates first, so sums and rounding are its own.
// Layout: the pairs of a warp's 32 positions share one region of the pool,
// entry k of lane l at warpOff[w] + 32 k + l, 16 bytes {neighbour | kind,
// A.x, A.y, A.z}; a region is sized by the warp's longest stored list.  An
// overflowed item, or every item of a block the pool has no room for, is
// listed in `ovf` for the scan.
template <bool BATCH>
__device__ __forceinline__ void emit_m_pairs(const ScParams &P0, int block, bool valid, int c, const uint32_t *scratch,
                                             const int4 *__restrict__ minfo,
                                             const float4 *__restrict__ mpos, const float4 *__restrict__ ppos_,
                                             uint4 *__restrict__ pool, long long poolCap, unsigned long long *__restrict__ poolUsed,
                                             long long *__restrict__ warpOff, int *__restrict__ cnt, int *__restrict__ perm,
                                             int cap, int *__restrict__ ovf, int *__restrict__ ovfCount,
                                             int *__restrict__ ovfN) {
    const PoolSlot<uint4> S = pool_take<SC_LIST_M>(P0, block, valid, c, pool, poolCap, poolUsed, warpOff, cnt, perm, cap, ovf,
                                                   ovfCount, nullptr, ovfN);
    if (S.n == 0) return;
    const int i = S.i;
    ScParams P = P0;
    rep_apply<BATCH>(P, minfo[i].w);
    const float4 p4 = mpos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
    const float prad = p4.w;
    CollisionDistCache cm, cp;
    // four pairs' entries, then their positions, in flight together
    for (int k0 = 0; k0 < S.n; k0 += 4) {
        uint32_t e[4];
        float4 t4[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e[q] = k0 + q < S.n ? scratch[sc_list_at(SC_LIST_M, i, k0 + q)] : 0u;
#pragma unroll
        for (int q = 0; q < 4; q++)
            t4[q] = k0 + q < S.n ? ((e[q] & SC_M_FROM_P) ? ppos_ : mpos)[e[q] & SC_M_INDEX] : p4;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (k0 + q >= S.n) break;
            const sc_f3 tpos = IM(sc_make_f3(t4[q].x, t4[q].y, t4[q].z));
            const sc_f3 nd = normalize(tpos - pp);
            const float cd = (e[q] & SC_M_FROM_P) ? cp.get(prad, t4[q].w) : cm.get(prad, t4[q].w);
            const sc_f3 a = tpos - nd * cd;
            S.out[(size_t)(k0 + q) * 32] = make_uint4(e[q], __float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z));
        }
    }
}

// The lean form of the same pool (ScParams.metabLean): 4-byte entries
// {neighbour | kind} only, in the same count-ordered warp regions; the
// relaxation re-evaluates the geometry from the neighbour's position each
// sub-iteration (a 16-byte gather that nearby items share in L1 / L2, and a
// square root and a division per pair) instead of streaming 12 more bytes
// per pair from HBM.
__device__ __forceinline__ void emit_m_pairs_lean(const ScParams &P, int block, bool valid, int c, const uint32_t *scratch,
                                                  uint32_t *__restrict__ pool, long long poolCap,
                                                  unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff,
                                                  int *__restrict__ cnt, int *__restrict__ perm, int cap,
                                                  int *__restrict__ ovf, int *__restrict__ ovfCount,
                                                  int *__restrict__ ovfN) {
    const PoolSlot<uint32_t> S = pool_take<SC_LIST_M>(P, block, valid, c, pool, poolCap, poolUsed, warpOff, cnt, perm, cap,
                                                      ovf, ovfCount, nullptr, ovfN);
    for (int k = 0; k < S.n; k++) S.out[(size_t)k * 32] = scratch[sc_list_at(SC_LIST_M, S.i, k)];
}

template <bool LEAN, bool BATCH>
__device__ __forceinline__ void build_m_block(
    const ScParams &P0, ScanWords &W, int block, CombStart cs, const float4 *__restrict__ comb,
    const int *__restrict__ nActivePtr, const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, const float4 *__restrict__ ppos_, uint32_t *__restrict__ pool, long long poolCap,
    unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff, uint32_t *scratch,
    int *__restrict__ cnt, int *__restrict__ perm, int cap, int *__restrict__ ovf, int *__restrict__ ovfCount,
    int *__restrict__ ovfN) {
    const int i = block * SC_THREADS + threadIdx.x;
    const bool valid = i < *nActivePtr;
    int c = 0;
    if (valid) {
        const int4 mi = minfo[i];
        ScParams P = P0;
        rep_apply<BATCH>(P, mi.w);
        if (mi.z & SC_ACTIVE) build_m_item(P, W, cs, comb, i, mpos, ppos_, scratch, c);
    }
    if (LEAN)
        emit_m_pairs_lean(P0, block, valid, c, scratch, pool, poolCap, poolUsed, warpOff, cnt, perm, cap, ovf, ovfCount,
                          ovfN);
    else
        emit_m_pairs<BATCH>(P0, block, valid, c, scratch, minfo, mpos, ppos_, reinterpret_cast<uint4 *>(pool), poolCap,
                            poolUsed, warpOff, cnt, perm, cap, ovf, ovfCount, ovfN);
}
template <bool LEAN, bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, 4) k_build_m(
    ScParams P0, CombStart cs, const float4 *__restrict__ comb, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, const float4 *__restrict__ ppos_, uint32_t *__restrict__ pool, long long poolCap,
    unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff, uint32_t *scratch,
    int *__restrict__ cnt, int *__restrict__ perm, int cap, int *__restrict__ ovf, int *__restrict__ ovfCount,
    int *__restrict__ ovfN) {
    __shared__ ScanWords W;
    build_m_block<LEAN, BATCH>(P0, W, blockIdx.x, cs, comb, nActivePtr, mpos, minfo, ppos_, pool, poolCap, poolUsed,
                               warpOff, scratch, cnt, perm, cap, ovf, ovfCount, ovfN);
}


struct RelaxMArgs {
    const uint32_t *__restrict__ cellStartM, *__restrict__ cellStartP;
    const int *__restrict__ nActivePtr;
    const float4 *__restrict__ mpos;
    const int4 *__restrict__ minfo;
    PairList<SC_LIST_M> L;
    const float4 *__restrict__ mvelIn;
    float4 *__restrict__ mvelOut;
    const float4 *__restrict__ ppos;
    const int4 *__restrict__ pinfo;
    const float4 *__restrict__ pvel;
    const uint4 *__restrict__ pool;     // pairs with their geometry (emit_m_pairs)
    const long long *__restrict__ warpOff;
    // the items whose list overflowed (k_build_m), with their pair counts and
    // regions of the overflow pool (ovfOff null: none is kept whole)
    const int *__restrict__ ovf, *__restrict__ ovfCount, *__restrict__ ovfN;
    const long long *__restrict__ ovfOff;
    const uint4 *__restrict__ ovfPool;
    // launches since the sort: from the second on both velocity buffers hold
    // the inactive items' velocities
    int age;
};

// The contribution of one colliding neighbour (a metabolic item, or a lipid
// with twice the weight) to dV and w, metabolites.cuh:196-203 / 235-242.
__device__ __forceinline__ void metab_pair(const Imager &IM, sc_f3 pp, sc_f3 ppv, float4 t4, float4 tv, float cd,
                                           bool fromP, sc_f3 &dV, float &w) {
    sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
    sc_f3 nd = normalize(tpos - pp);
    float k = fromP ? 2.0f : 1.0f;
    w += k;
    dV += (tpos - nd * cd + sc_make_f3(tv.x, tv.y, tv.z) - ppv) * 0.9f * k;
}

// One pair's neighbour velocity: a metabolic item's, or a lipid's.
__device__ __forceinline__ float4 metab_pair_vel(const RelaxMArgs &A, uint32_t e) {
    return ((e & SC_M_FROM_P) ? A.pvel : A.mvelIn)[e & SC_M_INDEX];
}

// One pair of a pool: its precomputed geometry and the neighbour's current
// velocity (metabolites.cuh:196-203 / 235-242).
__device__ __forceinline__ void metab_pool_term(uint4 E, float4 tv, sc_f3 ppv, sc_f3 &dV, float &w) {
    const float kw = (E.x & SC_M_FROM_P) ? 2.0f : 1.0f;
    const sc_f3 a = sc_make_f3(__uint_as_float(E.y), __uint_as_float(E.z), __uint_as_float(E.w));
    w += kw;
    dV += (a + sc_make_f3(tv.x, tv.y, tv.z) - ppv) * 0.9f * kw;
}

// An item whose list overflowed: the reference's loops over the 27 cells.
template <bool BATCH>
__device__ __noinline__ void relax_metab_scan_item(const ScParams &P0, const RelaxMArgs &A, int i) {
    if (i < 0) return;
    const int4 mi = A.minfo[i];
    if (!(mi.z & SC_ACTIVE)) return;
    ScParams P = P0;
    rep_apply<BATCH>(P, mi.w);
    float4 v4 = A.mvelIn[i];
    float4 p4 = A.mpos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
    const float prad = p4.w;
    const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = pp + pv;
    sc_f3 dV = sc_zero3();
    float w = 0.0f;
    CollisionDistCache cm, cp;
    const float lim = P.maxInt;
    cells27(P, pp, reach(P, pp, lim, SC_BINNED_M | SC_BINNED_P), [&](uint32_t key) {
        for (uint32_t j = A.cellStartM[key], e = A.cellStartM[key + 1]; j < e; j++) {
            if ((int)j == i) continue;
            if (!active_m(P, A.minfo, (int)j)) continue;
            float4 t4 = A.mpos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) continue;
            if (cm.collides(prad, t4.w, delta))
                metab_pair(IM, pp, ppv, t4, A.mvelIn[j], cm.get(prad, t4.w), false, dV, w);
        }
        for (uint32_t j = A.cellStartP[key], e = A.cellStartP[key + 1]; j < e; j++) {
            if (!active_lipid(P, A.pinfo, (int)j)) continue;
            float4 t4 = A.ppos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) continue;
            if (cp.collides(prad, t4.w, delta))
                metab_pair(IM, pp, ppv, t4, A.pvel[j], cp.get(prad, t4.w), true, dV, w);
        }
    });
    st3(A.mvelOut, i, pv + dV / fmaxf(w, 1.0f), v4.w);
}

// Lists of the overflow pool longer than this are walked by a whole warp,
// shorter ones by one thread (both in relax_metab_overflow): a list that
// overflowed because the main pool had no room for its block fits the list
// capacity, one that outgrew the capacity (a wall pile's) holds hundreds to
// thousands of pairs.  With the list capacity capped (pair_list_limit, the
// tests' way into the overflow paths) the bound is four times the cap, so
// ordinary lists take both walks.
#define SC_POOL_WARP_MIN SC_LIST_M
__device__ __forceinline__ int pool_warp_min(const ScParams &P) {
    return P.listLimit < SC_POOL_WARP_MIN / 4 ? 4 * P.listLimit : SC_POOL_WARP_MIN;
}

// The items whose list overflowed, by `blocks` blocks of which this is block
// `blk`.  First a thread each: an item the overflow pool had no room for
// scans its neighbourhood; one whose region there is short walks it as
// k_relax_metab walks the main pool.  Then a warp for each longer region,
// warp-stride so the long lists of a wall pile spread over the device: the
// lanes load 32 entries and the neighbours' velocities at once and each forms
// its pair's term and weight; lanes 0-2 add the terms' components and lane 3
// the weights in list order from shared memory -- the sums a thread walking
// the list forms, at one gather latency per 32 pairs.
#define SC_TERM_ROW 5   // x, y, z, weight (odd row length: no bank conflicts)
template <bool BATCH>
__device__ __noinline__ void relax_metab_overflow(const ScParams &P, const RelaxMArgs &A, int blk, int blocks,
                                                  float (*sTerm)[32][SC_TERM_ROW]) {
    const int nOvf = *A.ovfCount, warpMin = pool_warp_min(P);
    for (int t = blk * SC_THREADS + threadIdx.x; t < nOvf; t += blocks * SC_THREADS) {
        const int i = A.ovf[t];
        const long long off = A.ovfOff ? A.ovfOff[t] : -1;
        if (off < 0) {
            relax_metab_scan_item<BATCH>(P, A, i);
            continue;
        }
        const int n = A.ovfN[t];
        if (i < 0 || n > warpMin || !(A.minfo[i].z & SC_ACTIVE)) continue;
        const float4 v4 = A.mvelIn[i], p4 = A.mpos[i];
        const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
        const sc_f3 ppv = sc_make_f3(p4.x, p4.y, p4.z) + pv;
        sc_f3 dV = sc_zero3();
        float w = 0.0f;
        const uint4 *__restrict__ e = A.ovfPool + off;
        for (int k0 = 0; k0 < n; k0 += 4) {
            uint4 E[4];
            float4 tv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) E[q] = k0 + q < n ? e[k0 + q] : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < 4; q++) tv[q] = k0 + q < n ? metab_pair_vel(A, E[q].x) : make_float4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (k0 + q < n) metab_pool_term(E[q], tv[q], ppv, dV, w);
        }
        st3(A.mvelOut, i, pv + dV / fmaxf(w, 1.0f), v4.w);
    }
    if (!A.ovfOff) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t = blk * (SC_THREADS / 32) + wid; t < nOvf; t += blocks * (SC_THREADS / 32)) {
        const int i = A.ovf[t], n = A.ovfN[t];
        const long long off = A.ovfOff[t];
        if (off < 0 || i < 0 || n <= warpMin || !(A.minfo[i].z & SC_ACTIVE)) continue;   // warp-uniform
        const float4 v4 = A.mvelIn[i], p4 = A.mpos[i];
        const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
        const sc_f3 ppv = sc_make_f3(p4.x, p4.y, p4.z) + pv;
        const uint4 *__restrict__ e = A.ovfPool + off;
        float acc = 0.0f;   // lanes 0-2: dV's components; lane 3: the weight
        for (int b = 0; b < n; b += 32) {
            float term[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (b + lane < n) {
                const uint4 E = e[b + lane];
                const float4 tv = metab_pair_vel(A, E.x);
                const float kw = (E.x & SC_M_FROM_P) ? 2.0f : 1.0f;
                const sc_f3 a = sc_make_f3(__uint_as_float(E.y), __uint_as_float(E.z), __uint_as_float(E.w));
                const sc_f3 d = (a + sc_make_f3(tv.x, tv.y, tv.z) - ppv) * 0.9f * kw;
                term[0] = d.x;
                term[1] = d.y;
                term[2] = d.z;
                term[3] = kw;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) sTerm[wid][lane][k] = term[k];
            __syncwarp();
            if (lane < 4) {
                const int m = min(32, n - b);
                for (int u = 0; u < m; u++) acc += sTerm[wid][u][lane];
            }
            __syncwarp();
        }
        const float dy = __shfl_sync(0xffffffffu, acc, 1), dz = __shfl_sync(0xffffffffu, acc, 2),
                    w = __shfl_sync(0xffffffffu, acc, 3);
        if (lane == 0) st3(A.mvelOut, i, pv + sc_make_f3(acc, dy, dz) / fmaxf(w, 1.0f), v4.w);
    }
}

// The metabolic sweep: the items whose list fits, in count order; at G = 8 the
// first `extra` blocks take the overflowed items (the longest lists start
// first).  Pairs are taken G at a time: the group's neighbour velocities and
// the next group's entries are all in flight together, so a thread waits
// about one memory latency per group instead of one per pair.  Entries are
// read once per launch (evict-first) and lie at a place known from the list
// position, so they are on their way with the item's own records; velocities
// are re-read by nearby items.  Inactive items' velocities are copied until
// both buffers hold them.
//
// G = 4 keeps four blocks per SM for sims that fill the device, where the
// pool's stream from HBM bounds the launch; G = 8 halves the rounds of sims
// that do not, where the rounds' latency does.
//
// At G = 4 a block's warps take its 32-item groups as they come free: the lists
// of every 256 items are ranked by length, so of a warp to a group the later
// ones would wait, their registers held, for the first.  sc_phase_relax_metab
// chooses how many groups a block has.
template <int G, bool BATCH>
__device__ __forceinline__ void relax_metab_item(const ScParams &P, const RelaxMArgs &A, int g) {
    if (g >= *A.nActivePtr) return;
    const int i = A.L.perm[g], c = A.L.cnt[g];
    const uint4 *pairs = A.pool + A.warpOff[g >> 5] + (g & 31);
    // after the sort the active items are exactly the binned ones
    const int binned = P.mAllActive ? (int)A.cellStartM[P.cells] : 0;
    if (i < 0) return;
    const bool act = P.mAllActive ? i < binned : (A.minfo[i].z & SC_ACTIVE) != 0;
    if (!act) {
        if (A.age == 0) A.mvelOut[i] = A.mvelIn[i];
        return;
    }
    if (c > min(SC_LIST_M, P.listLimit)) return;
    const float4 v4 = A.mvelIn[i], p4 = A.mpos[i];
    uint4 E[G];
#pragma unroll
    for (int q = 0; q < G; q++) E[q] = q < c ? __ldcs(pairs + (size_t)q * 32) : make_uint4(0, 0, 0, 0);
    const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = sc_make_f3(p4.x, p4.y, p4.z) + pv;
    sc_f3 dV = sc_zero3();
    float w = 0.0f;
    for (int k0 = 0; k0 < c; k0 += G) {
        float4 tv[G];
        uint4 En[G];
#pragma unroll
        for (int q = 0; q < G; q++) tv[q] = k0 + q < c ? metab_pair_vel(A, E[q].x) : make_float4(0, 0, 0, 0);
#pragma unroll
        for (int q = 0; q < G; q++) {
            const int k = k0 + G + q;
            En[q] = k < c ? __ldcs(pairs + (size_t)k * 32) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int q = 0; q < G; q++) {
            if (k0 + q < c) metab_pool_term(E[q], tv[q], ppv, dV, w);
            E[q] = En[q];
        }
    }
    st3(A.mvelOut, i, pv + dV / fmaxf(w, 1.0f), v4.w);
}
template <int G, bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, G == 4 ? 4 : 2) k_relax_metab(ScParams P, RelaxMArgs A, int extra,
                                                                            int groups) {
    if constexpr (G == 8) {
        __shared__ float sTerm[SC_THREADS / 32][32][SC_TERM_ROW];
        if ((int)blockIdx.x < extra) {
            if (*A.ovfCount > 0) relax_metab_overflow<BATCH>(P, A, blockIdx.x, extra, sTerm);
            return;
        }
        relax_metab_item<G, BATCH>(P, A, ((int)blockIdx.x - extra) * SC_THREADS + threadIdx.x);   // groups = 8
    } else {
        __shared__ int s_next;
        if (threadIdx.x == 0) s_next = SC_THREADS / 32;
        __syncthreads();
        const int lane = threadIdx.x & 31;
        for (int q = threadIdx.x >> 5; q < groups;) {
            relax_metab_item<G, BATCH>(P, A, ((int)blockIdx.x * groups + q) * 32 + lane);
            int n = 0;
            if (lane == 0) n = atomicAdd(&s_next, 1);
            q = __shfl_sync(0xffffffffu, n, 0);
        }
    }
}

// The lean pool's sweep: per pair the neighbour's position and velocity are
// gathered and the reference's term (metab_pair) evaluated in full, pairs
// taken SC_METAB_GROUP at a time as in k_relax_metab.  The image test of a
// periodic box is decided once per item (Imager), the collision distance per
// neighbour kind (the lipids' and the metabolic items' radii are each one
// value in practice, CollisionDistCache recomputes it when they are not).
//
// With OVF the first `extra` blocks take the overflowed items, in sims that do
// not fill the device; in those that do, the walk's stack and shared memory
// cost the sweep more than a launch (196,613 + 983,041 items, five steps 29.1 /
// 27.3 ms with and without).  Waits for gathers bound the sweep, and its spills
// did: two pairs at a time at three blocks per SM have none, 24.4 ms, against
// 26.9 for four at four, 25.1 for four at three and 24.6 for two at four.
#define SC_METAB_GROUP 2
template <bool BATCH, bool OVF>
__global__ void __launch_bounds__(SC_THREADS, 3) k_relax_metab_lean(ScParams P, RelaxMArgs A, int extra) {
    if constexpr (OVF) {
        __shared__ float sTerm[SC_THREADS / 32][32][SC_TERM_ROW];
        if ((int)blockIdx.x < extra) {
            if (*A.ovfCount > 0) relax_metab_overflow<BATCH>(P, A, blockIdx.x, extra, sTerm);
            return;
        }
    }
    const int g = ((int)blockIdx.x - extra) * SC_THREADS + threadIdx.x;   // list position (count-ordered)
    if (g >= *A.nActivePtr) return;
    const int i = A.L.perm[g];
    if (i < 0) return;
    if (BATCH) rep_apply<BATCH>(P, A.minfo[i].w);
    const bool act = P.mAllActive ? i < (int)A.cellStartM[P.cells] : (A.minfo[i].z & SC_ACTIVE) != 0;
    if (!act) {
        if (A.age == 0) A.mvelOut[i] = A.mvelIn[i];
        return;
    }
    const float4 v4 = A.mvelIn[i];
    const int c = A.L.cnt[g];
    if (c > min(SC_LIST_M, P.listLimit)) return;
    const float4 p4 = A.mpos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
    const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
    const sc_f3 ppv = pp + pv;
    sc_f3 dV = sc_zero3();
    float w = 0.0f;
    CollisionDistCache cm, cp;
    const uint32_t *pairs = reinterpret_cast<const uint32_t *>(A.pool) + A.warpOff[g >> 5] + (g & 31);
    uint32_t E[SC_METAB_GROUP];
#pragma unroll
    for (int q = 0; q < SC_METAB_GROUP; q++) E[q] = q < c ? __ldcs(pairs + (size_t)q * 32) : 0u;
    for (int k0 = 0; k0 < c; k0 += SC_METAB_GROUP) {
        float4 t4[SC_METAB_GROUP], tv[SC_METAB_GROUP];
        uint32_t En[SC_METAB_GROUP];
#pragma unroll
        for (int q = 0; q < SC_METAB_GROUP; q++) {
            const bool on = k0 + q < c;
            const bool fromP = (E[q] & SC_M_FROM_P) != 0;
            const int j = (int)(E[q] & SC_M_INDEX);
            t4[q] = on ? (fromP ? A.ppos : A.mpos)[j] : make_float4(0, 0, 0, 0);
            tv[q] = on ? (fromP ? A.pvel : A.mvelIn)[j] : make_float4(0, 0, 0, 0);
        }
#pragma unroll
        for (int q = 0; q < SC_METAB_GROUP; q++) {
            const int k = k0 + SC_METAB_GROUP + q;
            En[q] = k < c ? __ldcs(pairs + (size_t)k * 32) : 0u;
        }
#pragma unroll
        for (int q = 0; q < SC_METAB_GROUP; q++) {
            if (k0 + q < c) {
                const bool fromP = (E[q] & SC_M_FROM_P) != 0;
                const float cd = fromP ? cp.get(p4.w, t4[q].w) : cm.get(p4.w, t4[q].w);
                metab_pair(IM, pp, ppv, t4[q], tv[q], cd, fromP, dV, w);
            }
            E[q] = En[q];
        }
    }
    st3(A.mvelOut, i, pv + dV / fmaxf(w, 1.0f), v4.w);
}

// The overflowed items in a launch of their own.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_relax_metab_overflow(ScParams P, RelaxMArgs A) {
    __shared__ float sTerm[SC_THREADS / 32][32][SC_TERM_ROW];
    if (*A.ovfCount > 0) relax_metab_overflow<BATCH>(P, A, blockIdx.x, gridDim.x, sTerm);
}

// ---- the same sweep on column-segment tiles (sc_tile.cuh) ---------------------
// Shared-memory header of a tile block; the tile arrays follow it.
struct TileMHeader {
    uint64_t bar;
    int nItems;
    int runBase[SC_TILE_NITEMCOL], runStart[SC_TILE_NITEMCOL + 1];
    TileRanges RM, RP;
};
#define SC_TILE_HDR_BYTES ((sizeof(TileMHeader) + 127) / 128 * 128)

// The block's geometry, both range tables and its item runs (the inner
// columns over [z0, z1)); ends with a block barrier.
__device__ __forceinline__ void tile_m_setup(const ScParams &P, const TileGeom &G, const uint32_t *__restrict__ cellStartM,
                                             const uint32_t *__restrict__ cellStartP, TileMHeader &H) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) tile_ranges(P, G, cellStartM, 0, P.tileCapM, H.RM);
    if (warp == 1) tile_ranges(P, G, cellStartP, P.tileCapM, P.tileCapP, H.RP);
    if (warp == 2) {
        int b = 0, l = 0;
        if (lane < SC_TILE_NITEMCOL) {
            const int gx = G.x0 + lane / SC_TILE_TY, gy = G.y0 + lane % SC_TILE_TY;
            if (gx < G.n && gy < G.n) {
                const uint32_t k0 = cell_key(P, (uint32_t)gx, (uint32_t)gy, 0);
                b = (int)cellStartM[k0 + (uint32_t)G.z0];
                l = (int)cellStartM[k0 + (uint32_t)G.z1] - b;
            }
        }
        int x = l;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < SC_TILE_NITEMCOL) {
            H.runBase[lane] = b;
            H.runStart[lane] = x - l;
        }
        if (lane == SC_TILE_NITEMCOL - 1) {
            H.runStart[SC_TILE_NITEMCOL] = x;
            H.nItems = x;
        }
    }
    __syncthreads();
}
// Slot of the block's t-th item.
__device__ __forceinline__ int tile_item(const TileMHeader &H, int t) {
    int q = 0;
#pragma unroll
    for (int k = 1; k < SC_TILE_NITEMCOL; k++) q += t >= H.runStart[k];
    return H.runBase[q] + (t - H.runStart[q]);
}

// Packed 16-bit list entries: 8 consecutive entries of an item share one
// 16-byte chunk, chunks warp-tiled (chunk q of item i at
// ((i/32) * K/8 + q) * 32 + i%32), so one load brings 8 entries.
__host__ __device__ __forceinline__ size_t sc_list16_at(int K, int i, int k) {
    return (((size_t)(i >> 5) * (size_t)(K / 8) + (size_t)(k >> 3)) * 32 + (size_t)(i & 31)) * 8 + (size_t)(k & 7);
}

// M list on tiles: entries are 16-bit tile offsets (metabolic slots first,
// then particle slots), in the reference's visiting order, packed.  An item whose
// neighbourhood leaves the tile, or whose list would overflow, is listed in
// `ovf` for the scanning kernel.
__global__ void __launch_bounds__(SC_THREADS) k_build_m_tile(ScParams P, const uint32_t *__restrict__ cellStartM,
                                                             const uint32_t *__restrict__ cellStartP,
                                                             const float4 *__restrict__ mpos, const int4 *__restrict__ minfo,
                                                             const float4 *__restrict__ ppos_, const int4 *__restrict__ pinfo,
                                                             uint16_t *__restrict__ list, int *__restrict__ cnt,
                                                             int *__restrict__ ovf, int *__restrict__ ovfCount) {
    extern __shared__ __align__(128) unsigned char smraw[];
    TileMHeader &H = *reinterpret_cast<TileMHeader *>(smraw);
    const int cap = P.tileCapM + P.tileCapP;
    float4 *spos = reinterpret_cast<float4 *>(smraw + SC_TILE_HDR_BYTES);
    uint8_t *sok = reinterpret_cast<uint8_t *>(spos + cap);
    TileGeom G;
    G.init(P, blockIdx.x);
    tile_m_setup(P, G, cellStartM, cellStartP, H);
    for (int r = 0; r < SC_TILE_NRANGE; r++) {
        for (int k = threadIdx.x; k < H.RM.len[r]; k += blockDim.x) {
            const int j = H.RM.base[r] + k, o = H.RM.off[r] + k;
            spos[o] = mpos[j];
            sok[o] = (minfo[j].z & SC_ACTIVE) ? 1 : 0;
        }
        for (int k = threadIdx.x; k < H.RP.len[r]; k += blockDim.x) {
            const int j = H.RP.base[r] + k, o = H.RP.off[r] + k;
            const int4 tin = pinfo[j];
            spos[o] = ppos_[j];
            sok[o] = ((tin.z & SC_ACTIVE) && tin.y == SC_PARTICLE_TYPE_LIPID) ? 1 : 0;
        }
    }
    __syncthreads();
    const int bits = P.bits;
    const uint32_t zmask = (1u << bits) - 1u;
    for (int t = threadIdx.x; t < H.nItems; t += blockDim.x) {
        const int i = tile_item(H, t);
        if (!(minfo[i].z & SC_ACTIVE)) {
            cnt[i] = 0;
            continue;
        }
        float4 p4 = mpos[i];
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
        const float prad = p4.w, lim = P.maxInt;
        CollisionDistCache cm, cp;
        int c = 0;
        bool miss = false;
        const int climit = min(SC_LIST_M, P.listLimit);
        cells27(P, pp, reach(P, pp, lim, SC_BINNED_M | SC_BINNED_P), [&](uint32_t key) {
            if (miss) return;
            const int r = G.range_of((int)(key >> (2 * bits)), (int)((key >> bits) & zmask), (int)(key & zmask));
            const int am = (int)cellStartM[key], em = (int)cellStartM[key + 1];
            const int ap = (int)cellStartP[key], ep = (int)cellStartP[key + 1];
            // a non-empty cell outside the tile, or clipped by its capacity
            if ((em > am && (r < 0 || am - H.RM.base[r] + (em - am) > H.RM.len[r])) ||
                (ep > ap && (r < 0 || ap - H.RP.base[r] + (ep - ap) > H.RP.len[r]))) {
                miss = true;
                return;
            }
            for (int j = am; j < em; j++) {
                const int o = H.RM.off[r] + (j - H.RM.base[r]);
                if (j == i || !sok[o]) continue;
                float4 t4 = spos[o];
                sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
                if (outside_cube(delta, lim)) continue;
                if (cm.collides(prad, t4.w, delta)) {
                    if (c < climit) list[sc_list16_at(SC_LIST_M, i, c)] = (uint16_t)o;
                    c++;
                }
            }
            for (int j = ap; j < ep; j++) {
                const int o = H.RP.off[r] + (j - H.RP.base[r]);
                if (!sok[o]) continue;
                float4 t4 = spos[o];
                sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
                if (outside_cube(delta, lim)) continue;
                if (cp.collides(prad, t4.w, delta)) {
                    if (c < climit) list[sc_list16_at(SC_LIST_M, i, c)] = (uint16_t)o;
                    c++;
                }
            }
        });
        if (miss || c > climit) {
            cnt[i] = INT_MAX;
            ovf[atomicAdd(ovfCount, 1)] = i;
        } else {
            cnt[i] = c;
        }
    }
}

// relaxMetabolicParticles on tiles: the block bulk-copies the positions and
// velocities of its tile, then walks each item's list in shared memory.
__global__ void __launch_bounds__(SC_THREADS) k_relax_metab_tile(ScParams P, RelaxMArgs A,
                                                                 const uint16_t *__restrict__ list,
                                                                 int *__restrict__ errorFlag) {
    extern __shared__ __align__(128) unsigned char smraw[];
    TileMHeader &H = *reinterpret_cast<TileMHeader *>(smraw);
    const int capM = P.tileCapM, cap = P.tileCapM + P.tileCapP;
    float4 *spos = reinterpret_cast<float4 *>(smraw + SC_TILE_HDR_BYTES);
    float4 *svel = spos + cap;
    // after an expired wait anywhere, the remaining blocks do nothing
    if (*(volatile int *)errorFlag == SC_DERR_TILE_TIMEOUT) return;
    TileGeom G;
    G.init(P, blockIdx.x);
    if (threadIdx.x == 0) mbar_init(&H.bar);
    tile_m_setup(P, G, A.cellStartM, A.cellStartP, H);
    if (threadIdx.x < 32) {  // warp 0 issues the bulk copies, a lane per range
        const int lane = threadIdx.x;
        uint32_t bytes = 0;
        for (int r = lane; r < SC_TILE_NRANGE; r += 32)
            bytes += 32u * (uint32_t)(max(H.RM.len[r], 0) + max(H.RP.len[r], 0));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
        if (lane == 0) mbar_expect_tx(&H.bar, bytes);
        __syncwarp();
        for (int r = lane; r < SC_TILE_NRANGE; r += 32) {
            if (H.RM.len[r] > 0) {
                const uint32_t nb = (uint32_t)H.RM.len[r] * 16u;
                bulk_copy(spos + H.RM.off[r], A.mpos + H.RM.base[r], nb, &H.bar);
                bulk_copy(svel + H.RM.off[r], A.mvelIn + H.RM.base[r], nb, &H.bar);
            }
            if (H.RP.len[r] > 0) {
                const uint32_t nb = (uint32_t)H.RP.len[r] * 16u;
                bulk_copy(spos + H.RP.off[r], A.ppos + H.RP.base[r], nb, &H.bar);
                bulk_copy(svel + H.RP.off[r], A.pvel + H.RP.base[r], nb, &H.bar);
            }
        }
    }
    // the thread's first item is loaded while the tile is in flight
    const int climit = min(SC_LIST_M, P.listLimit);
    int t = threadIdx.x;
    int i = t < H.nItems ? tile_item(H, t) : -1;
    int4 in = i >= 0 ? A.minfo[i] : make_int4(0, 0, 0, 0);
    int c = i >= 0 ? A.L.cnt[i] : 0;
    float4 v4 = i >= 0 ? A.mvelIn[i] : make_float4(0, 0, 0, 0);
    float4 p4 = i >= 0 ? A.mpos[i] : make_float4(0, 0, 0, 0);
    if (!mbar_wait_bounded(&H.bar, 1ll << 31)) {
        if (threadIdx.x == 0) atomicCAS(errorFlag, 0, SC_DERR_TILE_TIMEOUT);
        mbar_wait_bounded(&H.bar, 1ll << 31);   // let the copies in flight land before the block exits
        return;
    }
    for (; t < H.nItems; t += blockDim.x) {
        if (t != (int)threadIdx.x) {
            i = tile_item(H, t);
            in = A.minfo[i];
            c = A.L.cnt[i];
            v4 = A.mvelIn[i];
            p4 = A.mpos[i];
        }
        if (!(in.z & SC_ACTIVE)) {
            A.mvelOut[i] = v4;
            continue;
        }
        if (c > climit) continue;
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_M | SC_BINNED_P);
        const float prad = p4.w;
        const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
        const sc_f3 ppv = pp + pv;
        sc_f3 dV = sc_zero3();
        float w = 0.0f;
        CollisionDistCache cm, cp;
        // 8 entries per load; the next chunk is loaded while this one is walked
        const uint4 *__restrict__ chunks = reinterpret_cast<const uint4 *>(list) +
                                           (size_t)(i >> 5) * (SC_LIST_M / 8) * 32 + (i & 31);
        uint4 cur = c > 0 ? chunks[0] : make_uint4(0, 0, 0, 0);
        for (int q = 0; 8 * q < c; q++) {
            const uint4 nxt = 8 * (q + 1) < c ? chunks[(size_t)(q + 1) * 32] : make_uint4(0, 0, 0, 0);
            const uint32_t words[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
            for (int kk = 0; kk < 8; kk++) {
                if (8 * q + kk >= c) break;
                const uint32_t e = (words[kk >> 1] >> (16 * (kk & 1))) & 0xffffu;
                const float4 t4 = spos[e], tv = svel[e];
                const bool fromP = (int)e >= capM;
                const float cd = fromP ? cp.get(prad, t4.w) : cm.get(prad, t4.w);
                metab_pair(IM, pp, ppv, t4, tv, cd, fromP, dV, w);
            }
            cur = nxt;
        }
        st3(A.mvelOut, i, pv + dV / fmaxf(w, 1.0f), v4.w);
    }
}

// Velocities of the slots past the binned items (inactive since the sort).
__global__ void __launch_bounds__(SC_THREADS) k_copy_tail(const uint32_t *__restrict__ binnedEnd,
                                                          const int *__restrict__ nActivePtr,
                                                          const float4 *__restrict__ in, float4 *__restrict__ out) {
    const int n = *nActivePtr;
    for (int i = (int)*binnedEnd + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = in[i];
}

// ---- metabolites.cuh:266-350 relaxMetabolicParticlePartners ----------------
// Only lipids change, and only their own velocity, which no other thread of
// this kernel reads: updated in place.  List: the colliding metabolic items.
__device__ __forceinline__ void build_lm_item(const ScParams &P, ScanWords &W, const uint32_t *__restrict__ cellStartM, int i,
                                              const float4 *__restrict__ ppos_, const float4 *__restrict__ mpos,
                                              const int4 *__restrict__ minfo, uint32_t *list, int &c) {
    float4 p4 = ppos_[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M);
    const float prad = p4.w, lim = P.maxInt;
    CollisionDistCache cc;
    scan_words(P, W, mpos, [&](uint32_t key) { return cellStartM[key]; }, pp, reach(P, pp, lim, SC_BINNED_M), lim,
               scan_mixed(P, IM, SC_BINNED_M), [&](int j, float4 t4) {
                   sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
                   if ((IM.wrap && outside_cube(delta, lim)) || !active_m(P, minfo, j)) return;
                   if (cc.collides(prad, t4.w, delta)) {
                       if (c < min(SC_LIST_LM, P.listLimit)) list[sc_list_at(SC_LIST_LM, i, c)] = (uint32_t)j;
                       c++;
                   }
               });
}

// LM pairs with their frozen geometry, as the M pairs: per pair
// A = tpos - normalize(tpos - pos) * collisionDistance
// (metabolites.cuh:320-332), the first float3 the reference's velocity term
// evaluates, in a pool region of the list position's warp (pool_take),
// 16 bytes {neighbour, A.x, A.y, A.z} per entry.  An overflowed lipid
// (cnt INT_MAX) is left to the scan of k_relax_partners.
// The active lipids, compacted (warp-aggregated appends: the order of the
// lists does not matter, each lipid's own list keeps the scan's order), so
// the LM build's warps hold only lipids.
__global__ void __launch_bounds__(SC_THREADS) k_lipid_select(const int *__restrict__ nActivePtr,
                                                             const int4 *__restrict__ pinfo, int *__restrict__ work,
                                                             int *__restrict__ workCount) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool lip = false;
    if (i < *nActivePtr) {
        const int4 in = pinfo[i];
        lip = (in.z & SC_ACTIVE) && in.y == SC_PARTICLE_TYPE_LIPID;
    }
    const unsigned m = __ballot_sync(0xffffffffu, lip);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(workCount, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lip) work[base + __popc(m & ((1u << lane) - 1u))] = i;
}

template <bool BATCH>
__device__ __forceinline__ void build_lm_block(
    const ScParams &P0, ScanWords &W, int block, const uint32_t *__restrict__ cellStartM, const int *__restrict__ lipids,
    const int *__restrict__ lipidCount, const int4 *__restrict__ pinfo, const float4 *__restrict__ ppos_,
    const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, uint4 *__restrict__ pool, long long poolCap,
    unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff, uint32_t *scratch,
    int *__restrict__ cnt, int *__restrict__ perm, int cap) {
    const int t = block * SC_THREADS + threadIdx.x;
    const bool valid = t < *lipidCount;
    int c = 0;
    if (valid) {
        ScParams P = P0;
        rep_apply<BATCH>(P, pinfo[lipids[t]].w);
        build_lm_item(P, W, cellStartM, lipids[t], ppos_, mpos, minfo, scratch, c);
    }
    const PoolSlot<uint4> S = pool_take<SC_LIST_LM>(P0, block, valid, c, pool, poolCap, poolUsed, warpOff, cnt, perm, cap,
                                                    nullptr, nullptr, lipids);
    if (S.n == 0) return;
    ScParams P = P0;
    rep_apply<BATCH>(P, pinfo[S.i].w);
    const float4 p4 = ppos_[S.i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_M);
    const float prad = p4.w;
    CollisionDistCache cc;
    for (int k0 = 0; k0 < S.n; k0 += 4) {
        uint32_t j[4];
        float4 t4[4];
#pragma unroll
        for (int q = 0; q < 4; q++) j[q] = k0 + q < S.n ? scratch[sc_list_at(SC_LIST_LM, S.i, k0 + q)] : 0u;
#pragma unroll
        for (int q = 0; q < 4; q++) t4[q] = k0 + q < S.n ? mpos[j[q]] : p4;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (k0 + q >= S.n) break;
            const sc_f3 tpos = IM(sc_make_f3(t4[q].x, t4[q].y, t4[q].z));
            const sc_f3 nd = normalize(tpos - pp);
            const sc_f3 a = tpos - nd * cc.get(prad, t4[q].w);
            S.out[(size_t)(k0 + q) * 32] = make_uint4(j[q], __float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z));
        }
    }
}

template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, 4) k_build_lm(
    ScParams P0, const uint32_t *__restrict__ cellStartM, const int *__restrict__ lipids,
    const int *__restrict__ lipidCount, const int4 *__restrict__ pinfo, const float4 *__restrict__ ppos_,
    const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, uint4 *__restrict__ pool, long long poolCap,
    unsigned long long *__restrict__ poolUsed, long long *__restrict__ warpOff, uint32_t *scratch,
    int *__restrict__ cnt, int *__restrict__ perm, int cap) {
    __shared__ ScanWords W;
    build_lm_block<BATCH>(P0, W, blockIdx.x, cellStartM, lipids, lipidCount, pinfo, ppos_, mpos, minfo, pool, poolCap,
                          poolUsed, warpOff, scratch, cnt, perm, cap);
}

// The three lists of the relaxation in one launch, blocks of the metabolic
// items first, then the lipids', then the particles': the lists read the same
// positions and none of the others.  A sim that does not fill the device has
// each build wait for its own few blocks' longest item (sc_phase_build_all).
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, 3) k_build_all(
    ScParams P, int nbM, int nbLM, CombStart cs, const float4 *__restrict__ comb, const int *__restrict__ nActiveM,
    const int *__restrict__ nActive, const float4 *__restrict__ mpos, const int4 *__restrict__ minfo,
    const float4 *__restrict__ ppos_, const int4 *__restrict__ pinfo,
    uint32_t *__restrict__ poolM, long long poolCapM, unsigned long long *__restrict__ poolUsedM,
    long long *__restrict__ warpOffM, uint32_t *scratchM, int *__restrict__ cntM, int *__restrict__ permM,
    int *__restrict__ ovfM, int *__restrict__ ovfCountM, int *__restrict__ ovfNM,
    const int *__restrict__ lipids, const int *__restrict__ lipidCount, uint4 *__restrict__ poolLM, long long poolCapLM,
    unsigned long long *__restrict__ poolUsedLM, long long *__restrict__ warpOffLM, uint32_t *scratchLM,
    int *__restrict__ cntLM, int *__restrict__ permLM,
    const int *__restrict__ nb, const int *__restrict__ bonds, uint32_t *__restrict__ list, int *__restrict__ cnt,
    int *__restrict__ classIdx, int *__restrict__ classCount, int *__restrict__ ovf, int *__restrict__ ovfCount,
    uint32_t *__restrict__ match, int *__restrict__ matchN, float4 *__restrict__ geo) {
    __shared__ ScanWords W;
    const int b = blockIdx.x;
    if (b < nbM)
        build_m_block<false, BATCH>(P, W, b, cs, comb, nActiveM, mpos, minfo, ppos_, poolM, poolCapM, poolUsedM,
                                    warpOffM, scratchM, cntM, permM, P.Nm, ovfM, ovfCountM, ovfNM);
    else if (b < nbM + nbLM)
        build_lm_block<BATCH>(P, W, b - nbM, cs.m, lipids, lipidCount, pinfo, ppos_, mpos, minfo, poolLM, poolCapLM,
                              poolUsedLM, warpOffLM, scratchLM, cntLM, permLM, P.N);
    else
        build_pp_block<BATCH>(P, W, b - nbM - nbLM, cs.p, nActive, ppos_, pinfo, nb, bonds, list, cnt, P.N, classIdx,
                              classCount, ovf, ovfCount, match, matchN, geo);
}

// metabolites.cuh:267-340 for one lipid: each listed metabolic neighbour
// adds its precomputed geometry and current velocity with weight 2, in list
// order; the pairs are taken four at a time (entries, then velocities, all
// in flight together).  An overflowed lipid scans its neighbourhood.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_relax_partners(
    ScParams P, const uint32_t *__restrict__ cellStartM, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ ppos_, const int4 *__restrict__ pinfo, float4 *__restrict__ pvel_,
    PairList<SC_LIST_LM> L, const uint4 *__restrict__ pool, const long long *__restrict__ warpOff,
    const float4 *__restrict__ mpos, const int4 *__restrict__ minfo, const float4 *__restrict__ mvel) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;   // list position (count-ordered)
    if (g >= *nActivePtr) return;
    // the positions are those of active lipids, -1 past them (k_build_lm)
    const int i = L.perm[g], c = L.cnt[g];
    const uint4 *pairs = pool + warpOff[g >> 5] + (g & 31);
    if (i < 0) return;
    float4 p4 = ppos_[i];
    float4 v4 = pvel_[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const float prad = p4.w;
    const sc_f3 pv = sc_make_f3(v4.x, v4.y, v4.z);
    sc_f3 dV = sc_zero3();
    float w = 0.0f;
    if (c <= min(SC_LIST_LM, P.listLimit)) {
        for (int k0 = 0; k0 < c; k0 += 4) {
            uint4 E[4];
            float4 tv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) E[q] = k0 + q < c ? __ldcs(pairs + (size_t)(k0 + q) * 32) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < 4; q++) tv[q] = k0 + q < c ? mvel[E[q].x] : make_float4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (k0 + q < c) {
                    const sc_f3 a = sc_make_f3(__uint_as_float(E[q].y), __uint_as_float(E[q].z), __uint_as_float(E[q].w));
                    w += 2.0f;
                    dV += (a + sc_make_f3(tv[q].x, tv[q].y, tv[q].z) - (pp + pv)) * 0.9f * 2.0f;
                }
            }
        }
    } else {
        rep_apply<BATCH>(P, pinfo[i].w);
        const Imager IM(P, pp, SC_BINNED_M);
        CollisionDistCache cc;
        const float lim = P.maxInt;
        scan27(P, cellStartM, pp, reach(P, pp, lim, SC_BINNED_M), [&](int j) {
            if (!active_m(P, minfo, j)) return;
            float4 t4 = mpos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) return;
            if (cc.collides(prad, t4.w, delta)) {
                const float cd = cc.cd;
                sc_f3 tpos = IM(sc_make_f3(t4.x, t4.y, t4.z));
                sc_f3 nd = normalize(tpos - pp);
                w += 2.0f;
                dV += (tpos - nd * cd + ld3(mvel, j) - (pp + pv)) * 0.9f * 2.0f;
            }
        });
    }
    st3(pvel_, i, pv + dV / fmaxf(w, 1.0f), v4.w);
}

// Alignment tests of complexify / transitionInteractions (interactions.cuh:319-324, 438-443).
__device__ __forceinline__ void alignment(bool ord, sc_f4 prot, sc_f4 trot, sc_f3 up, sc_f3 tup, sc_f3 delta,
                                          const sc_rule &r, float *oa, float *rpa) {
    sc_f4 ro = rule_ori(r);
    sc_f3 rp = rule_pos(r);
    *oa = ord ? dot(sc_rotate(up, ro), tup) : dot(sc_rotate(tup, ro), up);
    *rpa = ord ? dot(sc_rotate(rp, prot), delta) / sc_normsq3(delta)
               : dot(sc_rotate(rp, trot), -delta) / sc_normsq3(delta);
}
__device__ __forceinline__ bool states_match(bool ord, int ps, int ts, const sc_rule &r) {
    int fs = r.first_partner_state, ss = r.second_partner_state;
    return ord ? ((fs < 0 || fs == ps) && (ss < 0 || ss == ts)) : ((ss < 0 || ss == ps) && (fs < 0 || fs == ts));
}
__device__ __forceinline__ bool group_active_in(const int *__restrict__ b, int nbv, int group) {
    for (int k = 0; k < min(nbv, SC_MAX_ACTIVE_INTERACTIONS); k++)
        if (b[3 * k + 1] == group) return true;
    return false;
}

// ---- interactions.cuh:216-346 complexify --------------------------------------
// New interactions are appended at slots [nb, nb') of the item's own list,
// which no neighbour reads (they read [0, nb)); nb' goes to the next buffer.
// The items complexify can act on, collected before the scan so the scan's
// warps hold only such items (they are a small, scattered part of the
// particles: left in place, almost every warp would carry one or two
// scanning lanes).  No rule of an item's type can add a bond when each is
// transition-only or its group is already active on the item (bonds are
// only added by the scan, so a blocked rule stays blocked); such an item's
// bond count is passed through here.
__global__ void __launch_bounds__(SC_THREADS) k_complexify_select(ScParams P, const int *__restrict__ nActivePtr,
                                                                  const int4 *__restrict__ info,
                                                                  const int *__restrict__ nbIn,
                                                                  int *__restrict__ nbOut,
                                                                  const int *__restrict__ bonds,
                                                                  int *__restrict__ work, int *__restrict__ workCount) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool open = false;
    if (i < *nActivePtr) {
        const int4 in = info[i];
        const int pnb = nbIn[i];
        int cs = 0, ce = 0;
        if ((in.z & SC_ACTIVE) && in.y >= 0 && 2 * in.y + 1 < P.nPidx) {
            cs = P.pidx[2 * in.y];
            ce = P.pidx[2 * in.y + 1];
        }
        for (int k = cs; k < ce && !open && pnb < SC_MAX_ACTIVE_INTERACTIONS; k++) {
            const sc_rule &pii = P.prules[k];
            open = !pii.only_via_transition &&
                   !(pii.group >= 0 && group_active_in(bonds + (size_t)i * 24, pnb, pii.group));
        }
        if (!open) nbOut[i] = pnb;
    }
    // warp-aggregated append (order within the list is free: items do not read what others add)
    const unsigned m = __ballot_sync(0xffffffffu, open);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(workCount, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (open) work[base + __popc(m & ((1u << lane) - 1u))] = i;
}

// The binding draw of a rule with a probability (an extension; the
// reference's rules carry none and always pass).
__device__ __forceinline__ bool bind_draw(const ScParams &P, const sc_rule &r, int pid, int tid, int step) {
    return !r.use_probability || sc_bind_uniform(P.seed, r.id, pid, tid, step) < r.probability;
}

template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_complexify(
    ScParams P, const uint32_t *__restrict__ cellStart, const int *__restrict__ work, const int *__restrict__ workCount,
    const float4 *__restrict__ pos, const float4 *__restrict__ rot, const int4 *__restrict__ info,
    const int *__restrict__ state, const int *__restrict__ nbIn, int *__restrict__ nbOut, int *bonds,
    const int *__restrict__ stepPtr, int prep) {
  const int step = prep ? -1 : *stepPtr;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < *workCount; t += gridDim.x * blockDim.x) {
    const int i = work[t];
    int4 in = info[i];
    rep_apply<BATCH>(P, in.w);
    int pnb = nbIn[i];
    const int cs = P.pidx[2 * in.y], ce = P.pidx[2 * in.y + 1];
    float4 p4 = pos[i];
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, ppos, SC_BINNED_P);
    const sc_f4 prot = ld4(rot, i);
    const int pid = in.x, ptype = in.y, pstate = state[i];
    const sc_f3 up = sc_rotate(sc_up(), prot);
    int *pb = bonds + (size_t)i * 24;
    const int nb0 = pnb;
    const float lim = P.maxInt;
    scan27(P, cellStart, ppos, reach(P, ppos, lim, SC_BINNED_P), [&](int j) {
        if (j == i) return;
        float4 t4 = pos[j];
        sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - ppos;
        if (outside_cube(delta, lim)) return;
        int4 tin = info[j];
        if (!(tin.z & SC_ACTIVE)) return;
        sc_f4 trot = ld4(rot, j);
        sc_f3 tup = sc_rotate(sc_up(), trot);
        const int ttype = tin.y;
        bool ord = p_order(ptype, pid, ttype, tin.x);
        for (int k = cs; k < ce; k++) {
            if (pnb >= SC_MAX_ACTIVE_INTERACTIONS) continue;
            const sc_rule &pii = P.prules[k];
            if (!((ptype == pii.first_partner_type && ttype == pii.second_partner_type) ||
                  (ptype == pii.second_partner_type && ttype == pii.first_partner_type)) ||
                pii.only_via_transition)
                continue;
            if (pii.group >= 0 && (group_active_in(pb, pnb, pii.group) ||
                                   group_active_in(bonds + (size_t)j * 24, nbIn[j], pii.group)))
                continue;
            float oa, rpa;
            alignment(ord, prot, trot, up, tup, delta, pii, &oa, &rpa);
            if (oa > pii.orientation_alignment_threshold &&
                fabs((double)rpa - 1.0) < (1.0 - (double)pii.position_alignment_threshold) &&
                states_match(ord, pstate, state[j], pii) && bind_draw(P, pii, pid, tin.x, step)) {
                pb[3 * pnb] = pii.id;
                pb[3 * pnb + 1] = pii.group;
                pb[3 * pnb + 2] = tin.x;
                pnb++;
            }
        }
    });
    (void)nb0;
    nbOut[i] = pnb;
  }
}

// ---- complexify by deterministic pair claim (sc_config.pair_claim) ----------
// The reference's scan appends a bond on the scanning item's side only, so
// two items can both bond a third that keeps just one of them (the TODO at
// interactions.cuh:297).  Here a step forms rule bonds in two kernels:
//   offer: every open item i that has a free bond slot visits its
//          neighbours as complexify does and, for each neighbour j that some
//          rule would bond it to, lowers claim[j] to the 64-bit key
//          (bits of |delta|^2, i) with atomicMin;
//   bind:  i and j bond when claim[i] names j and claim[j] names i.  Both
//          sides take the first rule that passes for the pair as seen from
//          the lower slot, so the two records always agree.
// At most one rule bond forms per item per step.  Keys and slots are fixed by
// the sort, so the result does not depend on thread scheduling.
struct ClaimItem {
    sc_f3 pos, up;
    sc_f4 rot;
    int id, type, state, nb, cs, ce;
    const int *b;
};
__device__ __forceinline__ ClaimItem claim_item(const ScParams &P, const float4 *__restrict__ pos,
                                                const float4 *__restrict__ rot, const int4 *__restrict__ info,
                                                const int *__restrict__ state, const int *__restrict__ nbIn,
                                                const int *bonds, int i) {
    ClaimItem a;
    const float4 p4 = pos[i];
    a.pos = sc_make_f3(p4.x, p4.y, p4.z);
    a.rot = ld4(rot, i);
    a.up = sc_rotate(sc_up(), a.rot);
    const int4 in = info[i];
    a.id = in.x;
    a.type = in.y;
    a.state = state[i];
    a.nb = nbIn[i];
    a.b = bonds + (size_t)i * 24;
    a.cs = a.ce = 0;
    if (in.y >= 0 && 2 * in.y + 1 < P.nPidx) {
        a.cs = P.pidx[2 * in.y];
        a.ce = P.pidx[2 * in.y + 1];
    }
    return a;
}
// The partner-mapped index of the first rule of a's type that would bond a
// to b (delta = b's position seen from a, minus a's), or -1.
__device__ __forceinline__ int claim_rule(const ScParams &P, const ClaimItem &a, const ClaimItem &b, sc_f3 delta,
                                          int step) {
    if (a.nb >= SC_MAX_ACTIVE_INTERACTIONS) return -1;
    const bool ord = p_order(a.type, a.id, b.type, b.id);
    for (int k = a.cs; k < a.ce; k++) {
        const sc_rule &pii = P.prules[k];
        if (!((a.type == pii.first_partner_type && b.type == pii.second_partner_type) ||
              (a.type == pii.second_partner_type && b.type == pii.first_partner_type)) ||
            pii.only_via_transition)
            continue;
        if (pii.group >= 0 && (group_active_in(a.b, a.nb, pii.group) || group_active_in(b.b, b.nb, pii.group)))
            continue;
        float oa, rpa;
        alignment(ord, a.rot, b.rot, a.up, b.up, delta, pii, &oa, &rpa);
        if (oa > pii.orientation_alignment_threshold &&
            fabs((double)rpa - 1.0) < (1.0 - (double)pii.position_alignment_threshold) &&
            states_match(ord, a.state, b.state, pii) && bind_draw(P, pii, a.id, b.id, step))
            return k;
    }
    return -1;
}
__device__ __forceinline__ unsigned long long claim_key(sc_f3 delta, int i) {
    return ((unsigned long long)sc_f2u(sc_normsq3(delta)) << 32) | (unsigned)i;
}

// Whether some rule of item a's type can bond it to an item of type b with
// the bonds bb[0, nbb): the part of claim_rule that needs no more of it.
__device__ __forceinline__ bool claim_open(const ScParams &P, const ClaimItem &a, int b, int nbb,
                                           const int *__restrict__ bb) {
    for (int k = a.cs; k < a.ce; k++) {
        const sc_rule &pii = P.prules[k];
        if (!((a.type == pii.first_partner_type && b == pii.second_partner_type) ||
              (a.type == pii.second_partner_type && b == pii.first_partner_type)) ||
            pii.only_via_transition)
            continue;
        if (pii.group >= 0 && (group_active_in(a.b, a.nb, pii.group) || group_active_in(bb, nbb, pii.group))) continue;
        return true;
    }
    return false;
}

// Three open items per warp, a lane per column of an item's neighbourhood:
// offers are taken by atomicMin, so their order is free.  With a thread per
// item 6 of a warp's 32 lanes were busy and an item's 27 cells were one chain
// of dependent loads; a lane's column takes its candidates' positions four at
// a time, and a candidate's records are only read once its type and bonds
// leave a rule open (under 10 % of the candidates in the cube at the measured
// mix).  A batch of 24 replicas (0.9 M particles): 290 us a step with a warp per
// item and a lane per cell, 117 us so; the large workload's third step 637 and
// 275 us (477 us with the four candidates' tests unrolled, at 115 registers).
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, 4) k_claim_offer(
    ScParams P0, const uint32_t *__restrict__ cellStart, const int *__restrict__ work, const int *__restrict__ workCount,
    const float4 *__restrict__ pos, const float4 *__restrict__ rot, const int4 *__restrict__ info,
    const int *__restrict__ state, const int *__restrict__ nbIn, const int *__restrict__ bonds,
    const int *__restrict__ stepPtr, int prep, unsigned long long *claim) {
  const int step = prep ? -1 : *stepPtr;
  const int lane = threadIdx.x & 31, col = lane % 9;
  const int ox = col / 3 - 1, oy = col % 3 - 1;
  const int n = lane < 27 ? *workCount : 0;
  const int stride = ((gridDim.x * blockDim.x) >> 5) * 3;
  for (int t = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 3 + lane / 9; t < n; t += stride) {
    const int i = work[t];
    ScParams P = P0;
    if (BATCH) rep_apply<BATCH>(P, info[i].w);
    const ClaimItem a = claim_item(P, pos, rot, info, state, nbIn, bonds, i);
    const float lim = P.maxInt;
    const Reach R = reach(P, a.pos, lim, SC_BINNED_P);
    if (a.nb >= SC_MAX_ACTIVE_INTERACTIONS || ox < R.xl || ox > R.xh || oy < R.yl || oy > R.yh) continue;
    const int g = cell_limit(P);
    int gx = (int)sc_grid_idx(a.pos.x, P.cell, g) + ox, gy = (int)sc_grid_idx(a.pos.y, P.cell, g) + oy;
    const int cz = (int)sc_grid_idx(a.pos.z, P.cell, g);
    // the column's z run, in two parts where a periodic one crosses the face
    int z0 = cz + R.zl, z1 = cz + R.zh, y0 = 0, y1 = -1;
    if (P.periodic) {
        gx = (int)wrap_cell(gx, g);
        gy = (int)wrap_cell(gy, g);
        if (z0 < 0) {
            y0 = y1 = g - 1;
            z0 = 0;
        } else if (z1 >= g) {
            y0 = y1 = 0;
            z1 = g - 1;
        }
    } else {
        if (min(gx, gy) < 0 || max(gx, gy) >= g) continue;
        z0 = max(z0, 0);
        z1 = min(z1, g - 1);
    }
    const Imager IM(P, a.pos, SC_BINNED_P);
    const uint32_t key = cell_key(P, (uint32_t)gx, (uint32_t)gy, 0);
    for (int part = 0; part < 2; part++) {
        if (part && y1 < y0) break;
        const int e = (int)cellStart[key + (uint32_t)(part ? y1 : z1) + 1u];
        for (int j0 = (int)cellStart[key + (uint32_t)(part ? y0 : z0)]; j0 < e; j0 += 4) {
            uint32_t near = 0;   // of the next four (reading up to three past the run: SC_CAND_PAD)
            float4 t4[4];
#pragma unroll
            for (int u = 0; u < 4; u++) t4[u] = pos[j0 + u];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (j0 + u < e && j0 + u != i &&
                    !outside_cube(IM(sc_make_f3(t4[u].x, t4[u].y, t4[u].z)) - a.pos, lim))
                    near |= 1u << u;
            while (near) {
                const int j = j0 + __ffs((int)near) - 1;
                near &= near - 1u;
                const int4 in = info[j];
                if (!(in.z & SC_ACTIVE) || !claim_open(P, a, in.y, nbIn[j], bonds + (size_t)j * 24)) continue;
                const ClaimItem b = claim_item(P, pos, rot, info, state, nbIn, bonds, j);
                const sc_f3 delta = IM(b.pos) - a.pos;
                if (claim_rule(P, a, b, delta, step) >= 0) atomicMin(&claim[j], claim_key(delta, i));
            }
        }
    }
  }
}

template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_claim_bind(
    ScParams P, const int *__restrict__ work, const int *__restrict__ workCount, const float4 *__restrict__ pos,
    const float4 *__restrict__ rot, const int4 *__restrict__ info, const int *__restrict__ state,
    const int *__restrict__ nbIn, int *__restrict__ nbOut, int *bonds, const int *__restrict__ stepPtr, int prep,
    const unsigned long long *__restrict__ claim) {
  const int step = prep ? -1 : *stepPtr;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < *workCount; t += gridDim.x * blockDim.x) {
    const int i = work[t];
    int pnb = nbIn[i];
    const unsigned long long key = claim[i];
    const int j = (int)(unsigned)(key & 0xffffffffull);
    if (key != ~0ull && (int)(unsigned)(claim[j] & 0xffffffffull) == i) {
        const int lo = min(i, j), hi = max(i, j);
        rep_apply<BATCH>(P, info[lo].w);
        const ClaimItem a = claim_item(P, pos, rot, info, state, nbIn, bonds, lo);
        const ClaimItem b = claim_item(P, pos, rot, info, state, nbIn, bonds, hi);
        const Imager IM(P, a.pos, SC_BINNED_P);
        const int k = claim_rule(P, a, b, IM(b.pos) - a.pos, step);
        if (k >= 0 && pnb < SC_MAX_ACTIVE_INTERACTIONS) {
            const sc_rule &pii = P.prules[k];
            int *pb = bonds + (size_t)i * 24;
            pb[3 * pnb] = pii.id;
            pb[3 * pnb + 1] = pii.group;
            pb[3 * pnb + 2] = i == lo ? b.id : a.id;
            pnb++;
        }
    }
    nbOut[i] = pnb;
  }
}

// ---- interactions.cuh:349-555 transitionInteractions -------------------------
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_transition(
    ScParams P, const uint32_t *__restrict__ cellStart, const int *__restrict__ nActivePtr,
    const int *__restrict__ stepPtr, const float4 *__restrict__ pos, const float4 *__restrict__ rot,
    const int4 *__restrict__ info, const int *__restrict__ stateIn, int *__restrict__ stateOut, const int *__restrict__ nbIn,
    int *__restrict__ nbOut, const int *__restrict__ bondsIn, int *__restrict__ bondsOut, int *lscs, int *spoly) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    const int step = *stepPtr;
    int4 in = info[i];
    rep_apply<BATCH>(P, in.w);
    int pnb = min(max(nbIn[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
    int pstate = stateIn[i];
    int b[SC_MAX_ACTIVE_INTERACTIONS * 3];
#pragma unroll
    for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS * 3; k++) b[k] = k < 3 * pnb ? bondsIn[(size_t)i * 24 + k] : 0;
    // Only bonds whose rule transitions or breaks after a transition act in
    // the scan: without one the scan would change nothing.
    bool acts = false;
#pragma unroll
    for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++)
        if (k < pnb && b[3 * k] >= 10) {
            const sc_rule &pii = rule_at(P, b[3 * k]);
            acts |= pii.transition_to >= 0 || pii.break_after_transition;
        }
    if ((in.z & SC_ACTIVE) && acts) {
        float4 p4 = pos[i];
        const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, ppos, SC_BINNED_P);
        const sc_f4 prot = ld4(rot, i);
        const int pid = in.x, ptype = in.y;
        const sc_f3 up = sc_rotate(sc_up(), prot);
        int src = -1;
        int tId = 0, tGroup = 0, tSet = 0, tFirst = 0, tSecond = 0, tFs = 0, tSs = 0, tPoly = 0;
        const float lim = P.maxInt;
        scan27(P, cellStart, ppos, reach(P, ppos, lim, SC_BINNED_P), [&](int j) {
            if (j == i) return;
            float4 t4 = pos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - ppos;
            if (outside_cube(delta, lim)) return;
            int4 tin = info[j];
            if (!(tin.z & SC_ACTIVE)) return;
            bool loaded = false;
            sc_f4 trot;
            sc_f3 tup;
            const int ttype = tin.y;
            const bool ord = p_order(ptype, pid, ttype, tin.x);
            for (int k = 0; k < pnb; k++) {
                if (b[3 * k] < 10) continue;
                if (b[3 * k + 2] != tin.x) continue;
                const sc_rule &pii = rule_at(P, b[3 * k]);
                if (!(pii.transition_to >= 0 || pii.break_after_transition)) continue;
                if (!loaded) { trot = ld4(rot, j); tup = sc_rotate(sc_up(), trot); loaded = true; }
                float oa, rpa;
                alignment(ord, prot, trot, up, tup, delta, pii, &oa, &rpa);
                bool aligned = pii.break_after_transition || !pii.wait_for_alignment ||
                               (oa > pii.orientation_alignment_threshold &&
                                fabs((double)rpa - 1.0) < (1.0 - (double)pii.position_alignment_threshold));
                if (!(aligned && (!pii.wait_for_state || states_match(ord, pstate, stateIn[j], pii)))) continue;
                if (pii.transition_to >= 0) {
                    const sc_rule &tpii = rule_at(P, pii.transition_to);
                    if (tpii.group >= 0 && tpii.group != pii.group) {
                        bool ga = false;
                        for (int l = 0; l < pnb; l++)
                            if (b[3 * l + 1] == tpii.group) { ga = true; break; }
                        if (!ga) ga = group_active_in(bondsIn + (size_t)j * 24, nbIn[j], tpii.group);
                        if (ga) continue;
                    }
                    if (!tpii.set_state || !((ptype == tpii.first_partner_type && tpii.first_partner_state >= 0) ||
                                             (ptype == tpii.second_partner_type && tpii.second_partner_state >= 0))) {
                        b[3 * k] = tpii.id;
                        b[3 * k + 1] = tpii.group;
                    } else {
                        src = k;
                        tId = tpii.id; tGroup = tpii.group; tSet = tpii.set_state;
                        tFirst = tpii.first_partner_type; tSecond = tpii.second_partner_type;
                        tFs = tpii.first_partner_state; tSs = tpii.second_partner_state; tPoly = tpii.polymerize;
                    }
                } else if (pii.break_after_transition) {
                    for (int l = k; l < pnb - 1; l++) {
                        b[3 * l] = b[3 * l + 3];
                        b[3 * l + 1] = b[3 * l + 4];
                        b[3 * l + 2] = b[3 * l + 5];
                    }
                    pnb--;
                    if (src > k) src--;
                    k--;
                }
            }
        });
        if (src >= 0) {
            b[3 * src] = tId;
            b[3 * src + 1] = tGroup;
            if (tSet) {
                if (ptype == tFirst && tFs >= 0) { pstate = tFs; lscs[i] = step; }
                if (ptype == tSecond && tSs >= 0) { pstate = tSs; lscs[i] = step; }
            }
            if (tPoly >= 0) {
                const sc_rule &poly = rule_at(P, tPoly);
                if (poly.first_partner_type == ptype || poly.second_partner_type == ptype) spoly[i] = tPoly;
            }
        }
    }
    stateOut[i] = pstate;
    nbOut[i] = pnb;
    for (int k = 0; k < 3 * pnb; k++) bondsOut[(size_t)i * 24 + k] = b[k];
}

// ---- interactions.cuh:558-740 polymerize --------------------------------------
// The reference runs it in place with atomicAdd slot / id allocation and
// cross-slot writes, so its outcome depends on thread scheduling.  Here the
// outcome is the one a one-item-at-a-time execution in slot (index) order
// gives, computed in parallel:
//  * k_poly_count / k_poly_offsets / k_poly_plan list the scheduled items in
//    index order (an ordered compaction), with the rank of each one's new
//    monomer among the items whose rule creates one: in slot order the k-th
//    creating item takes index lastActive + 1 + k and id nextId + k (when
//    the index is below the capacity), so neither needs a serial counter;
//  * an item's processing reads and writes its own bonds and those of its
//    previous monomer (pmi, found by id among the binned particles, whose
//    ids no processing changes) and writes its new monomer's slot.  An item
//    whose previous monomer is not itself listed or shared with another item,
//    and which is nobody's previous monomer, shares its footprint with no
//    other: those run at once (k_poly_apply), the others in slot order by one
//    thread (k_poly_finish).  An item holds one bond of its rule's group, so
//    what another's processing can do to its previous monomer is to take it
//    away; a list with an item that holds more runs in slot order as a whole.
__device__ __forceinline__ bool poly_scheduled(const PFields &F, int n0, int i) {
    return i < n0 && (F.info[i].z & SC_ACTIVE) && F.spoly[i] >= 0;
}
__device__ __forceinline__ bool poly_creates(const ScParams &P, const PFields &F, int i) {
    const sc_rule &poly = rule_at(P, F.spoly[i]);
    const bool first = poly.first_partner_type == F.info[i].y;
    return (first ? poly.second_partner_type : poly.first_partner_type) >= 0;
}
// First bond of the rule's group (the active polymerisation bond), -1 if none.
__device__ __forceinline__ int poly_api(const sc_rule &poly, const int *pb, int pnb) {
    for (int k = 0; k < pnb; k++)
        if (pb[3 * k + 1] == poly.group) return k;
    return -1;
}
// The binned particle whose id is `target` (the last one in scan order).
__device__ __forceinline__ int poly_find(const ScParams &P, const uint32_t *cellStart, const PFields &F, int i,
                                         int target) {
    float4 p4 = F.pos[i];
    int pmi = -1;
    scan27(P, cellStart, sc_make_f3(p4.x, p4.y, p4.z), [&](int j) {
        if (j == i) return;
        int4 tin = F.info[j];
        if (!(tin.z & SC_ACTIVE)) return;
        if (tin.x == target) pmi = j;
    });
    return pmi;
}

// Removes the first bond of `group` from item m's bonds (shifting the rest).
__device__ __forceinline__ int poly_drop_group(int *mb, int mnb, int group) {
    for (int k = 0; k < mnb; k++) {
        if (mb[3 * k + 1] == group) {
            for (int l = k; l < mnb - 1; l++) {
                mb[3 * l] = mb[3 * l + 3]; mb[3 * l + 1] = mb[3 * l + 4]; mb[3 * l + 2] = mb[3 * l + 5];
            }
            return mnb - 1;
        }
    }
    return mnb;
}

// One scheduled item: `pmi` its previous monomer (`planned`: found before the
// items ahead of it ran, and good as long as its bond names that particle), its
// new monomer at newIdx with id newId (used when newIdx < N).
__device__ void poly_one(const ScParams &P, const uint32_t *cellStart, const PFields &F, int i, int step, int pmi,
                         bool planned, int newIdx, int newId) {
    int4 in = F.info[i];
    const sc_rule &poly = rule_at(P, F.spoly[i]);
    const int pid = in.x, ptype = in.y;
    int *pb = F.bonds + (size_t)i * 24;
    int pnb = min(max(F.nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
    const int api = poly_api(poly, pb, pnb);
    if (planned && !(api >= 0 && pmi >= 0 && F.info[pmi].x == pb[3 * api + 2]))
        pmi = api >= 0 ? poly_find(P, cellStart, F, i, pb[3 * api + 2]) : -1;
    float4 p4 = F.pos[i];
    const sc_f3 ppos = sc_make_f3(p4.x, p4.y, p4.z);
    const bool first = poly.first_partner_type == ptype;
    const int newType = first ? poly.second_partner_type : poly.first_partner_type;
    const int newState = first ? poly.second_partner_state : poly.first_partner_state;
    const int spolyId = F.spoly[i];
    if (newType >= 0) {
        float nr = 0.0f;
        int nh = 0;
        if (newType < P.nTypes) { nr = P.types[newType].radius; nh = P.types[newType].hydrophobic; }
        if (newIdx < P.N) {
            sc_f3 rp = rule_pos(poly);
            sc_f4 ro = rule_ori(poly);
            sc_f4 prot = ld4(F.rot, i);
            sc_f3 npos = ppos + sc_rotate(ptype < newType ? rp : -rp, prot);
            if (P.periodic) npos = sc_wrap3(npos, P.simSize);
            sc_f4 nrot = sc_qmul(prot, ptype < newType ? ro : sc_qinv(ro));
            // Particle(newId, newType, 0, radius, hydrophobic, pos, rot): types.cuh:192-221
            F.pos[newIdx] = make_float4(npos.x, npos.y, npos.z, nr);
            F.vel[newIdx] = make_float4(0, 0, 0, 0);
            st4(F.rot, newIdx, nrot);
            F.angvel[newIdx] = make_float4(0, 0, 0, 1);
            F.posnoise[newIdx] = make_float4(0, 0, 0, 0);
            F.angnoise[newIdx] = make_float4(0, 0, 0, 1);
            F.dbg[newIdx] = make_float4(0, 0, 0, 0);
            F.info[newIdx] = make_int4(newId, newType, SC_ACTIVE, (int)(int8_t)nh);
            F.state[newIdx] = newState >= 0 ? newState : 0;
            F.lscs[newIdx] = newState >= 0 ? step : -1;
            F.spoly[newIdx] = -1;
            int *nbp = F.bonds + (size_t)newIdx * 24;
            int nnb = 0;
            nbp[0] = spolyId; nbp[1] = poly.group; nbp[2] = pid;
            nnb = 1;
            if (pmi >= 0) {
                int *mb = F.bonds + (size_t)pmi * 24;
                int mnb = poly_drop_group(mb, min(max(F.nb[pmi], 0), SC_MAX_ACTIVE_INTERACTIONS), poly.group);
                if (mnb < SC_MAX_ACTIVE_INTERACTIONS) {
                    mb[3 * mnb] = SC_INTERACTION_TYPE_CHAIN; mb[3 * mnb + 1] = SC_INTERACTION_GROUP_FORWARD;
                    mb[3 * mnb + 2] = newId;
                }
                mnb++;
                F.nb[pmi] = mnb;
                nbp[3] = SC_INTERACTION_TYPE_CHAIN; nbp[4] = SC_INTERACTION_GROUP_BACKWARD; nbp[5] = F.info[pmi].x;
                nnb = 2;
                pb[3 * api] = spolyId;
                pb[3 * api + 2] = newId;
            } else {
                if (pnb < SC_MAX_ACTIVE_INTERACTIONS) {
                    pb[3 * pnb] = spolyId; pb[3 * pnb + 1] = poly.group; pb[3 * pnb + 2] = newId;
                }
                pnb++;
            }
            for (int k = 3 * nnb; k < 24; k++) nbp[k] = 0;
            F.nb[newIdx] = nnb;
        }
    } else {
        // End of the chain; the reference's out-of-bounds stores without a
        // previous monomer / active bond (interactions.cuh:728, 731-734) are skipped.
        if (pmi >= 0) {
            int *mb = F.bonds + (size_t)pmi * 24;
            F.nb[pmi] = poly_drop_group(mb, min(max(F.nb[pmi], 0), SC_MAX_ACTIVE_INTERACTIONS), poly.group);
        }
        if (api >= 0) {
            for (int l = api; l < pnb - 1; l++) {
                pb[3 * l] = pb[3 * l + 3]; pb[3 * l + 1] = pb[3 * l + 4]; pb[3 * l + 2] = pb[3 * l + 5];
            }
            pnb--;
        }
    }
    F.nb[i] = pnb;
    F.spoly[i] = -1;
}

// Per block of SC_THREADS items: (scheduled, creating) counts.
__global__ void __launch_bounds__(SC_THREADS) k_poly_count(ScParams P, PFields F, const ScCounters *ctr,
                                                           int2 *blk) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n0 = ctr->nActive;
    const bool s = poly_scheduled(F, n0, i);
    const bool c = s && poly_creates(P, F, i);
    const int ns = __syncthreads_count(s), nc = __syncthreads_count(c);
    if (threadIdx.x == 0) blk[blockIdx.x] = make_int2(ns, nc);
}

// Exclusive offsets of the block counts (one CTA), the totals, and the
// conflict flag cleared.
#define SC_POLY_SCAN_THREADS 1024
__global__ void __launch_bounds__(SC_POLY_SCAN_THREADS) k_poly_offsets(const int2 *__restrict__ blk, int2 *off,
                                                                       int nblk, ScCounters *ctr) {
    __shared__ int2 s_w[SC_POLY_SCAN_THREADS / 32];
    __shared__ int2 s_carry;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_carry = make_int2(0, 0);
    __syncthreads();
    for (int b0 = 0; b0 < nblk; b0 += SC_POLY_SCAN_THREADS) {
        const int b = b0 + t;
        const int2 v = b < nblk ? blk[b] : make_int2(0, 0);
        int2 x = v;  // inclusive warp scan
        for (int d = 1; d < 32; d *= 2) {
            const int ax = __shfl_up_sync(0xffffffffu, x.x, d), ay = __shfl_up_sync(0xffffffffu, x.y, d);
            if (lane >= d) { x.x += ax; x.y += ay; }
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int2 w = s_w[lane];
            for (int d = 1; d < 32; d *= 2) {
                const int ax = __shfl_up_sync(0xffffffffu, w.x, d), ay = __shfl_up_sync(0xffffffffu, w.y, d);
                if (lane >= d) { w.x += ax; w.y += ay; }
            }
            s_w[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const int2 before = warp ? s_w[warp - 1] : make_int2(0, 0);
        const int2 carry = s_carry;
        if (b < nblk) off[b] = make_int2(carry.x + before.x + x.x - v.x, carry.y + before.y + x.y - v.y);
        __syncthreads();
        if (t == 0) s_carry = make_int2(carry.x + s_w[31].x, carry.y + s_w[31].y);
        __syncthreads();
    }
    if (t == 0) {
        ctr->polyCount = s_carry.x;
        ctr->polyCreates = s_carry.y;
        ctr->polyConflict = 0;
    }
}

// Lists the scheduled items in index order with their monomer ranks, finds
// each one's previous monomer and counts the claims on it, SC_POLY_LISTED more
// when it is itself scheduled; an item with two bonds of its rule's group sends
// the whole list through the serial path.
#define SC_POLY_LISTED 0x10000
__global__ void __launch_bounds__(SC_THREADS) k_poly_plan(ScParams P, const uint32_t *__restrict__ cellStart, PFields F,
                                                          ScCounters *ctr, const int2 *__restrict__ off, int *list,
                                                          int *rank, int *pmiOut, int *claim) {
    __shared__ int2 s_w[SC_THREADS / 32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n0 = ctr->nActive;
    const bool s = poly_scheduled(F, n0, i);
    const bool c = s && poly_creates(P, F, i);
    const unsigned bs = __ballot_sync(0xffffffffu, s), bc = __ballot_sync(0xffffffffu, c);
    const unsigned below = (1u << lane) - 1u;
    if (lane == 0) s_w[warp] = make_int2(__popc(bs), __popc(bc));
    __syncthreads();
    if (!s) return;
    int2 o = off[blockIdx.x];
    for (int w = 0; w < warp; w++) { o.x += s_w[w].x; o.y += s_w[w].y; }
    const int slot = o.x + __popc(bs & below);
    list[slot] = i;
    rank[slot] = c ? o.y + __popc(bc & below) : -1;
    const sc_rule &poly = rule_at(P, F.spoly[i]);
    const int *pb = F.bonds + (size_t)i * 24;
    const int api = poly_api(poly, pb, min(max(F.nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS));
    const int pmi = api >= 0 ? poly_find(P, cellStart, F, i, pb[3 * api + 2]) : -1;
    pmiOut[slot] = pmi;
    if (pmi >= 0) atomicAdd(&claim[pmi], poly_scheduled(F, n0, pmi) ? 1 + SC_POLY_LISTED : 1);
    int held = 0;
    for (int k = 0; k < min(max(F.nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS); k++) held += pb[3 * k + 1] == poly.group;
    if (held > 1) ctr->polyConflict = 1;
}

// Whether a listed item's footprint meets another's (the claims are complete).
__device__ __forceinline__ bool poly_meets(const int *claim, int i, int pmi) {
    return claim[i] != 0 || (pmi >= 0 && claim[pmi] != 1);
}

// The items that share nothing with another, all at once.
__global__ void __launch_bounds__(SC_THREADS) k_poly_apply(ScParams P, const uint32_t *__restrict__ cellStart, PFields F,
                                                           const ScCounters *ctr, const int *__restrict__ list,
                                                           const int *__restrict__ rank, const int *__restrict__ pmiIn,
                                                           const int *claim) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= ctr->polyCount) return;
    const int i = list[slot], pmi = pmiIn[slot];
    if (ctr->polyConflict || poly_meets(claim, i, pmi)) return;
    const int r = rank[slot];
    poly_one(P, cellStart, F, i, ctr->step, pmi, false, r >= 0 ? ctr->lastActive + 1 + r : P.N,
             r >= 0 ? ctr->nextId + r : -1);
}

// The items left, in slot order by one thread, while the others look through
// the list for them; then the claims are cleared and the counters advance:
// lastActive by every creating item (the reference increments it before its
// capacity test), nextId and nActive by those that fit.
__global__ void __launch_bounds__(SC_THREADS) k_poly_finish(ScParams P, const uint32_t *__restrict__ cellStart, PFields F,
                                                            ScCounters *ctr, const int *__restrict__ list,
                                                            const int *__restrict__ rank, const int *__restrict__ pmiIn,
                                                            int *claim) {
    __shared__ int s_left[SC_THREADS];
    const int count = ctr->polyCount;
    if (count == 0) return;
    const int last0 = ctr->lastActive, next0 = ctr->nextId;
    const bool all = ctr->polyConflict != 0;
    for (int k0 = 0; k0 < count; k0 += SC_THREADS) {
        const int k = k0 + threadIdx.x;
        s_left[threadIdx.x] = k < count && (all || poly_meets(claim, list[k], pmiIn[k]));
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int u = 0; u < min(SC_THREADS, count - k0); u++) {
                if (!s_left[u]) continue;
                const int r = rank[k0 + u];
                poly_one(P, cellStart, F, list[k0 + u], ctr->step, pmiIn[k0 + u], true, r >= 0 ? last0 + 1 + r : P.N,
                         r >= 0 ? next0 + r : -1);
            }
        }
        __syncthreads();
    }
    for (int k = threadIdx.x; k < count; k += SC_THREADS)
        if (pmiIn[k] >= 0) claim[pmiIn[k]] = 0;
    if (threadIdx.x) return;
    const int R = ctr->polyCreates;
    const int made = max(0, min(R, P.N - 1 - last0));
    ctr->lastActive = last0 + R;
    ctr->nextId = next0 + made;
    ctr->nActive += made;
    ctr->polyCount = 0;
}

// ---- interactions.cuh:743-822 propagateState (sc_config.propagate_state) -----
// The reference's kernel, whose launch its step leaves commented out
// (main.cu:618-631); it runs after polymerize when the config asks for it.
// Each active particle below the count after polymerize walks its 27 cells in
// order and, for every active neighbour inside the interaction cube that is
// the partner of one of its rule bonds (type >= 10) whose rule sets
// propagateState, takes the neighbour's state and last state-change step when
// that step is later than its own as updated so far.  Neighbours are read
// from the state before the pass (state and lscs are double-buffered).  A
// particle without such a bond keeps its state and scans nothing.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_propagate_state(
    ScParams P, const uint32_t *__restrict__ cellStart, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ pos, const int4 *__restrict__ info, const int *__restrict__ stateIn,
    int *__restrict__ stateOut, const int *__restrict__ lscsIn, int *__restrict__ lscsOut, const int *__restrict__ nb,
    const int *__restrict__ bonds) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    const int4 in = info[i];
    int st = stateIn[i], ls = lscsIn[i];
    const int pnb = min(max(nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
    int partner[SC_MAX_ACTIVE_INTERACTIONS];
    unsigned prop = 0u;  // bit k: bond k propagates
#pragma unroll
    for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++) {
        const int t = k < pnb ? bonds[(size_t)i * 24 + 3 * k] : 0;
        partner[k] = k < pnb ? bonds[(size_t)i * 24 + 3 * k + 2] : 0;
        if (k < pnb && t >= 10 && rule_at(P, t).propagate_state) prop |= 1u << k;
    }
    if ((in.z & SC_ACTIVE) && prop) {
        rep_apply<BATCH>(P, in.w);
        const float4 p4 = pos[i];
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_P);
        scan27(P, cellStart, pp, [&](int j) {
            if (j == i) return;
            const int4 tin = info[j];
            if (!(tin.z & SC_ACTIVE)) return;
            const float4 t4 = pos[j];
            const sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, P.maxInt)) return;
#pragma unroll
            for (int k = 0; k < SC_MAX_ACTIVE_INTERACTIONS; k++) {
                if (((prop >> k) & 1u) && partner[k] == tin.x) {
                    const int tl = lscsIn[j];
                    if (tl > ls) {
                        ls = tl;
                        st = stateIn[j];
                    }
                }
            }
        });
    }
    stateOut[i] = st;
    lscsOut[i] = ls;
}

// ---- metabolites.cuh:352-431 diffuseMetabolites ------------------------------
// List: the metabolic items within maxDiffusionDistance (cube, then sphere),
// built after applyVelocities and read by all diffusion sub-iterations.
__device__ __forceinline__ void build_d_item(const ScParams &P, ScanWords &W, const uint32_t *__restrict__ cellStart, int i,
                                             const float4 *__restrict__ pos, const int4 *__restrict__ info,
                                             uint32_t *list, int &c) {
    float4 p4 = pos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    Imager IM(P, pp, SC_BINNED_M);
    const float lim = P.maxDiff;
    // The items have moved since their sort.  When each moved once, by no
    // more than a cell, the neighbours of an item two cells or more from
    // every face (sorted into cells one or more from it) have not crossed
    // one: no image is nearer than they are.
    if (IM.wrap && P.movedOnce && P.simSize >= 7.0f * P.cell && *P.farMove == 0) {
        const int n = P.nUsed;
        const int cx = (int)sc_grid_idx(pp.x, P.cell, n), cy = (int)sc_grid_idx(pp.y, P.cell, n),
                  cz = (int)sc_grid_idx(pp.z, P.cell, n);
        IM.wrap = min(cx, min(cy, cz)) < 2 || max(cx, max(cy, cz)) > n - 3;
    }
    const sc_sqrt_le within = sc_sqrt_le_make(lim);
    const int limit = min(SC_LIST_D, P.listLimit);
    uint32_t *out = list + sc_list_at(SC_LIST_D, i, 0);
    scan_words(P, W, pos, [&](uint32_t key) { return cellStart[key]; }, pp, reach(P, pp, lim, SC_BINNED_M), lim, IM.wrap,
               [&](int j, float4 t4) {
                   if (j == i || !active_m(P, info, j)) return;
                   sc_f3 delta;
                   if (IM.wrap) {
                       delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
                       if (outside_cube(delta, lim)) return;
                   } else {
                       delta = sc_make_f3(t4.x, t4.y, t4.z) - pp;
                   }
                   if (sc_sqrt_le_test(within, sc_normsq3(delta))) {
                       if (c < limit) *out = (uint32_t)j;
                       out += 32;
                       c++;
                   }
               });
}

template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS, 4) k_build_d(ScParams P, const uint32_t *__restrict__ cellStart,
                                                        const int *__restrict__ nActivePtr,
                                                        const float4 *__restrict__ pos, const int4 *__restrict__ info,
                                                        uint32_t *__restrict__ list, uint32_t *scratch,
                                                        int *__restrict__ cnt, int *__restrict__ perm, int cap,
                                                        int *__restrict__ ovf, int *__restrict__ ovfCount) {
    __shared__ ScanWords W;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < *nActivePtr;
    int c = 0;
    if (valid) {
        const int4 in = info[i];
        ScParams Q = P;
        rep_apply<BATCH>(Q, in.w);
        if (in.z & SC_ACTIVE) build_d_item(Q, W, cellStart, i, pos, info, scratch, c);
    }
    emit_count_ordered<SC_LIST_D>(valid, c, P.listLimit, cap, scratch, list, cnt, perm, ovf, ovfCount);
}

// The full diffusion lists of the overflowed positions (listed by k_build_d;
// their counts are in cnt): each takes a contiguous region of the overflow
// pool by atomicAdd and writes its neighbours there in build_d_item's order,
// for diffuse_pool; a position the pool has no room for keeps offset -1 (it
// scans).  The demand is counted in full for the pool's growth at the next
// synchronisation.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_build_d_ovf(ScParams P0, const uint32_t *__restrict__ cellStart,
                                                            const float4 *__restrict__ pos,
                                                            const int4 *__restrict__ info, const int *__restrict__ ovf,
                                                            const int *__restrict__ ovfCount, const int *__restrict__ cnt,
                                                            const int *__restrict__ perm, long long *__restrict__ ovfOff,
                                                            uint32_t *__restrict__ pool, long long cap,
                                                            unsigned long long *__restrict__ demand) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < *ovfCount; t += gridDim.x * blockDim.x) {
        const int g = ovf[t], i = perm[g], n = cnt[g];
        // regions start on 16-byte boundaries (whole chunks of four entries)
        const unsigned long long n4 = (unsigned long long)((n + 3) & ~3);
        const unsigned long long base = n > 0 ? atomicAdd(demand, n4) : 0ull;
        if (i < 0 || n <= 0 || base + n4 > (unsigned long long)cap) {
            ovfOff[g] = -1;
            continue;
        }
        ovfOff[g] = (long long)base;
        ScParams P = P0;
        rep_apply<BATCH>(P, info[i].w);
        const float4 p4 = pos[i];
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_M);
        const float lim = P.maxDiff;
        const sc_sqrt_le within = sc_sqrt_le_make(lim);
        uint32_t *out = pool + base;
        int k = 0;
        scan27(P, cellStart, pp, reach(P, pp, lim, SC_BINNED_M), [&](int j) {
            if (j == i || !active_m(P, info, j)) return;
            const float4 t4 = pos[j];
            const sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) return;
            if (sc_sqrt_le_test(within, sc_normsq3(delta)) && k < n) out[k++] = (uint32_t)j;
        });
    }
}

// An item's amounts, Q float4 per item: eight-amount rows (32 bytes,
// aligned) in one access.
template <int Q>
__device__ __forceinline__ void met_row(const float4 *__restrict__ met, int j, float4 (&v)[Q]) {
    if (Q == 2) {
        ld_row8(met + (size_t)j * 2, v[0], v[1]);
    } else {
#pragma unroll
        for (int q = 0; q < Q; q++) v[q] = met[(size_t)j * Q + q];
    }
}
template <int SP>
__device__ __forceinline__ void met_store(float4 *__restrict__ met, int i, const float (&pm)[SP]) {
    if (SP == 8) {
        st_row8(met + (size_t)i * 2, make_float4(pm[0], pm[1], pm[2], pm[3]), make_float4(pm[4], pm[5], pm[6], pm[7]));
    } else {
#pragma unroll
        for (int q = 0; q < SP / 4; q++)
            met[(size_t)i * (SP / 4) + q] = make_float4(pm[4 * q], pm[4 * q + 1], pm[4 * q + 2], pm[4 * q + 3]);
    }
}
// One neighbour's amounts against the item's, the first S of SP amounts
// (metabolites.cuh:352-431, the exchange of one pair).
template <int SP>
__device__ __forceinline__ void diffuse_term(const float4 (&v)[SP / 4], const float (&pm)[SP], float (&dm)[SP],
                                             int S) {
#pragma unroll
    for (int q = 0; q < SP / 4; q++) {
        const float tm[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int k = 4 * q + c;
            if (k < S) {
                const float diff = tm[c] - pm[k];
                if (sc_diffuse_exceeds(diff)) dm[k] += diff * 0.1f;
            }
        }
    }
}

// The overflowed diffusion positions (k_build_d), the first entry of each one's
// region of the overflow pool by position (-1: it scans).
struct DiffuseOvf {
    const int *__restrict__ ovf, *__restrict__ count;
    const long long *__restrict__ off;
    const uint32_t *__restrict__ pool;
};

// The positions whose overflowed list is kept whole in the overflow pool
// (k_build_d_ovf), one warp per position, by `blocks` blocks of which this is
// block `blk`: the lanes gather 32 neighbours'
// amounts at once and each computes its neighbour's terms (zero where the
// threshold drops the pair; a kept term is never zero), then lane k adds the
// kept terms of amount k in list order from shared memory -- the sums a
// thread walking the list forms, term by term, while the list's pile-sized
// length costs one gather latency per 32 neighbours instead of per 4.
template <int SP>
__device__ __forceinline__ void diffuse_pool(const ScParams &P, const int4 *__restrict__ info,
                                             const PairList<SC_LIST_D> &L, const DiffuseOvf &O,
                                             const float4 *__restrict__ metIn, float4 *__restrict__ metOut, int blk,
                                             int blocks, float (*sTerm)[32][SP + 1]) {
    constexpr int Q = SP / 4;
    const int *__restrict__ ovf = O.ovf;
    const long long *__restrict__ ovfOff = O.off;
    const uint32_t *__restrict__ ovfPool = O.pool;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int S = P.S;
    const int n = *O.count;
    for (int t = blk * (SC_THREADS / 32) + wid; t < n; t += blocks * (SC_THREADS / 32)) {
        const int g = ovf[t];
        const long long off = ovfOff[g];
        const int i = L.perm[g];
        if (off < 0 || i < 0) continue;   // scanned by k_diffuse
        float pm[SP];
        {
            float4 v[Q];
            met_row<Q>(metIn, i, v);
#pragma unroll
            for (int q = 0; q < Q; q++) {
                pm[4 * q] = v[q].x; pm[4 * q + 1] = v[q].y; pm[4 * q + 2] = v[q].z; pm[4 * q + 3] = v[q].w;
            }
        }
        // lane k's amount and its running sum
        float mine = 0.0f, dm = 0.0f;
#pragma unroll
        for (int k = 0; k < SP; k++)
            if (lane == k) mine = pm[k];
        if (info[i].z & SC_ACTIVE) {
            const int c = L.cnt[g];
            const uint32_t *__restrict__ e = ovfPool + off;
            for (int b = 0; b < c; b += 32) {
                float term[SP];
#pragma unroll
                for (int k = 0; k < SP; k++) term[k] = 0.0f;
                if (b + lane < c) {
                    float4 v[Q];
                    met_row<Q>(metIn, (int)e[b + lane], v);
#pragma unroll
                    for (int q = 0; q < Q; q++) {
                        const float tm[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
                        for (int cc = 0; cc < 4; cc++) {
                            const int k = 4 * q + cc;
                            const float diff = tm[cc] - pm[k];
                            if (k < S && sc_diffuse_exceeds(diff)) term[k] = diff * 0.1f;
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < SP; k++) sTerm[wid][lane][k] = term[k];
                __syncwarp();
                if (lane < S) {
                    const int m = min(32, c - b);
                    for (int u = 0; u < m; u++) {
                        const float x = sTerm[wid][u][lane];
                        if (x != 0.0f) dm += x;
                    }
                }
                __syncwarp();
            }
            if (lane < S) mine += dm;
        }
        if (lane < SP) reinterpret_cast<float *>(metOut)[(size_t)i * SP + lane] = mine;
    }
}

template <int SP>
__global__ void __launch_bounds__(SC_THREADS) k_diffuse_pool(ScParams P, const int4 *__restrict__ info,
                                                             PairList<SC_LIST_D> L, DiffuseOvf O,
                                                             const float4 *__restrict__ metIn,
                                                             float4 *__restrict__ metOut) {
    __shared__ float sTerm[SC_THREADS / 32][32][SP + 1];
    if (*O.count > 0) diffuse_pool<SP>(P, info, L, O, metIn, metOut, blockIdx.x, gridDim.x, sTerm);
}

// With POOL the first `extra` blocks take the positions of the overflow pool
// (they write other items and read what the others read; the longest lists
// start first); k_diffuse_pool takes them otherwise: its shared memory in this
// kernel takes L1 from the gathers that bound it (large workload: 330 -> 361 us
// a launch), while a sim that does not fill the device saves a launch.
// Inactive items' amounts are copied until both buffers hold them (age:
// launches since the amounts were last out of step).  Twelve amounts keep to
// three blocks per SM without spills (983,041 items, 118 us a launch with four
// rows in flight, 106 us with two at four blocks, 97 us so).  Eight and four
// amounts fit as they are, in a loop of their own: written as one with the
// twelve's, the eight's spills (8,388,608 items 334 -> 407 us).
template <int SP, bool BATCH, bool POOL>
__global__ void __launch_bounds__(SC_THREADS, SP == 12 ? 3 : 0) k_diffuse(ScParams P, const uint32_t *__restrict__ cellStart,
                                                        const int *__restrict__ nActivePtr,
                                                        const float4 *__restrict__ pos, const int4 *__restrict__ info,
                                                        PairList<SC_LIST_D> L, const float4 *__restrict__ metIn,
                                                        float4 *__restrict__ metOut, DiffuseOvf O, int extra, int age) {
    constexpr int Q = SP / 4;
    if constexpr (POOL) {
        __shared__ float sTerm[SC_THREADS / 32][32][SP + 1];   // odd row length: no bank conflicts either way
        if ((int)blockIdx.x < extra) {
            if (*O.count > 0) diffuse_pool<SP>(P, info, L, O, metIn, metOut, blockIdx.x, extra, sTerm);
            return;
        }
    }
    const int g = ((int)blockIdx.x - extra) * SC_THREADS + threadIdx.x;   // list position (count-ordered)
    if (g >= *nActivePtr) return;
    const int i = L.perm[g];
    if (i < 0) return;
    if (BATCH) rep_apply<BATCH>(P, info[i].w);
    float pm[SP];
    {
        float4 v[Q];
        met_row<Q>(metIn, i, v);
#pragma unroll
        for (int q = 0; q < Q; q++) {
            pm[4 * q] = v[q].x; pm[4 * q + 1] = v[q].y; pm[4 * q + 2] = v[q].z; pm[4 * q + 3] = v[q].w;
        }
    }
    // after the sort the active items are exactly the binned ones
    const bool act = P.mAllActive ? i < (int)cellStart[P.cells] : (info[i].z & SC_ACTIVE) != 0;
    if (!act) {
        if (age > 0) return;
        met_store<SP>(metOut, i, pm);   // the amounts' bits, unchanged
        return;
    }
    float dm[SP];
#pragma unroll
    for (int k = 0; k < SP; k++) dm[k] = 0.0f;
    const int S = P.S;
    const int c = L.cnt[g];
    if (c <= min(SC_LIST_D, P.listLimit)) {
        const uint4 *__restrict__ chunks = sc_list4_chunks(L.list, SC_LIST_D, g);
        uint4 E = c > 0 ? chunks[0] : make_uint4(0, 0, 0, 0);
        // four entries per list load; their amounts are gathered together (two
        // and two of twelve amounts, which would spill) and the next chunk of
        // the list is loaded while this one is applied
        for (int k0 = 0; k0 < c; k0 += 4) {
            const uint4 En = k0 + 4 < c ? chunks[(size_t)(k0 / 4 + 1) * 32] : make_uint4(0, 0, 0, 0);
            const int e[4] = {(int)E.x, (int)E.y, (int)E.z, (int)E.w};
            if constexpr (SP == 12) {
#pragma unroll
                for (int h = 0; h < 4; h += 2) {
                    float4 v[2][Q];
#pragma unroll
                    for (int kk = 0; kk < 2; kk++)
                        if (k0 + h + kk < c) met_row<Q>(metIn, e[h + kk], v[kk]);
#pragma unroll
                    for (int kk = 0; kk < 2; kk++) {
                        if (k0 + h + kk >= c) break;
                        diffuse_term<SP>(v[kk], pm, dm, S);
                    }
                }
                E = En;
                continue;
            }
            float4 v[4][Q];
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
                if (k0 + kk < c) met_row<Q>(metIn, e[kk], v[kk]);
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                if (k0 + kk >= c) break;
                diffuse_term<SP>(v[kk], pm, dm, S);
            }
            E = En;
        }
    } else if (O.off && O.off[g] >= 0) {
        return;   // an overflowed list kept whole in the overflow pool: diffuse_pool
    } else {
        float4 p4 = pos[i];
        const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
        const Imager IM(P, pp, SC_BINNED_M);
        const float lim = P.maxDiff;
        const sc_sqrt_le within = sc_sqrt_le_make(lim);
        scan27(P, cellStart, pp, reach(P, pp, lim, SC_BINNED_M), [&](int j) {
            if (j == i) return;
            if (!active_m(P, info, j)) return;
            float4 t4 = pos[j];
            sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
            if (outside_cube(delta, lim)) return;
            if (sc_sqrt_le_test(within, sc_normsq3(delta))) {
                float4 v[Q];
                met_row<Q>(metIn, j, v);
                diffuse_term<SP>(v, pm, dm, S);
            }
        });
    }
#pragma unroll
    for (int k = 0; k < SP; k++)
        if (k < S) pm[k] += dm[k];
    met_store<SP>(metOut, i, pm);
}

// ---- metabolites.cuh:18-88 removeInterferingMetabolicParticles -------------
// Only the item's own flags change and no other thread reads metabolic
// flags here: updated in place.
template <bool BATCH>
__global__ void __launch_bounds__(SC_THREADS) k_remove_interfering(
    ScParams P, const uint32_t *__restrict__ cellStartP, const int *__restrict__ nActivePtr,
    const float4 *__restrict__ mpos, int4 *__restrict__ minfo, const float4 *__restrict__ ppos_,
    const int4 *__restrict__ pinfo) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nActivePtr) return;
    int4 in = minfo[i];
    if (!(in.z & SC_ACTIVE)) return;
    rep_apply<BATCH>(P, in.w);
    float4 p4 = mpos[i];
    const sc_f3 pp = sc_make_f3(p4.x, p4.y, p4.z);
    const Imager IM(P, pp, SC_BINNED_P);
    const float prad = p4.w;
    int flags = in.z;
    const float lim = P.maxInt;
    scan27(P, cellStartP, pp, reach(P, pp, lim, SC_BINNED_P), [&](int j) {
        if (!active_lipid(P, pinfo, j)) return;
        float4 t4 = ppos_[j];
        sc_f3 delta = IM(sc_make_f3(t4.x, t4.y, t4.z)) - pp;
        if (outside_cube(delta, lim)) return;
        float dist = sc_norm3(delta);
        float interf = (float)((double)(prad + t4.w) + 0.001);
        if (dist <= interf) flags = flags & ~SC_ACTIVE;
    });
    if (flags != in.z) minfo[i].z = flags;
}

// ---- dynamics.cuh:824-844 reduceParticles (frames.dat records) --------------
__device__ __forceinline__ void reduce_common(sc_reduced_particle &r, int4 in, int state, float4 p4, float4 r4,
                                              float4 d4) {
    r.id = in.x;
    r.type = in.y;
    r.flags = in.z | (((int)(int8_t)state & 0x0000000F) << 16);
    r.radius = sc_f2h(p4.w);
    r.pos[0] = sc_f2h(p4.x); r.pos[1] = sc_f2h(p4.y); r.pos[2] = sc_f2h(p4.z);
    r.rot[0] = sc_f2h(r4.x); r.rot[1] = sc_f2h(r4.y); r.rot[2] = sc_f2h(r4.z); r.rot[3] = sc_f2h(r4.w);
    r.debug_vector[0] = sc_f2h(d4.x); r.debug_vector[1] = sc_f2h(d4.y);
    r.debug_vector[2] = sc_f2h(d4.z); r.debug_vector[3] = sc_f2h(d4.w);
}

__global__ void __launch_bounds__(SC_THREADS) k_reduce_particles(const int *__restrict__ nActivePtr, int cap,
                                                                 PFields F, sc_reduced_particle *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cap) return;
    sc_reduced_particle r;
    memset(&r, 0, sizeof r);
    if (i < *nActivePtr) reduce_common(r, F.info[i], F.state[i], F.pos[i], F.rot[i], F.dbg[i]);
    out[i] = r;
}

__global__ void __launch_bounds__(SC_THREADS) k_reduce_metabolic(const int *__restrict__ nActivePtr, int cap, int sp4,
                                                                 MFields F, sc_reduced_metabolic_particle *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cap) return;
    sc_reduced_metabolic_particle r;
    memset(&r, 0, sizeof r);
    if (i < *nActivePtr) {
        reduce_common(r.p, F.info[i], F.state[i], F.pos[i], F.rot[i], F.dbg[i]);
        float4 m = F.met[(size_t)i * sp4];
        r.metabolites[0] = sc_f2h(m.x); r.metabolites[1] = sc_f2h(m.y);
        r.metabolites[2] = sc_f2h(m.z); r.metabolites[3] = sc_f2h(m.w);
    }
    out[i] = r;
}

// ---- launchers ------------------------------------------------------------------
static inline int nblocks(int n) { return (n + SC_THREADS - 1) / SC_THREADS; }

// The instantiation of a kernel for this launch: replica-aware in batched sims.
#define SC_BATCHED(kern) (c.P.nRep > 1 ? kern<true> : kern<false>)

void sc_phase_move_brownian(ScLaunchCtx &c, bool metabolic) {
    ScBuffers &B = *c.B;
    if (!metabolic) {
        PFields F = B.P();
        if (c.P.N <= 0) return;
        SC_BATCHED(k_move_brownian)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(&B.ctr->nActive, F.info, F.pos, F.dbg, F.posnoise,
                                                                  F.angnoise, c.P, c.P.moveNoise, SC_STREAM_P_UNIFORM,
                                                                  SC_STREAM_P_NORMAL, &B.ctr->step);
    } else {
        MFields F = B.M();
        if (c.P.Nm <= 0) return;
        SC_BATCHED(k_move_brownian)<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(&B.ctr->nActiveM, F.info, F.pos, F.dbg, F.posnoise,
                                                                   F.angnoise, c.P, c.P.metabNoise,
                                                                   SC_STREAM_M_UNIFORM, SC_STREAM_M_NORMAL,
                                                                   &B.ctr->step);
    }
    (*c.launches)++;
}

static PairList<SC_LIST_PP> pp_list(const ScLaunchCtx &c) {
    PairList<SC_LIST_PP> L;
    L.list = c.B->listPP;
    L.cnt = c.B->cntPP;
    L.cap = c.P.N;
    L.perm = nullptr;
    return L;
}

static void ensure_pp(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (B.validPP) return;
    PFields F = B.P();
    cudaMemsetAsync(B.ctr->ppClassCount, 0, sizeof(B.ctr->ppClassCount) + sizeof(B.ctr->ovfPP), c.st);
    SC_BATCHED(k_build_pp)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, &B.ctr->nActive, F.pos, F.info, F.nb,
                                                         F.bonds, B.listPP, B.cntPP, c.P.N, B.classPP,
                                                         B.ctr->ppClassCount, B.ovfPP, &B.ctr->ovfPP, B.matchPP,
                                                         B.matchN, B.geoPP);
    k_bond_plan<<<std::min(nblocks(c.P.N), c.gridCap), SC_THREADS, 0, c.st>>>(
        c.P, pp_list(c), B.classPP, B.ctr->ppClassCount, F.bonds, B.matchPP, B.matchN, B.bondRec);
    (*c.launches) += 2;
    B.validPP = true;
    B.relaxAge = B.noiseAge = 0;
}

// Every list of the relaxation in one launch (k_build_all), where none is built
// and the blocks fit the device at four per SM.  A launch each and so, ten
// steps: 4,096 + 8,192 items 7.7 / 6.9 ms, 38,000 + 76,000 10.4 / 9.5; with four
// sims in flight 2.35 / 2.10 and 5.88 / 5.74, but 65,536 + 131,072 6.82 / 6.91.
// Streams of their own beside the noise phases gain as much for one sim and
// lose for several (4,096, four in flight: 2.9 ms).
void sc_phase_build_all(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    const int nbP = nblocks(c.P.N), nbM = nblocks(c.P.Nm);
    if (c.P.N <= 0 || c.P.Nm <= 0 || nbM + 2 * nbP > c.gridCap / 2 || c.P.tileCapM > 0 || c.P.metabLean ||
        !B.scratchApart || B.validPP || B.validM || B.validLM)
        return;
    MFields M = B.M();
    PFields F = B.P();
    // every counter of the lists: the diffusion's too, which the builds' scratch invalidates
    cudaMemsetAsync(B.ctr->ppClassCount, 0, sizeof(ScCounters) - offsetof(ScCounters, ppClassCount), c.st);
    const CombStart cs{B.cellStartM, B.cellStartP};
    k_combine<<<(int)std::min<long long>(((long long)c.P.N + c.P.Nm + SC_THREADS - 1) / SC_THREADS, 8 * c.gridCap),
                SC_THREADS, 0, c.st>>>(c.P, B.keysM[B.sortCurM], B.keysP[B.sortCurP], cs, M.pos, M.info, F.pos, F.info,
                                       B.comb);
    k_lipid_select<<<nbP, SC_THREADS, 0, c.st>>>(&B.ctr->nActive, F.info, B.workP, &B.ctr->workCount);
    SC_BATCHED(k_build_all)<<<nbM + 2 * nbP, SC_THREADS, 0, c.st>>>(
        c.P, nbM, nbP, cs, B.comb, &B.ctr->nActiveM, &B.ctr->nActive, M.pos, M.info, F.pos, F.info,
        B.listM, (long long)B.poolCapM, &B.ctr->poolM, B.warpOffM, B.listD, B.cntM, B.permM, B.ovfM, &B.ctr->ovfM, B.ovfNM,
        B.workP, &B.ctr->workCount, reinterpret_cast<uint4 *>(B.listLM),
        (long long)(sc_list_words(SC_LIST_LM, c.P.N) / 4), &B.ctr->poolLM, B.warpOffLM, B.scratchLM, B.cntLM, B.permLM,
        F.nb, F.bonds, B.listPP, B.cntPP, B.classPP, B.ctr->ppClassCount, B.ovfPP, &B.ctr->ovfPP, B.matchPP, B.matchN,
        B.geoPP);
    k_bond_plan<<<std::min(nbP, c.gridCap), SC_THREADS, 0, c.st>>>(
        c.P, pp_list(c), B.classPP, B.ctr->ppClassCount, F.bonds, B.matchPP, B.matchN, B.bondRec);
    SC_BATCHED(k_build_m_ovf)<<<std::min(nbM, c.gridCap / 4), SC_THREADS, 0, c.st>>>(
        c.P, B.cellStartM, B.cellStartP, M.pos, M.info, F.pos, F.info, B.ovfM, &B.ctr->ovfM, B.ovfNM, B.ovfOffM,
        B.ovfPoolM, (long long)B.ovfPoolCapM, &B.ctr->poolOvfM);
    (*c.launches) += 5;
    B.validPP = B.validM = B.validLM = true;
    B.validD = false;
    B.relaxAge = B.noiseAge = 0;
}

void sc_phase_coordinate_noise(ScLaunchCtx &c, float frac) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    ensure_pp(c);
    PFields F = B.P(), X = B.Pnext();
    const int g = std::min(nblocks(c.P.N), c.gridCap);
    SC_BATCHED(k_coordinate_noise)<<<g, SC_THREADS, 0, c.st>>>(
        c.P, B.cellStartP, &B.ctr->nActive, B.classPP, B.ctr->ppClassCount, F.pos, F.info, F.nb, F.bonds, pp_list(c),
        B.matchPP, B.matchN, F.posnoise, F.angnoise, X.posnoise, X.angnoise, frac, B.noiseAge);
    (*c.launches)++;
    B.noiseAge = 1;
    B.cp[FP_POSNOISE] ^= 1;
    B.cp[FP_ANGNOISE] ^= 1;
}

void sc_phase_apply_noise(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N > 0) {
        PFields F = B.P();
        k_apply_noise<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(&B.ctr->nActive, F.info, F.vel, F.posnoise, F.angvel,
                                                                F.angnoise);
        (*c.launches)++;
    }
    if (c.P.Nm > 0) {
        MFields M = B.M();
        k_apply_noise<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(&B.ctr->nActiveM, M.info, M.vel, M.posnoise,
                                                                 M.angvel, M.angnoise);
        (*c.launches)++;
    }
}

void sc_phase_relax(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    ensure_pp(c);
    PFields F = B.P(), X = B.Pnext();
    RelaxArgs A{B.cellStartP, F.pos, F.info, F.nb, F.bonds, pp_list(c),
                F.vel, F.rot, F.angvel, X.vel, X.rot, X.angvel, F.dbg, B.classPP, B.ctr->ppClassCount,
                B.matchPP, B.matchN, B.geoPP, B.bondRec, B.ovfPP, &B.ctr->ovfPP, &B.ctr->ppClassCount[3], B.relaxAge};
    const int nb = nblocks(c.P.N);
    const bool batch = c.P.nRep > 1;
    if (c.side[0]) {
        // particles that fill the device: a kernel per class, each at its own
        // occupancy, on three streams
        cudaEventRecord(c.fork, c.st);
        cudaStreamWaitEvent(c.side[0], c.fork, 0);
        cudaStreamWaitEvent(c.side[1], c.fork, 0);
        const int g = std::min(nb, c.gridCap);
        (batch ? k_relax<0, true> : k_relax<0, false>)<<<std::min(12 * nb, 6 * c.gridCap), relax_threads(0), 0,
                                                         c.st>>>(c.P, A);
        (batch ? k_relax<2, true> : k_relax<2, false>)<<<g, SC_THREADS, 0, c.side[0]>>>(c.P, A);
        (batch ? k_relax<1, true> : k_relax<1, false>)<<<g, SC_THREADS, 0, c.side[1]>>>(c.P, A);
        cudaEventRecord(c.join[0], c.side[0]);
        cudaEventRecord(c.join[1], c.side[1]);
        cudaStreamWaitEvent(c.st, c.join[0], 0);
        cudaStreamWaitEvent(c.st, c.join[1], 0);
        (*c.launches) += 2;
    } else {
        // fewer: one launch, with more threads per polar item while the
        // particles take less than a block per SM (milliseconds a step with
        // and without, at 1 : 2 metabolic items: 4,096 0.86 / 0.95, 32,000
        // 1.03 / 1.09, 45,000 1.20 / 1.21, 65,536 1.41 / 1.30)
        const bool lanes = nb <= c.gridCap / (2048 / SC_THREADS);
        auto kern = lanes ? (batch ? k_relax<SC_RELAX_ALL_LANES, true> : k_relax<SC_RELAX_ALL_LANES, false>)
                          : (batch ? k_relax<SC_RELAX_ALL, true> : k_relax<SC_RELAX_ALL, false>);
        kern<<<std::min((2 + (lanes ? SC_POLAR_LANES : 1)) * nb + 4, c.gridCap), SC_THREADS, 0, c.st>>>(c.P, A);
    }
    B.relaxAge = std::min(B.relaxAge + 1, 2);
    B.cp[FP_VEL] ^= 1;
    B.cp[FP_ROT] ^= 1;
    B.cp[FP_ANGVEL] ^= 1;
    (*c.launches)++;
}

// Largest dynamic shared memory of the tile kernels; called once per device.
void sc_tile_init() {
    const int most = 227 * 1024;
    cudaFuncSetAttribute(k_build_m_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    cudaFuncSetAttribute(k_relax_metab_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}
size_t sc_tile_bytes(int capM, int capP, int perSlot) { return SC_TILE_HDR_BYTES + (size_t)(capM + capP) * perSlot; }

// The metabolic relaxation's pair list (and pool) for the current
// positions, unless it is already built.
void sc_phase_build_m(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.Nm <= 0) return;
    MFields M = B.M();
    PFields F = B.P();
    const bool tiles = c.P.tileCapM > 0;
    if (!B.validM) {
        // the diffusion list's buffer is the build scratch (that list is rebuilt after the next move anyway)
        B.validD = false;
        cudaMemsetAsync(&B.ctr->ovfM, 0, sizeof(int), c.st);
        cudaMemsetAsync(&B.ctr->poolM, 0, sizeof(B.ctr->poolM) + sizeof(B.ctr->poolOvfM), c.st);
        if (tiles) {
            k_build_m_tile<<<tile_blocks(c.P), SC_THREADS, sc_tile_bytes(c.P.tileCapM, c.P.tileCapP, 17), c.st>>>(
                c.P, B.cellStartM, B.cellStartP, M.pos, M.info, F.pos, F.info, reinterpret_cast<uint16_t *>(B.listM),
                B.cntM, B.ovfM, &B.ctr->ovfM);
        } else {
            const CombStart cs{B.cellStartM, B.cellStartP};
            k_combine<<<(int)std::min<long long>(((long long)c.P.N + c.P.Nm + SC_THREADS - 1) / SC_THREADS, 8 * c.gridCap),
                        SC_THREADS, 0, c.st>>>(c.P, B.keysM[B.sortCurM], B.keysP[B.sortCurP], cs, M.pos, M.info, F.pos,
                                               F.info, B.comb);
            (*c.launches)++;
            (c.P.nRep > 1 ? (c.P.metabLean ? k_build_m<true, true> : k_build_m<false, true>)
                          : (c.P.metabLean ? k_build_m<true, false> : k_build_m<false, false>))<<<
                nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(
                c.P, cs, B.comb, &B.ctr->nActiveM, M.pos, M.info, F.pos, B.listM, (long long)B.poolCapM, &B.ctr->poolM,
                B.warpOffM, B.listD, B.cntM, B.permM, c.P.Nm, B.ovfM, &B.ctr->ovfM, B.ovfNM);
            // the overflowed items' full lists
            SC_BATCHED(k_build_m_ovf)<<<std::min(nblocks(c.P.Nm), c.gridCap / 4), SC_THREADS, 0, c.st>>>(
                c.P, B.cellStartM, B.cellStartP, M.pos, M.info, F.pos, F.info, B.ovfM, &B.ctr->ovfM, B.ovfNM,
                B.ovfOffM, B.ovfPoolM, (long long)B.ovfPoolCapM, &B.ctr->poolOvfM);
            (*c.launches)++;
        }
        (*c.launches)++;
        B.validM = true;
    }
}

void sc_phase_relax_metab(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.Nm <= 0) return;
    MFields M = B.M(), X = B.Mnext();
    PFields F = B.P();
    const bool tiles = c.P.tileCapM > 0;
    sc_phase_build_m(c);
    PairList<SC_LIST_M> L;
    L.list = B.listM;
    L.cnt = B.cntM;
    L.cap = c.P.Nm;
    L.perm = tiles ? nullptr : B.permM;
    RelaxMArgs A{B.cellStartM, B.cellStartP, &B.ctr->nActiveM, M.pos, M.info, L, M.vel, X.vel, F.pos, F.info, F.vel,
                 reinterpret_cast<const uint4 *>(B.listM), B.warpOffM, B.ovfM, &B.ctr->ovfM, B.ovfNM,
                 tiles ? nullptr : B.ovfOffM, B.ovfPoolM, B.relaxMAge};
    const int nb = nblocks(c.P.Nm);
    if (tiles) {
        k_relax_metab_tile<<<tile_blocks(c.P), SC_THREADS, sc_tile_bytes(c.P.tileCapM, c.P.tileCapP, 32), c.st>>>(
            c.P, A, reinterpret_cast<const uint16_t *>(B.listM), &B.ctr->error);
        k_copy_tail<<<std::max(1, c.gridCap / 8), SC_THREADS, 0, c.st>>>(
            B.cellStartM + c.P.cells, &B.ctr->nActiveM, M.vel, X.vel);
        SC_BATCHED(k_relax_metab_overflow)<<<std::min(nb, c.gridCap / 4), SC_THREADS, 0, c.st>>>(c.P, A);
        (*c.launches) += 3;
    } else {
        // 256 items times this a block of the sweep: up to eight where that
        // leaves four waves of blocks (8,388,608 items 414 us a launch at one,
        // 386 at four, 383 at eight), one below, where fewer blocks than the
        // device holds cost more (500,009 items, five steps: 11.9 ms at one,
        // 12.4 at four)
        const int sweep = std::max(1, std::min(8, nb / (2 * c.gridCap)));
        const bool batch = c.P.nRep > 1, small = nb <= c.gridCap / 4;   // at most two blocks per SM: all resident at G = 8
        const int extra = small ? std::min(nb, c.gridCap / 2) : 0;
        auto *const lean = batch ? (small ? k_relax_metab_lean<true, true> : k_relax_metab_lean<true, false>)
                                 : (small ? k_relax_metab_lean<false, true> : k_relax_metab_lean<false, false>);
        if (c.P.metabLean)
            lean<<<extra + nb, SC_THREADS, 0, c.st>>>(c.P, A, extra);
        else if (small)
            (batch ? k_relax_metab<8, true> : k_relax_metab<8, false>)<<<extra + nb, SC_THREADS, 0, c.st>>>(c.P, A, extra,
                                                                                                          8);
        else
            (batch ? k_relax_metab<4, true> : k_relax_metab<4, false>)<<<(nb + sweep - 1) / sweep, SC_THREADS, 0,
                                                                         c.st>>>(c.P, A, 0, 8 * sweep);
        (*c.launches)++;
        if (!extra) {
            SC_BATCHED(k_relax_metab_overflow)<<<std::min(nb, c.gridCap), SC_THREADS, 0, c.st>>>(c.P, A);
            (*c.launches)++;
        }
    }
    B.relaxMAge = 1;
    B.cm[FM_VEL] ^= 1;
}

// The lipid-metabolic pair list of relax_partners, unless it is already built.
void sc_phase_build_lm(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    MFields M = B.M();
    PFields F = B.P();
    if (!B.validLM) {
        if (B.scratchInD) B.validD = false;
        cudaMemsetAsync(&B.ctr->poolLM, 0, sizeof(B.ctr->poolLM) + sizeof(B.ctr->workCount), c.st);
        k_lipid_select<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(&B.ctr->nActive, F.info, B.workP, &B.ctr->workCount);
        SC_BATCHED(k_build_lm)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(
            c.P, B.cellStartM, B.workP, &B.ctr->workCount, F.info, F.pos, M.pos, M.info,
            reinterpret_cast<uint4 *>(B.listLM),
            (long long)(sc_list_words(SC_LIST_LM, c.P.N) / 4), &B.ctr->poolLM, B.warpOffLM, B.scratchLM, B.cntLM, B.permLM,
            c.P.N);
        (*c.launches)++;
        (*c.launches)++;
        B.validLM = true;
    }
}

void sc_phase_relax_partners(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    MFields M = B.M();
    PFields F = B.P();
    sc_phase_build_lm(c);
    PairList<SC_LIST_LM> L;
    L.list = B.listLM;
    L.cnt = B.cntLM;
    L.cap = c.P.N;
    L.perm = B.permLM;
    SC_BATCHED(k_relax_partners)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(c.P, B.cellStartM, &B.ctr->nActive, F.pos, F.info,
                                                               F.vel, L, reinterpret_cast<const uint4 *>(B.listLM),
                                                               B.warpOffLM, M.pos, M.info, M.vel);
    (*c.launches)++;
}

void sc_phase_apply_velocities(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N > 0) {
        PFields F = B.P();
        SC_BATCHED(k_apply_velocities)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(&B.ctr->nActive, F.info, F.pos, F.vel, F.rot,
                                                                     F.angvel, c.P, 0.45f, nullptr);
        (*c.launches)++;
    }
    if (c.P.Nm > 0) {
        MFields M = B.M();
        SC_BATCHED(k_apply_velocities)<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(&B.ctr->nActiveM, M.info, M.pos, M.vel, M.rot,
                                                                      M.angvel, c.P, 0.45f, &B.ctr->farMove);
        (*c.launches)++;
    }
}

void sc_phase_complexify(ScLaunchCtx &c, bool prep) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    PFields F = B.P(), X = B.Pnext();
    cudaMemsetAsync(&B.ctr->workCount, 0, sizeof(int), c.st);
    k_complexify_select<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(c.P, &B.ctr->nActive, F.info, F.nb, X.nb, F.bonds,
                                                                  B.workP, &B.ctr->workCount);
    const int blocks = std::min(nblocks(c.P.N), c.gridCap);
    if (!c.P.pairClaim) {
        SC_BATCHED(k_complexify)<<<blocks, SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, B.workP, &B.ctr->workCount, F.pos, F.rot,
                                                      F.info, F.state, F.nb, X.nb, F.bonds, &B.ctr->step, prep);
        (*c.launches) += 2;
    } else {
        cudaMemsetAsync(B.claimP, 0xff, (size_t)c.P.N * sizeof(unsigned long long), c.st);
        SC_BATCHED(k_claim_offer)<<<std::min(nblocks(c.P.N) * 11, 4 * c.gridCap), SC_THREADS, 0, c.st>>>(
            c.P, B.cellStartP, B.workP, &B.ctr->workCount, F.pos, F.rot, F.info, F.state, F.nb, F.bonds, &B.ctr->step,
            prep, B.claimP);
        SC_BATCHED(k_claim_bind)<<<blocks, SC_THREADS, 0, c.st>>>(c.P, B.workP, &B.ctr->workCount, F.pos, F.rot, F.info, F.state,
                                                      F.nb, X.nb, F.bonds, &B.ctr->step, prep, B.claimP);
        (*c.launches) += 3;
    }
    B.cp[FP_NB] ^= 1;
}

void sc_phase_transition(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    PFields F = B.P(), X = B.Pnext();
    SC_BATCHED(k_transition)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, &B.ctr->nActive, &B.ctr->step, F.pos, F.rot,
                                                           F.info, F.state, X.state, F.nb, X.nb, F.bonds, X.bonds,
                                                           F.lscs, F.spoly);
    B.cp[FP_STATE] ^= 1;
    B.cp[FP_NB] ^= 1;
    B.cp[FP_BONDS] ^= 1;
    (*c.launches)++;
}

void sc_phase_polymerize(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0 || !c.mayPolymerize) return;
    PFields F = B.P();
    const int nb = nblocks(c.P.N);
    k_poly_count<<<nb, SC_THREADS, 0, c.st>>>(c.P, F, B.ctr, B.polyBlk);
    k_poly_offsets<<<1, SC_POLY_SCAN_THREADS, 0, c.st>>>(B.polyBlk, B.polyBlk + nb, nb, B.ctr);
    k_poly_plan<<<nb, SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, F, B.ctr, B.polyBlk + nb, B.polyList, B.polyRank,
                                             B.polyPmi, B.polyClaim);
    k_poly_apply<<<nb, SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, F, B.ctr, B.polyList, B.polyRank, B.polyPmi,
                                              B.polyClaim);
    k_poly_finish<<<1, SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, F, B.ctr, B.polyList, B.polyRank, B.polyPmi,
                                              B.polyClaim);
    (*c.launches) += 5;
}

void sc_phase_propagate_state(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.N <= 0) return;
    PFields F = B.P(), X = B.Pnext();
    SC_BATCHED(k_propagate_state)<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(
        c.P, B.cellStartP, &B.ctr->nActive, F.pos, F.info, F.state, X.state, F.lscs, X.lscs, F.nb, F.bonds);
    B.cp[FP_STATE] ^= 1;
    B.cp[FP_LSCS] ^= 1;
    (*c.launches)++;
}

void sc_phase_diffuse(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.Nm <= 0) return;
    MFields M = B.M(), X = B.Mnext();
    if (!B.validD) {
        // the build scratch follows the list in the same buffer
        cudaMemsetAsync(&B.ctr->ovfD, 0, sizeof(int), c.st);
        cudaMemsetAsync(&B.ctr->poolOvfD, 0, sizeof(B.ctr->poolOvfD), c.st);
        SC_BATCHED(k_build_d)<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(c.P, B.cellStartM, &B.ctr->nActiveM, M.pos, M.info,
                                                             B.listD, B.listD + sc_list_words(SC_LIST_D, c.P.Nm),
                                                             B.cntD, B.permD, c.P.Nm, B.ovfD, &B.ctr->ovfD);
        SC_BATCHED(k_build_d_ovf)<<<std::min(nblocks(c.P.Nm), c.gridCap / 4), SC_THREADS, 0, c.st>>>(
            c.P, B.cellStartM, M.pos, M.info, B.ovfD, &B.ctr->ovfD, B.cntD, B.permD, B.ovfOffD, B.ovfPoolD,
            (long long)B.ovfPoolCapD, &B.ctr->poolOvfD);
        (*c.launches) += 2;
        B.validD = true;
    }
    PairList<SC_LIST_D> L;
    L.list = B.listD;
    L.cnt = B.cntD;
    L.cap = c.P.Nm;
    L.perm = B.permD;
    const DiffuseOvf O{B.ovfD, &B.ctr->ovfD, B.ovfOffD, B.ovfPoolD};
    const int nb = nblocks(c.P.Nm);
    const bool batch = c.P.nRep > 1, fork = c.side[0] != nullptr;
    const int extra = fork ? 0 : std::min(nb, c.gridCap / 2);
    if (fork) {   // beside the others on a side stream
        cudaEventRecord(c.fork, c.st);
        cudaStreamWaitEvent(c.side[0], c.fork, 0);
        auto pool = c.P.SP == 4 ? k_diffuse_pool<4> : c.P.SP == 8 ? k_diffuse_pool<8> : k_diffuse_pool<12>;
        pool<<<std::min(nb, c.gridCap), SC_THREADS, 0, c.side[0]>>>(c.P, M.info, L, O, M.met, X.met);
        (*c.launches)++;
    }
    auto kern =
        c.P.SP == 4 ? (fork ? (batch ? k_diffuse<4, true, false> : k_diffuse<4, false, false>)
                            : (batch ? k_diffuse<4, true, true> : k_diffuse<4, false, true>))
        : c.P.SP == 8 ? (fork ? (batch ? k_diffuse<8, true, false> : k_diffuse<8, false, false>)
                              : (batch ? k_diffuse<8, true, true> : k_diffuse<8, false, true>))
                      : (fork ? (batch ? k_diffuse<12, true, false> : k_diffuse<12, false, false>)
                              : (batch ? k_diffuse<12, true, true> : k_diffuse<12, false, true>));
    kern<<<extra + nb, SC_THREADS, 0, c.st>>>(c.P, B.cellStartM, &B.ctr->nActiveM, M.pos, M.info, L, M.met, X.met, O,
                                              extra, B.diffuseAge);
    if (fork) {
        cudaEventRecord(c.join[0], c.side[0]);
        cudaStreamWaitEvent(c.st, c.join[0], 0);
    }
    B.diffuseAge = 1;
    B.cm[FM_MET] ^= 1;
    (*c.launches)++;
}

void sc_phase_remove_interfering(ScLaunchCtx &c) {
    ScBuffers &B = *c.B;
    if (c.P.Nm <= 0) return;
    MFields M = B.M();
    PFields F = B.P();
    SC_BATCHED(k_remove_interfering)<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(c.P, B.cellStartP, &B.ctr->nActiveM, M.pos, M.info,
                                                                    F.pos, F.info);
    (*c.launches)++;
}

void sc_phase_reduce(ScLaunchCtx &c, int slot) {
    ScBuffers &B = *c.B;
    if (c.P.N > 0) {
        k_reduce_particles<<<nblocks(c.P.N), SC_THREADS, 0, c.st>>>(&B.ctr->nActive, c.P.N, B.P(),
                                                                     slot ? B.redP2 : B.redP);
        (*c.launches)++;
    }
    if (c.P.Nm > 0) {
        k_reduce_metabolic<<<nblocks(c.P.Nm), SC_THREADS, 0, c.st>>>(&B.ctr->nActiveM, c.P.Nm, c.P.SP / 4, B.M(),
                                                                      slot ? B.redM2 : B.redM);
        (*c.launches)++;
    }
}
