// sc_grid.cu -- grid binning of the step on sm_103a (grid.cuh:13-139 of the
// reference, whose version is updateIndices -> CUB SortPairs of the whole
// 256/304-byte struct over all 32 key bits -> memset + updateGridRanges).
//
// Here:
//   1. k_sort_keys: cell key of every slot (inactive -> all-ones in the used
//      bits) and the digit histograms of every pass, one read of pos + info;
//   2. k_onesweep: one LSD pass per 8-bit digit over only the 3*bits+1 key bits
//      (Adinets & Merrill, "Onesweep: A Faster Least Significant Digit Radix
//      Sort for GPUs", 2022): each CTA ranks its tile's keys stably, each warp its
//      own in shared memory, publishes its digit counts, resolves its global offsets by a
//      decoupled look-back over predecessor tiles, and scatters (key, slot);
//      sorting the used bits only is the same total order as CUB's 32-bit
//      stable sort, so the permutation is identical;
//   3. k_cell_start: exclusive cell-start table (cells + 1 entries), which is
//      the reference's gridRanges [start, end) for every non-empty cell;
//   4. k_gather_*: every SoA field moved by the permutation.
#include "sc_launch.h"

#include <algorithm>

// Keys per thread of a sort pass at most (sort_ipt).
#define SORT_IPT 16
#define SORT_SMS 152
#define SORT_KEYS 4
#define SORT_LOOK 8   // tiles a look-back reads at a time
#define LB_AGG 0x40000000u
#define LB_INC 0x80000000u
#define LB_FLAGS 0xC0000000u
#define LB_VALUE 0x3FFFFFFFu
#define LB_SPIN_LIMIT (1 << 22)

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The sets one launch sorts, grid y being the set: both of a small sim, whose
// passes are as long as one tile's latency, or one.
struct SortPair {
    ScSortSet s[2];
};
__host__ __device__ static inline size_t sort_tiles(long long n, int ipt) {
    return (size_t)((n + SC_THREADS * ipt - 1) / (SC_THREADS * ipt));
}

// In a batched sim the key is the item's replica's key base plus its cell
// in that replica's grid: replicas sort into consecutive key ranges.
//
// Past a block per SM a thread takes SORT_KEYS items, their loads together, so
// that fewer blocks add to each of the histogram's words: 262,144 items 12.4 us
// at one item, 6.1 us at four.  The kernel also clears what the passes behind
// it look at first (the look-back words and tile counters) and farMove, and
// marks a set with a position outside a periodic box (a bit of the first digit
// count: words of their own behind the counts make the clearing memset 2 us
// longer, of 80 for a sort of 262,144 items).
template <bool BATCH, int KEYS>
__global__ void __launch_bounds__(SC_THREADS) k_sort_keys(SortPair sets, ScParams P, uint32_t inactiveKey, int passes,
                                                          int ipt, ScCounters *ctr) {
    __shared__ uint32_t sh[4 * 256];
    const ScSortSet &S = sets.s[blockIdx.y];
    const int n = S.n, blocks = (int)sort_tiles(n, KEYS), lbWords = passes * (int)sort_tiles(n, ipt) * 256;
    if ((int)blockIdx.x >= blocks) return;
    const float4 *__restrict__ pos = S.pos;
    const int4 *__restrict__ info = S.info;
    uint32_t *__restrict__ keys = S.keys[0], *__restrict__ hist = S.hist;
    for (int t = threadIdx.x; t < passes * 256; t += blockDim.x) sh[t] = 0;
    __syncthreads();
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = blocks * SC_THREADS;
    int4 in[KEYS];
    sc_f3 p[KEYS];
    bool outside = false;
#pragma unroll
    for (int r = 0; r < KEYS; r++) {
        const int i = min(first + r * stride, n - 1);
        in[r] = __ldg(info + i);
        p[r] = ld3(pos, i);
    }
#pragma unroll
    for (int r = 0; r < KEYS; r++) {
        const int i = first + r * stride;
        if (i >= n) break;
        uint32_t k = inactiveKey;
        if (in[r].z & SC_ACTIVE) {
            rep_apply<BATCH>(P, in[r].w);
            int lim = cell_limit(P);
            k = cell_key(P, sc_grid_idx(p[r].x, P.cell, lim), sc_grid_idx(p[r].y, P.cell, lim),
                         sc_grid_idx(p[r].z, P.cell, lim));
            outside |= P.periodic && !in_box(p[r], P.simSize);
        }
        keys[i] = k;
        for (int d = 0; d < passes; d++) atomicAdd(&sh[d * 256 + ((k >> (8 * d)) & 0xffu)], 1u);
    }
    for (int w = first; w < lbWords; w += stride) S.lookback[w] = 0;
    if (first < 4) S.tileCounter[first] = 0;
    if (first == 4) ctr->farMove = 0;
    if (__syncthreads_or(outside) && threadIdx.x == 0) atomicOr(hist, SC_SORT_OUTSIDE);
    for (int t = threadIdx.x; t < passes * 256; t += blockDim.x)
        if (sh[t]) atomicAdd(&hist[t], sh[t]);
}

// Exclusive scan of 256 values held one per thread (block of 256).
__device__ __forceinline__ uint32_t block_exclusive_scan256(uint32_t v, uint32_t *warp_sums) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t pre = 0;
    for (int w = 0; w < warp; w++) pre += warp_sums[w];
    return pre + x - v;
}

// One pass.  Bound by latency at these sizes (L2 holds the keys): with the
// warps ranking their own keys without a barrier per round and eight tiles
// looked back at a time, a pass over 262,144 keys takes 9.7 us, 14.4 with a
// block-wide round per 256 keys and a tile at a time.
template <int IPT>
__global__ void __launch_bounds__(SC_THREADS) k_onesweep(SortPair sets, int pass, ScCounters *ctr) {
    const ScSortSet &S = sets.s[blockIdx.y];
    const int n = S.n, tiles = (int)sort_tiles(n, IPT), shift = 8 * pass;
    if ((int)blockIdx.x >= tiles) return;
    const uint32_t *__restrict__ keysIn = S.keys[pass & 1], *__restrict__ valsIn = pass ? S.vals[pass & 1] : nullptr;
    uint32_t *__restrict__ keysOut = S.keys[~pass & 1], *__restrict__ valsOut = S.vals[~pass & 1];
    const uint32_t *__restrict__ hist = S.hist + 256 * pass;
    uint32_t *lookback = S.lookback + (size_t)pass * tiles * 256;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_cnt[8][256];   // a warp's keys per digit so far; then its first key's rank
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_wsum[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = (uint32_t)atomicAdd(&S.tileCounter[pass], 1);
#pragma unroll
    for (int w = 0; w < 8; w++) s_cnt[w][tid] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const long long base = ((long long)tile * 8 + warp) * (32 * IPT) + lane;   // a warp's keys lie together
    const uint32_t ltmask = (1u << lane) - 1u;

    uint32_t key[IPT], val[IPT], rank[IPT];
#pragma unroll
    for (int r = 0; r < IPT; r++) {
        long long idx = base + r * 32;
        if (idx < n) {
            key[r] = __ldg(keysIn + idx);
            val[r] = valsIn ? __ldg(valsIn + idx) : (uint32_t)idx;
        } else {
            key[r] = 0;
            val[r] = 0;
        }
    }
    // Stable ranking: tile order is (warp, round, lane).  Within a round the
    // warp match gives the rank among equal digits, behind the warp's count of
    // the rounds before; the warps' counts then become their offsets.
#pragma unroll
    for (int r = 0; r < IPT; r++) {
        const bool valid = base + r * 32 < n;
        const uint32_t d = valid ? ((key[r] >> shift) & 0xffu) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = valid ? s_cnt[warp][d] : 0u;
        __syncwarp();
        rank[r] = before + __popc(peers & ltmask);
        if (valid && (peers & ltmask) == 0) s_cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Decoupled look-back: thread tid owns digit tid.
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const uint32_t c = s_cnt[w][tid];
        s_cnt[w][tid] = cnt;
        cnt += c;
    }
    uint32_t excl = 0;
    if (tile == 0) {
        st_relaxed(&lookback[tid], LB_INC | cnt);
    } else {
        st_relaxed(&lookback[(size_t)tile * 256 + tid], LB_AGG | cnt);
        // SORT_LOOK tiles' words on their way at once; a word that is not
        // there yet is waited for when its turn comes
        bool found = false;
        for (long long pred = (long long)tile - 1; pred >= 0 && !found; pred -= SORT_LOOK) {
            uint32_t v[SORT_LOOK];
#pragma unroll
            for (int u = 0; u < SORT_LOOK; u++)
                v[u] = pred >= u ? ld_relaxed(&lookback[(size_t)(pred - u) * 256 + tid]) : LB_INC;
#pragma unroll
            for (int u = 0; u < SORT_LOOK; u++) {
                if (found) continue;
                for (int spins = 0; !(v[u] & LB_FLAGS);) {
                    if (++spins > LB_SPIN_LIMIT) {
                        set_error(ctr, SC_DERR_LOOKBACK_TIMEOUT);
                        v[u] = LB_INC;
                        break;
                    }
                    __nanosleep(32);
                    v[u] = ld_relaxed(&lookback[(size_t)(pred - u) * 256 + tid]);
                }
                excl += v[u] & LB_VALUE;
                found = v[u] & LB_INC;
            }
        }
        st_relaxed(&lookback[(size_t)tile * 256 + tid], LB_INC | (excl + cnt));
    }
    uint32_t gofs = block_exclusive_scan256(hist[tid] & ~SC_SORT_OUTSIDE, s_wsum);
    s_base[tid] = gofs + excl;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < IPT; r++) {
        long long idx = base + r * 32;
        if (idx < n) {
            uint32_t d = (key[r] >> shift) & 0xffu;
            uint32_t dst = s_base[d] + s_cnt[warp][d] + rank[r];
            keysOut[dst] = key[r];
            valsOut[dst] = val[r];
        }
    }
}

// cellStart[c] = first sorted slot whose key >= c, for c in [0, cells];
// inactive keys (>= cells) count as cells.  One binary search per cell.
__global__ void k_cell_start(SortPair sets, int cur, uint32_t cells) {
    const ScSortSet &S = sets.s[blockIdx.y];
    const uint32_t *__restrict__ keys = S.keys[cur];
    const int n = S.n;
    long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c > (long long)cells) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (int)(((unsigned)lo + (unsigned)hi) >> 1);
        uint32_t k = __ldg(keys + mid);
        if ((long long)k < c) lo = mid + 1;
        else hi = mid;
    }
    S.cellStart[c] = (uint32_t)lo;
}

// The gathers load every field of the source slot before storing any: the
// destination arrays are other buffers, but the compiler cannot know that,
// and interleaved loads and stores would keep one load in flight per thread.
__global__ void __launch_bounds__(SC_THREADS) k_gather_particles(const uint32_t *__restrict__ perm, int n, PFields src,
                                                                 PFields dst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s = (int)perm[i];
    const float4 pos = src.pos[s], vel = src.vel[s], rot = src.rot[s], angvel = src.angvel[s];
    const float4 posnoise = src.posnoise[s], angnoise = src.angnoise[s], dbg = src.dbg[s];
    const int4 info = src.info[s];
    const int state = src.state[s], lscs = src.lscs[s], spoly = src.spoly[s], nb = src.nb[s];
    dst.pos[i] = pos;
    dst.vel[i] = vel;
    dst.rot[i] = rot;
    dst.angvel[i] = angvel;
    dst.posnoise[i] = posnoise;
    dst.angnoise[i] = angnoise;
    dst.dbg[i] = dbg;
    dst.info[i] = info;
    dst.state[i] = state;
    dst.lscs[i] = lscs;
    dst.spoly[i] = spoly;
    dst.nb[i] = nb;
    int nw = min(max(nb, 0), SC_MAX_ACTIVE_INTERACTIONS) * 3;
    const int *b = src.bonds + (size_t)s * 24;
    int *o = dst.bonds + (size_t)i * 24;
    for (int k = 0; k < nw; k++) o[k] = b[k];
}

// One step of the metabolic gather: optionally the two double-buffered
// fields (vel, met) into their other buffers, one single-buffer 16-byte field
// and one single-buffer int field into their spares (null: not gathered).
__global__ void __launch_bounds__(SC_THREADS) k_gather_mfield(const uint32_t *__restrict__ perm, int n, int sp4,
                                                              const float4 *__restrict__ vel, float4 *__restrict__ vel2,
                                                              const float4 *__restrict__ met, float4 *__restrict__ met2,
                                                              const float4 *__restrict__ a, float4 *__restrict__ a2,
                                                              const int *__restrict__ c, int *__restrict__ c2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = (int)perm[i];
    float4 v = make_float4(0, 0, 0, 0), x = make_float4(0, 0, 0, 0), mt[3];
    int y = 0;
    if (vel) v = vel[s];
    if (a) x = a[s];
    if (c) y = c[s];
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (met && k < sp4) mt[k] = met[(size_t)s * sp4 + k];
    if (vel) vel2[i] = v;
    if (a) a2[i] = x;
    if (c) c2[i] = y;
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (met && k < sp4) met2[(size_t)i * sp4 + k] = mt[k];
}

// ---- host-side launchers -----------------------------------------------------

int sc_sort_passes_for(const ScParams &P) { return ((P.keyBits > 0 ? P.keyBits : 3 * P.bits + 1) + 7) / 8; }

// Four or eight keys per thread while every tile has an SM of its own, sixteen
// beyond: a pass of few tiles is the latency of one tile's rounds of ranking
// (a whole sort of 32,768 items 61 us at sixteen, 52 at eight, 49 at four;
// 131,072: 74, 63, 63; 200,000: 75, 66, 74); past an SM each there is nothing
// left to gain (262,144: 75, 74, 75) and fewer tiles look back less.
static int sort_ipt(long long n) {
    return sort_tiles(n, 4) <= SORT_SMS ? 4 : sort_tiles(n, 8) <= SORT_SMS ? 8 : SORT_IPT;
}


// Words of one pass's look-back table for up to cap items, whatever their number.
size_t sc_sort_lookback_words(int cap) {
    return std::max<size_t>(std::min<size_t>(sort_tiles(cap, 4), SORT_SMS), sort_tiles(cap, SORT_IPT)) * 256;
}

// Both sets of a sim are sorted by the same launches while either's tiles fit the
// device at four keys a thread: 4,096 + 8,192 items, ten steps 6.94 / 6.76 ms,
// four sims in flight 2.10 / 2.06; 65,536 + 131,072 12.4 / 12.3.
bool sc_sort_together(int n, int m) { return n > 0 && m > 0 && sort_ipt(std::max(n, m)) == 4; }

// Sorts the keys of one item set or two (sc_sort_together) and finds their
// cells' starts; returns the buffer index (0/1) holding the sorted keys and the
// permutations.
int sc_launch_sort(cudaStream_t st, const ScSortSet *sets, int count, const ScParams &P, ScCounters *ctr,
                   long long *launches) {
    int passes = sc_sort_passes_for(P);
    int keyBits = P.keyBits > 0 ? P.keyBits : 3 * P.bits + 1;
    uint32_t inactiveKey = keyBits >= 32 ? 0xffffffffu : ((1u << keyBits) - 1u);
    const SortPair pair{{sets[0], sets[count - 1]}};
    const int n = std::max(pair.s[0].n, pair.s[1].n), ipt = sort_ipt(n);
    auto *const pass = ipt == 4 ? k_onesweep<4> : ipt == 8 ? k_onesweep<8> : k_onesweep<SORT_IPT>;
    for (int k = 0; k < count; k++) cudaMemsetAsync(sets[k].hist, 0, 4 * 256 * sizeof(uint32_t), st);
    if (n > 0) {
        const bool one = sort_tiles(n, 1) <= SORT_SMS;
        auto *const make = P.nRep > 1 ? (one ? k_sort_keys<true, 1> : k_sort_keys<true, SORT_KEYS>)
                                      : (one ? k_sort_keys<false, 1> : k_sort_keys<false, SORT_KEYS>);
        make<<<dim3((unsigned)sort_tiles(n, one ? 1 : SORT_KEYS), count), SC_THREADS, 0, st>>>(pair, P, inactiveKey,
                                                                                              passes, ipt, ctr);
        for (int d = 0; d < passes; d++)
            pass<<<dim3((unsigned)sort_tiles(n, ipt), count), SC_THREADS, 0, st>>>(pair, d, ctr);
        (*launches) += 1 + passes;
    } else {
        // the tile counters and farMove behind them
        cudaMemsetAsync(ctr->tileCounter, 0, sizeof(ctr->tileCounter) + sizeof(ctr->farMove), st);
    }
    const int cur = n > 0 ? passes & 1 : 0;
    const unsigned blocks = (unsigned)(((long long)P.cells + 1 + SC_THREADS - 1) / SC_THREADS);
    k_cell_start<<<dim3(blocks, count), SC_THREADS, 0, st>>>(pair, cur, P.cells);
    (*launches)++;
    return cur;
}

void sc_launch_gather_particles(cudaStream_t st, const uint32_t *perm, int n, const PFields &src, const PFields &dst,
                                long long *launches) {
    if (n <= 0) return;
    k_gather_particles<<<(n + SC_THREADS - 1) / SC_THREADS, SC_THREADS, 0, st>>>(perm, n, src, dst);
    (*launches)++;
}

// The metabolic gather through the spares (ScBuffers::mChain4 / mChain1):
// from parity 0 field k moves from chain entry k + 1 to entry k, fields in
// ascending order; from parity 1 from entry k to k + 1, in descending order
// (each launch writes the buffer the previous one read).  vel and met go to
// their other buffers in the first launch.  Flips the parity and the two
// double-buffered fields.
void sc_launch_gather_metabolic(cudaStream_t st, const uint32_t *perm, int n, int sp4, ScBuffers &B,
                                long long *launches) {
    if (n > 0) {
        const MFields src = B.M(), dst = B.Mnext();
        const int par = B.mParity;
        for (int t = 0; t < ScBuffers::kM4; t++) {
            const int k = par ? ScBuffers::kM4 - 1 - t : t;
            const float4 *a = par ? B.mChain4[k] : B.mChain4[k + 1];
            float4 *a2 = par ? B.mChain4[k + 1] : B.mChain4[k];
            const int *c = nullptr;
            int *c2 = nullptr;
            if (t < ScBuffers::kM1) {
                const int q = par ? ScBuffers::kM1 - 1 - t : t;
                c = par ? B.mChain1[q] : B.mChain1[q + 1];
                c2 = par ? B.mChain1[q + 1] : B.mChain1[q];
            }
            k_gather_mfield<<<(n + SC_THREADS - 1) / SC_THREADS, SC_THREADS, 0, st>>>(
                perm, n, sp4, t == 0 ? src.vel : nullptr, dst.vel, t == 0 ? src.met : nullptr, dst.met, a, a2, c, c2);
            (*launches)++;
        }
    }
    B.setMParity(1 - B.mParity);
    B.cm[FM_VEL] ^= 1;
    B.cm[FM_MET] ^= 1;
}
