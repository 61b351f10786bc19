// sc_observe.cu -- ensemble observables reduced in double precision: mean
// squared displacement from a marked origin, mean |v|^2, active and bond
// counts, metabolite totals, and the pair-distance histogram (the radial
// distribution before normalisation).  No counterpart in the reference; the
// long sums are the ones that need FP64.
//
// Every reduction runs in a fixed order: a fixed grid strides over the
// slots, each block reduces its threads' partial sums by a fixed tree into
// one row of a partials table, and one block sums the rows in block order,
// so repeated calls on the same state give the same bytes.
#include "sc_launch.h"

namespace {

constexpr int OBS_BLOCKS = 512;
constexpr int OBS_TOTAL_ROWS = 256;   // rows brought in at a time

// Row layout of the partials table.
enum { O_MSD, O_MSD_N, O_V2, O_ACTIVE, O_BONDS, O_MET, O_COLS = O_MET + SC_AOS_NUM_METABOLITES };

// Within half a box (and in a walled one) a difference is its own image; the
// division, which double precision is slowest at, is left to the others.
__device__ __forceinline__ double min_image(double d, double box, bool periodic) {
    if (!periodic || fabs(d) <= 0.5 * box) return d;
    return d - box * rint(d / box);
}

// The warp's sums of 16 columns: lane 2c returns column c's, taken in the tree
// lane + 16, + 8, + 4, + 2, + 1.  A step needs half the lanes per column, so
// the other half takes another column's: 16 additions for the 80 of a tree per
// column (double precision adds two lanes a clock and SM).
__device__ __forceinline__ double warp_sums(double *v, int lane) {
#pragma unroll
    for (int o = 16, half = 8; half > 0; o >>= 1, half >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int c = 0; c < half; c++) {
            const double keep = up ? v[c + half] : v[c], give = up ? v[c] : v[c + half];
            v[c] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Partial sums over a set's slots, one row per block: grid y is the set.  Bound
// by the double-precision unit (a warp's instruction takes it 16 clocks, the
// conversions too), not by the slots' bytes: 131,072 particles and
// 262,144 metabolic items 58 us, 126 with a launch per set, a tree per column
// and a barrier after each.
__global__ void __launch_bounds__(SC_THREADS) k_observe(ScObserveSet P, ScObserveSet M, double box,
                                                        int periodic, double *__restrict__ partials) {
    static_assert(O_COLS <= 16, "warp_sums takes 16 columns");
    __shared__ double sh[SC_THREADS / 32][O_COLS];
    const ScObserveSet &F = blockIdx.y ? M : P;
    double acc[16];
#pragma unroll
    for (int c = 0; c < 16; c++) acc[c] = 0.0;
    const int n = *F.nActive;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 in = F.info[i];
        if (!(in.z & SC_ACTIVE)) continue;
        acc[O_ACTIVE] += 1.0;
        const float4 p = F.pos[i], v = F.vel[i];
        acc[O_V2] += ((double)v.x * v.x + (double)v.y * v.y) + (double)v.z * v.z;
        if (F.mark && in.x >= 0 && in.x < F.markCap) {
            const float4 m = F.mark[in.x];
            if (m.w != 0.0f) {
                const double dx = min_image((double)p.x - (double)m.x, box, periodic != 0);
                const double dy = min_image((double)p.y - (double)m.y, box, periodic != 0);
                const double dz = min_image((double)p.z - (double)m.z, box, periodic != 0);
                acc[O_MSD] += (dx * dx + dy * dy) + dz * dz;
                acc[O_MSD_N] += 1.0;
            }
        }
        if (F.nb) acc[O_BONDS] += (double)min(max(F.nb[i], 0), SC_MAX_ACTIVE_INTERACTIONS);
        if (F.met)
#pragma unroll
            for (int s = 0; s < SC_AOS_NUM_METABOLITES; s++)
                if (s < F.S) acc[O_MET + s] += (double)F.met[(size_t)i * F.sp + s];
    }
    const int lane = threadIdx.x & 31;
    const double t = warp_sums(acc, lane);
    if (!(lane & 1) && (lane >> 1) < O_COLS) sh[threadIdx.x >> 5][lane >> 1] = t;
    __syncthreads();
    if (threadIdx.x < O_COLS) {
        double r = 0.0;
        for (int w = 0; w < SC_THREADS / 32; w++) r += sh[w][threadIdx.x];
        partials[((size_t)blockIdx.y * OBS_BLOCKS + blockIdx.x) * O_COLS + threadIdx.x] = r;
    }
}

// Column sums of a set's rows of the partials table, rows in order: a thread
// per column adds what the block has brought into shared memory.  The chain of
// 512 additions is all it takes: 23 us for both sets, 2 x 30 when every
// addition also waited for its own load.
__global__ void __launch_bounds__(OBS_TOTAL_ROWS) k_observe_total(const double *__restrict__ partials,
                                                                  double *__restrict__ out) {
    __shared__ double row[OBS_TOTAL_ROWS][O_COLS];
    const double *src = partials + (size_t)blockIdx.x * OBS_BLOCKS * O_COLS;
    double s = 0.0;
    for (int r0 = 0; r0 < OBS_BLOCKS; r0 += OBS_TOTAL_ROWS) {
#pragma unroll
        for (int c = 0; c < O_COLS; c++)
            (&row[0][0])[c * OBS_TOTAL_ROWS + threadIdx.x] = src[(size_t)r0 * O_COLS + c * OBS_TOTAL_ROWS + threadIdx.x];
        __syncthreads();
        if (threadIdx.x < O_COLS)
#pragma unroll 32
            for (int r = 0; r < OBS_TOTAL_ROWS; r++) s += row[r][threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x < O_COLS) out[blockIdx.x * O_COLS + threadIdx.x] = s;
}

__global__ void __launch_bounds__(SC_THREADS) k_mark(const int *__restrict__ nActivePtr, const float4 *__restrict__ pos,
                                                     const int4 *__restrict__ info, float4 *__restrict__ mark,
                                                     int markCap) {
    const int n = *nActivePtr;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 in = info[i];
        if ((in.z & SC_ACTIVE) && in.x >= 0 && in.x < markCap) {
            const float4 p = pos[i];
            mark[in.x] = make_float4(p.x, p.y, p.z, 1.0f);
        }
    }
}

// Ordered pairs (i, j), i != j, of the requested types closer than rMax,
// binned by distance; the neighbourhood is the 27 cells of i's cell (rMax is
// at most the cell size, so no pair is missed).  Counts are gathered per
// block in shared memory, in 32 bits with the carries going straight to the
// global histogram, and added to it once.
//
// The bin is the double-precision expression's; double precision (two lanes a
// clock and SM) is only asked where single precision cannot tell.  A float
// difference of two coordinates is within 2^-24 of the exact one, which puts
// the bin position t = r nBins / rMax within 4e-7 t: unless an edge lies within
// 1e-6 (t + 1), its whole part is the bin.  Pairs seen through a face lose more
// to the image's rounding, less than 1e-6 of the box: they are ruled out well
// outside rMax and binned in double otherwise, as are differences of more than
// a box and NaN.  If both types are the same, each pair of particles in cells is
// found once, from its lower slot, and counts twice (the slots are still in the
// cells they were sorted into, so the neighbourhoods are mutual).  A particle
// made since the sort lies past them in no cell: it finds all its neighbours
// there and none finds it.
// 131,072 particles in a box of 252, all types / two: 1.85 / 0.23 ms with every
// candidate in double and 64-bit counters, 0.12 / 0.06.
__global__ void __launch_bounds__(SC_THREADS) k_pair_histogram(ScParams P, const uint32_t *__restrict__ cellStart,
                                                               const int *__restrict__ nActivePtr,
                                                               const float4 *__restrict__ pos,
                                                               const int4 *__restrict__ info, int typeA, int typeB,
                                                               double rMax, int nBins,
                                                               unsigned long long *__restrict__ counts) {
    extern __shared__ unsigned int hist[];
    for (int b = threadIdx.x; b < nBins; b += blockDim.x) hist[b] = 0u;
    __syncthreads();
    const int n = *nActivePtr, cells = cell_limit(P);
    const double box = P.simSize, r2max = rMax * rMax;
    const bool periodic = P.periodic != 0, same = typeA == typeB;
    const int binned = (int)cellStart[P.cells];
    const float L = P.simSize, half = 0.5f * L, far = (float)rMax * 1.0001f + 1e-5f * L;
    const float toBin = (float)((double)nBins / rMax);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 in = info[i];
        if (!(in.z & SC_ACTIVE) || (typeA >= 0 && in.y != typeA)) continue;
        const float4 p = pos[i];
        const bool halved = same && i < binned;
        const unsigned int weight = halved ? 2u : 1u;
        auto pair = [&](int j, const float4 &q) {
            float ax = fabsf(q.x - p.x), ay = fabsf(q.y - p.y), az = fabsf(q.z - p.z);
            const float most = fmaxf(ax, fmaxf(ay, az));
            if (periodic) {
                ax = ax > half ? fabsf(ax - L) : ax;
                ay = ay > half ? fabsf(ay - L) : ay;
                az = az > half ? fabsf(az - L) : az;
            }
            const float d2 = ax * ax + ay * ay + az * az;
            if (j == i || (most <= 1.01f * L && d2 > far * far)) return;
            const int4 tin = info[j];
            if (!(tin.z & SC_ACTIVE) || (typeB >= 0 && tin.y != typeB)) return;
            const float t = sqrtf(d2) * toBin, edge = 1e-6f * t + 1e-6f;
            int b = (int)(t + edge);
            if (!(d2 <= far * far) || (periodic && most > 0.499f * L) || b != (int)(t - edge)) {
                const double dx = min_image((double)q.x - (double)p.x, box, periodic);
                const double dy = min_image((double)q.y - (double)p.y, box, periodic);
                const double dz = min_image((double)q.z - (double)p.z, box, periodic);
                const double r2 = (dx * dx + dy * dy) + dz * dz;
                b = r2 < r2max ? (int)(sqrt(r2) * (double)nBins / rMax) : nBins;
            }
            if (b < nBins) {
                const unsigned int old = atomicAdd(&hist[b], weight);
                if (old + weight < old) atomicAdd(&counts[b], 1ull << 32);
            }
        };
        const uint32_t from = halved ? (uint32_t)i + 1u : 0u;
        const int cx = (int)sc_grid_idx(p.x, P.cell, cells), cy = (int)sc_grid_idx(p.y, P.cell, cells),
                  cz = (int)sc_grid_idx(p.z, P.cell, cells);
        const bool wraps = periodic && (cz < 1 || cz > cells - 2);   // the z run is not one slot range
        for (int col = 0; col < 9; col++) {
            int gx = cx + col / 3 - 1, gy = cy + col % 3 - 1;
            if (periodic) {
                gx = wrap_cell(gx, cells);
                gy = wrap_cell(gy, cells);
            } else if (gx < 0 || gy < 0 || gx >= cells || gy >= cells) {
                continue;
            }
            const uint32_t base = cell_key(P, (uint32_t)gx, (uint32_t)gy, 0);
            for (int oz = wraps ? -1 : 1; oz <= 1; oz++) {
                const uint32_t z0 = wraps ? wrap_cell(cz + oz, cells) : (uint32_t)max(cz - 1, 0);
                const uint32_t z1 = wraps ? z0 : (uint32_t)min(cz + 1, cells - 1);
                const uint32_t e = cellStart[base + z1 + 1];
                for (uint32_t j = max(cellStart[base + z0], from); j < e; j += 4) {
                    float4 q[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) q[u] = pos[min(j + u, e - 1)];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (j + u < e) pair((int)(j + u), q[u]);
                }
            }
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nBins; b += blockDim.x)
        if (hist[b]) atomicAdd(&counts[b], (unsigned long long)hist[b]);
}

}  // namespace

void sc_launch_mark(cudaStream_t st, const int *nActive, const float4 *pos, const int4 *info, float4 *mark,
                    int markCap) {
    k_mark<<<OBS_BLOCKS, SC_THREADS, 0, st>>>(nActive, pos, info, mark, markCap);
}

int sc_observe_cols() { return O_COLS; }
int sc_observe_rows() { return 2 * OBS_BLOCKS; }

void sc_launch_observe(cudaStream_t st, const ScObserveSet &P, const ScObserveSet &M, double box, int periodic,
                       double *partials, double *out) {
    k_observe<<<dim3(OBS_BLOCKS, 2), SC_THREADS, 0, st>>>(P, M, box, periodic, partials);
    k_observe_total<<<2, OBS_TOTAL_ROWS, 0, st>>>(partials, out);
}

void sc_launch_pair_histogram(cudaStream_t st, const ScParams &P, const uint32_t *cellStart, const int *nActive,
                              const float4 *pos, const int4 *info, int typeA, int typeB, double rMax, int nBins,
                              unsigned long long *counts, int gridCap) {
    k_pair_histogram<<<gridCap, SC_THREADS, (size_t)nBins * sizeof(unsigned int), st>>>(
        P, cellStart, nActive, pos, info, typeA, typeB, rMax, nBins, counts);
}
