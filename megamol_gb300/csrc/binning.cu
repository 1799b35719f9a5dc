// Cell binning: typed particle lists -> float4 xyzr records + cell keys, their stable sort by cell with
// every particle's gather record in sorted order, and the per-cell start table of the sorted order.
// Two sorts give the same permutation bit for bit: a counting sort by cell (histogram, scan of the cell
// counts = the start table, scatter of the indices, records in index order within the cells; taken while no
// cell holds more than BIN_CELL_MAX particles) and a stable LSD radix sort (onesweep: one read and
// one write of the keys per 8- or 9-bit digit, decoupled look-back across tiles), which runs alone for
// sparse frames and as the device-side fallback of the counting sort.
//
// Reference semantics (plugins/datatools/src/ParticlesToDensity.cpp):
//   - particle components are read through SimpleSphericalParticles' accessors, i.e. converted to
//     float with static_cast (SimpleSphericalParticles.h:86-130, Accessor.h:33-117); FLOAT_XYZ,
//     DOUBLE_XYZ and SHORT_XYZ lists use the list's global radius (ParticlesToDensity.cpp:460-463,569-571)
//   - the cell of a particle is (p - min) / sliceDist in float (:564-568).
// The bin used for sorting is floor() of that quotient clamped to [-1, res] (one underflow and one
// overflow bin per axis collect everything outside the box); the footprint decisions later use the
// reference's truncation of the same quotient.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "p2v_common.cuh"
#include "p2v_internal.h"
#include "particle_record.cuh"

namespace p2v {

namespace {

template<class T>
__device__ __forceinline__ T load_unaligned(const uint8_t* p) {
    T v;
    uint8_t* d = reinterpret_cast<uint8_t*>(&v);
#pragma unroll
    for (int i = 0; i < (int) sizeof(T); ++i)
        d[i] = p[i];
    return v;
}

template<class T, bool ALIGNED>
__device__ __forceinline__ float load_comp(const uint8_t* p) {
    if (ALIGNED)
        return static_cast<float>(*reinterpret_cast<const T*>(p));
    return static_cast<float>(load_unaligned<T>(p));
}

__device__ __forceinline__ int32_t clamp_cell(float q) {
    // floor of the cell quotient, clamped to +-2^30 so it always fits an int
    float f = floorf(q);
    f = fminf(fmaxf(f, -1073741824.0f), 1073741824.0f);
    return static_cast<int32_t>(f);
}

__device__ __forceinline__ uint32_t lane_id() {
    return threadIdx.x & 31u;
}

// True when the particle's kernel support holds no grid node along some axis, by a margin that the density
// gather's own node ranges cannot contradict: the gather would add nothing for it. q: the particle's position
// in cells, (p - min) / h as the bin key takes it. In node units the nodes around the particle lie at in-cell
// offsets 0 and 1 from its offset phi = q - floor(q); neither is inside the support when phi and 1 - phi both
// exceed eps / h by 1e-3 plus the rounding of q and of a position the gather forms from a cell up to twice the
// grid size away (the gather's exactly rounded in-cell offset differs from phi by less than that).
__device__ __forceinline__ bool support_misses_nodes(const float q[3], float r, const GridGeo& g) {
    const float eps = g.kernel == 0 ? g.sigma * r : 3.0f * (g.sigma * r);
    bool miss = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float phi = q[a] - floorf(q[a]);
        const float eh = eps * g.ihh[a];
        const float m = 1e-3f + 1e-6f * static_cast<float>(g.s[a]) + 4e-7f * fabsf(q[a]);
        miss = miss || (phi - eh > m && (1.0f - phi) - eh > m);
    }
    return miss;
}

// A particle's bin key (nbins: invalid), its cell c and its position q in cells.
__device__ __forceinline__ bool cell_key(const float4& p, const GridGeo& g, uint32_t& key, int32_t c[3], float q[3]) {
    const float pc[3] = {p.x, p.y, p.z};
    bool valid = isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(p.w) && p.w > 0.0f;
    uint32_t bin[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        q[a] = (pc[a] - g.minf[a]) / g.hf[a];
        valid = valid && fabsf(q[a]) < 1073741824.0f;
        c[a] = clamp_cell(q[a]);
        const int32_t b = c[a] < -1 ? -1 : (c[a] > g.s[a] ? g.s[a] : c[a]);
        bin[a] = static_cast<uint32_t>(b + 1);
    }
    key = valid ? (bin[2] * g.nb[1] + bin[1]) * g.nb[0] + bin[0] : g.nbins;
    return valid;
}

// Grid-stride over the list: each thread packs several particles and keeps running reductions, so the
// frame-wide maxima and counts cost one atomic per block rather than per 256 particles. empty_flag (a power of
// two above every cell key, or 0): added to the key of a particle whose support holds no node, so that the
// sort puts those particles after every other (in cell order) and the cell start table, which the density
// gather walks, leaves them out. counts (nullable; the counting sort): particles per key, keys in [0, nbins] (nbins: the
// invalid particles); rank then receives each particle's arrival rank in its cell, its slot there until the cells are put
// in index order (no pass over the keys for it).
constexpr int PACK_AHEAD = 2;  // (4: mixed 64M 0.43 against 0.39 ms)

template<class T, int NC, bool ALIGNED>
__global__ void __launch_bounds__(256, 6) pack_keys_kernel(ListDesc L, GridGeo g, float4* __restrict__ xyzr,
    uint32_t* __restrict__ keys, uint32_t* __restrict__ counts, uint8_t* __restrict__ rank,
    FrameScalars* __restrict__ fs, uint32_t empty_flag) {
    chain_begin();
    __shared__ int s_part[8][8];
    int32_t cell[3] = {INT32_MAX, INT32_MAX, INT32_MAX};
    int32_t cellhi[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    uint32_t rbits = 0u, drop = 0u;
    const uint64_t step = (uint64_t) gridDim.x * blockDim.x;
    // PACK_AHEAD particles per round: their loads, and the counting additions whose old values are the ranks, are in
    // flight together
    for (uint64_t i0 = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i0 < L.count; i0 += PACK_AHEAD * step) {
        float4 p[PACK_AHEAD];
        uint32_t key[PACK_AHEAD];
#pragma unroll
        for (int u = 0; u < PACK_AHEAD; ++u) {
            const uint64_t i = i0 + u * step;
            p[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (i < L.count) {
                const uint8_t* rec = L.data + i * L.stride;
                p[u].x = load_comp<T, ALIGNED>(rec);
                p[u].y = load_comp<T, ALIGNED>(rec + sizeof(T));
                p[u].z = load_comp<T, ALIGNED>(rec + 2 * sizeof(T));
                p[u].w = NC == 4 ? load_comp<T, ALIGNED>(rec + 3 * sizeof(T)) : L.global_radius;
            }
        }
#pragma unroll
        for (int u = 0; u < PACK_AHEAD; ++u) {
            const uint64_t i = i0 + u * step;
            if (i >= L.count)
                break;
            int32_t c[3];
            float q[3];
            if (cell_key(p[u], g, key[u], c, q)) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    cell[a] = min(cell[a], c[a]);
                    cellhi[a] = max(cellhi[a], c[a]);
                }
                rbits = max(rbits, __float_as_uint(p[u].w));
                if (empty_flag && support_misses_nodes(q, p[u].w, g))
                    key[u] |= empty_flag;
            } else {
                ++drop;
            }
            const uint64_t o = L.offset + i;
            // streaming stores: the cell counts should stay in L2
            __stcs(xyzr + o, p[u]);
            __stcs(keys + o, key[u]);
        }
        if (counts) {
            uint32_t rk[PACK_AHEAD];
#pragma unroll
            for (int u = 0; u < PACK_AHEAD; ++u)
                if (i0 + u * step < L.count)
                    rk[u] = atomicAdd(counts + key[u], 1u);
#pragma unroll
            for (int u = 0; u < PACK_AHEAD; ++u)
                if (i0 + u * step < L.count)
                    __stcs(rank + L.offset + i0 + u * step, (uint8_t) min(rk[u], 255u));
        }
    }
    // The block's extremes, all as maxima (a minimum of c is a maximum of ~c), one quantity per thread of the first eight,
    // in the order of FrameScalars' first words. An extreme that is no news costs a load: additions to one address are
    // served one after the other, about 10 ns a block.
    const int w = threadIdx.x >> 5;
    const int part[7] = {(int) rbits, ~cell[0], ~cell[1], ~cell[2], cellhi[0], cellhi[1], cellhi[2]};
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const int m = __reduce_max_sync(0xffffffffu, part[q]);
        if (lane_id() == 0)
            s_part[q][w] = m;
    }
    drop = __reduce_add_sync(0xffffffffu, drop);
    if (lane_id() == 0)
        s_part[7][w] = (int) drop;
    __syncthreads();
    const int q = threadIdx.x;
    if (q < 7) {
        int m = s_part[q][0];
#pragma unroll
        for (int k = 1; k < 8; ++k)
            m = max(m, s_part[q][k]);
        int* const at = q == 0 ? reinterpret_cast<int*>(&fs->rmax_bits) : (q < 4 ? &fs->cmin[q - 1] : &fs->cmax[q - 4]);
        const int now = *reinterpret_cast<volatile int*>(at);
        if (q >= 1 && q < 4) {
            if (~m < now)
                atomicMin(at, ~m);
        } else if (m > now) {
            atomicMax(at, m);
        }
    } else if (q == 7) {
        uint32_t d = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            d += (uint32_t) s_part[7][k];
        if (d)
            atomicAdd(&fs->n_dropped, d);
    }
}

// ---------------------------------------------------------------------------------------------
// Onesweep LSD radix sort of (key, value) pairs with 8- or 9-bit digits: a key of B bits takes
// ceil(B / 9) passes (a 256^3 grid's 25-bit bin keys take 9 + 8 + 8 bits, three passes).
// ---------------------------------------------------------------------------------------------
constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;  // 4096 keys per tile
constexpr int MAX_RADIX = 512;
constexpr int MAX_PASSES = 5;
constexpr int HIST_WORDS = MAX_PASSES * MAX_RADIX;    // digit histograms, pass p at p * MAX_RADIX
// after the histograms: one tile counter per radix pass, and the count of finished histogram blocks
constexpr int LOOKBACK_WINDOW = 8;  // predecessor tiles a look-back round reads at once (4: 3.55, 16: 3.49 ms)
constexpr uint32_t FLAG_AGG = 1u << 30;
constexpr uint32_t FLAG_PRE = 2u << 30;
constexpr uint32_t FLAG_MASK = 3u << 30;
constexpr uint32_t COUNT_MASK = (1u << 30) - 1u;

struct SortPlan {
    int passes;
    int shift[MAX_PASSES];
    int bits[MAX_PASSES];
};

// odd: an odd number of passes, so the sorted keys end in buffer 1 (8-bit digits where a pass is added)
SortPlan sort_plan(uint32_t max_key, bool odd = false) {
    int nb = 0;
    while (nb < 32 && (max_key >> nb) != 0u)
        ++nb;
    nb = std::max(nb, 1);
    SortPlan pl{};
    pl.passes = (nb + 8) / 9;
    if (odd && (pl.passes & 1) == 0)
        ++pl.passes;
    // the first (nb - 8 * passes) passes take 9 bits, the others 8
    int nine = std::max(0, nb - 8 * pl.passes);
    int sh = 0;
    for (int p = 0; p < pl.passes; ++p) {
        pl.bits[p] = p < nine ? 9 : 8;
        pl.shift[p] = sh;
        sh += pl.bits[p];
    }
    return pl;
}

// The radix path runs unless the counting sort (bin_tile_sums / bin_starts / scatter_bins / records) took the
// frame: with a gate, every radix kernel returns at once when the frame's fullest cell fits the counting
// sort's per-cell ordering.
__device__ __forceinline__ bool radix_skipped(const FrameScalars* gate) {
    return gate != nullptr && gate->bin_maxcount <= BIN_CELL_MAX;
}

// Digit histograms of every pass over the keys, and (the block that finishes last) their exclusive scans in place: the
// digits' first destinations. Also clears the passes' look-back words. The first nblk blocks (of 256 threads) take part;
// `done` counts the finished ones (zero before).
__device__ __forceinline__ void radix_hist(const uint32_t* __restrict__ keys, uint32_t n, const SortPlan& pl,
                                           uint32_t* __restrict__ hist, uint32_t* __restrict__ done,
                                           uint32_t* __restrict__ status, uint64_t status_words, uint32_t nblk) {
    if (blockIdx.x >= nblk)
        return;
    __shared__ uint32_t sh[HIST_WORDS];
    __shared__ uint32_t s_last, s_sum[8];
    for (int i = threadIdx.x; i < HIST_WORDS; i += blockDim.x)
        sh[i] = 0;
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < status_words / 4; i += (uint64_t) nblk * blockDim.x)
        reinterpret_cast<uint4*>(status)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += nblk * blockDim.x) {
        const uint32_t k = keys[j];
        for (int p = 0; p < pl.passes; ++p)
            atomicAdd(&sh[p * MAX_RADIX + ((k >> pl.shift[p]) & ((1u << pl.bits[p]) - 1u))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < pl.passes * MAX_RADIX; i += blockDim.x)
        if (sh[i])
            atomicAdd(&hist[i], sh[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(done, 1u) == nblk - 1u ? 1u : 0u;
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    for (int p = 0; p < pl.passes; ++p) {
        uint32_t* h = hist + p * MAX_RADIX + 2 * threadIdx.x;  // two digits per thread
        const uint32_t a = __ldcg(h), b = __ldcg(h + 1);
        uint32_t incl = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t) o)
                incl += t;
        }
        if (lane == 31)
            s_sum[w] = incl;
        __syncthreads();
        uint32_t pre = incl - a - b;
        for (uint32_t k = 0; k < w; ++k)
            pre += s_sum[k];
        h[0] = pre;
        h[1] = pre + a;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) radix_hist_kernel(const uint32_t* __restrict__ keys, uint32_t n, SortPlan pl,
    uint32_t* __restrict__ hist, uint32_t* __restrict__ done, uint32_t* __restrict__ status, uint64_t status_words) {
    chain_begin();
    radix_hist(keys, n, pl, hist, done, status, status_words, gridDim.x);
}

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
    return *reinterpret_cast<const volatile uint32_t*>(p);
}

__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) {
    *reinterpret_cast<volatile uint32_t*>(p) = v;
}

// One pass over digit (key >> shift) & (RADIX - 1). Tiles are taken in launch order from a counter; each
// tile ranks its keys stably (per-warp digit counters), publishes its digit counts, resolves its global offsets by decoupled look-back, stages the tile in digit order in shared
// memory and writes runs of equal digits contiguously.
// The look-back waits are bounded (wait_polls polls of a predecessor that has published nothing). A wait
// that runs out records ERR_LOOKBACK_TIMEOUT; every other wait then stops at its next poll and later passes
// return at once. A tile that gave up adds only the counts it saw, so its destinations stay at or below the
// true ones (inside the output); boundary_starts_kernel then replaces the unfinished output by a valid one.
template<bool GATHER, int BITS>
__global__ void __launch_bounds__(SORT_THREADS, 3) onesweep_kernel(const uint32_t* __restrict__ keys_in,
    const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
    int shift, const uint32_t* __restrict__ digit_offsets, uint32_t* __restrict__ tile_counter,
    uint32_t* __restrict__ status, uint32_t* __restrict__ err, const float4* __restrict__ xyzr_in,
    float4* __restrict__ rec_a, int4* __restrict__ rec_b, float4* __restrict__ xyzr_out, GridGeo geo,
    const FrameScalars* __restrict__ gate, uint32_t wait_polls, int32_t hold_tile) {
    chain_begin();
    if (radix_skipped(gate) || (ld_volatile(err) & ERR_LOOKBACK_TIMEOUT))
        return;
    constexpr int RADIX = 1 << BITS;
    constexpr uint32_t DMASK = RADIX - 1u;
    constexpr int DPT = RADIX / SORT_THREADS;  // digits per thread in the per-digit phases
    extern __shared__ __align__(16) uint32_t sort_smem[];
    uint32_t* s_keys = sort_smem;                                                  // [SORT_TILE]
    uint32_t* s_vals = s_keys + SORT_TILE;                                         // [SORT_TILE]
    uint32_t(*s_whist)[RADIX] = reinterpret_cast<uint32_t(*)[RADIX]>(s_vals + SORT_TILE);  // [SORT_WARPS][RADIX]
    uint32_t* s_base = s_vals + SORT_TILE + SORT_WARPS * RADIX;  // global destination of each digit's first item, less s_local
    uint32_t* s_local = s_base + RADIX;                          // tile-local exclusive offset of each digit
    __shared__ uint32_t s_scan[SORT_WARPS];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x;
    const int w = tid >> 5;
    const uint32_t lane = lane_id();
    if (tid == 0)
        s_tile = atomicAdd(tile_counter, 1u);
    static_assert(SORT_WARPS * RADIX <= SORT_TILE, "the ranking's lane masks take the staging buffers");
    for (int i = tid; i < SORT_WARPS * RADIX / 4; i += SORT_THREADS) {
        reinterpret_cast<uint4*>(&s_whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(s_keys)[i] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(s_vals)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * SORT_TILE;

    // warp-striped load: item i of lane l of warp w is element base + w*32*ITEMS + i*32 + l, so the
    // ranking order (i, lane) is the input order within the warp and warps follow each other.
    uint32_t k[SORT_ITEMS], v[SORT_ITEMS], rk[SORT_ITEMS];
    const uint32_t wbase = base + w * 32 * SORT_ITEMS;
#pragma unroll
    for (int i = 0; i < SORT_ITEMS; ++i) {
        const uint32_t j = wbase + i * 32 + lane;
        k[i] = j < n ? keys_in[j] : 0u;
        v[i] = j < n ? (vals_in ? vals_in[j] : j) : 0u;  // no input values: the identity (particle indices)
    }
    const uint32_t lt_mask = (1u << lane) - 1u;
    // The lanes that hold the same digit set their bits in the digit's word (two sets of words by turns, so that an item's
    // are cleared while the next one's are set). A ballot per digit bit finds the same lanes in four instructions a bit,
    // and issue bound the pass: a key pass over 64 M keys 0.42 -> 0.38 ms.
    uint32_t* const hist_w = s_whist[w];
    uint32_t* const lanes_w[2] = {s_keys + w * RADIX, s_vals + w * RADIX};
#pragma unroll
    for (int i = 0; i < SORT_ITEMS; ++i) {
        const bool valid = wbase + i * 32 + lane < n;
        const uint32_t d = (k[i] >> shift) & DMASK;
        uint32_t* const same = lanes_w[i & 1] + d;
        if (valid)
            atomicOr(same, 1u << lane);
        __syncwarp();
        const uint32_t peers = *same;
        const uint32_t b = hist_w[d];
        __syncwarp();
        const uint32_t before = peers & lt_mask;
        if (valid && before == 0u) {
            hist_w[d] = b + __popc(peers);
            *same = 0u;
        }
        rk[i] = b + __popc(before);
    }
    __syncthreads();

    // per digit (thread tid owns digits tid*DPT .. tid*DPT + DPT-1): exclusive offsets over warps, counts
    uint32_t count[DPT];
    uint32_t tsum = 0;
#pragma unroll
    for (int e = 0; e < DPT; ++e) {
        const int d = tid * DPT + e;
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ++ww) {
            const uint32_t c = s_whist[ww][d];
            s_whist[ww][d] = run;
            run += c;
        }
        count[e] = run;
        tsum += run;
        // publish the tile aggregate (or the inclusive prefix for tile 0) before looking back
        if ((int32_t) tile != hold_tile)
            st_volatile(status + (size_t) tile * RADIX + d, (tile == 0 ? FLAG_PRE : FLAG_AGG) | run);
    }
    // tile-local exclusive scan over digits (block scan of the per-thread digit sums)
    uint32_t incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t) o)
            incl += t;
    }
    if (lane == 31)
        s_scan[w] = incl;
    __syncthreads();
    uint32_t wpre = 0;
    for (int ww = 0; ww < w; ++ww)
        wpre += s_scan[ww];
    uint32_t run = wpre + incl - tsum;
#pragma unroll
    for (int e = 0; e < DPT; ++e) {
        s_local[tid * DPT + e] = run;
        run += count[e];
    }

    // decoupled look-back per digit, LOOKBACK_WINDOW predecessors per round: the window's loads are independent,
    // so a round costs one memory latency however many of its tiles have only published their aggregate (the
    // inclusive prefixes trail the tiles in flight by ~30 tiles on large frames: walking them one load at a time
    // made the look-back the key passes' bottleneck). A round consumes the window's tiles up to the first one
    // that has published nothing; a round that consumes none is a poll of the bounded wait.
#pragma unroll
    for (int e = 0; e < DPT; ++e) {
        const int d = tid * DPT + e;
        uint32_t excl = 0;
        if (tile > 0) {
            int32_t t = (int32_t) tile - 1;
            uint32_t spins = 0;
            bool done = false;
            while (!done) {
                uint32_t sv[LOOKBACK_WINDOW];
#pragma unroll
                for (int q = 0; q < LOOKBACK_WINDOW; ++q)
                    sv[q] = t - q >= 0 ? ld_volatile(status + (size_t) (t - q) * RADIX + d) : FLAG_PRE;
                int used = 0;
#pragma unroll
                for (int q = 0; q < LOOKBACK_WINDOW; ++q) {
                    if (done || used < q || (sv[q] & FLAG_MASK) == 0u)
                        continue;  // stop at the first tile without a published count
                    excl += sv[q] & COUNT_MASK;
                    done = (sv[q] & FLAG_MASK) == FLAG_PRE;
                    used = q + 1;
                }
                if (done)
                    break;
                t -= used;
                if (used == 0) {
                    if (++spins > wait_polls) {
                        atomicOr(err, ERR_LOOKBACK_TIMEOUT);
                        break;
                    }
                    if (ld_volatile(err) & ERR_LOOKBACK_TIMEOUT)
                        break;  // another wait gave up: the pass is void
                }
            }
            if ((int32_t) tile != hold_tile)
                st_volatile(status + (size_t) tile * RADIX + d, FLAG_PRE | (excl + count[e]));
        }
        s_base[d] = digit_offsets[d] + excl - s_local[d];
    }
    __syncthreads();

    // stage the tile in digit order, then write runs of equal digits contiguously
#pragma unroll
    for (int i = 0; i < SORT_ITEMS; ++i) {
        const uint32_t j = wbase + i * 32 + lane;
        if (j < n) {
            const uint32_t dd = (k[i] >> shift) & DMASK;
            const uint32_t lp = s_local[dd] + s_whist[w][dd] + rk[i];
            s_keys[lp] = k[i];
            s_vals[lp] = v[i];
        }
    }
    __syncthreads();
    const uint32_t tile_n = n - base < (uint32_t) SORT_TILE ? n - base : (uint32_t) SORT_TILE;
    if (!GATHER) {
        for (uint32_t j = tid; j < tile_n; j += SORT_THREADS) {
            const uint32_t kk = s_keys[j];
            const uint32_t dd = (kk >> shift) & DMASK;
            const uint32_t dst = s_base[dd] + j;
            keys_out[dst] = kk;
            vals_out[dst] = s_vals[j];
        }
        return;
    }
    // last pass: emit every particle's gather record (and its xyzr) in sorted order. The xyzr reads are
    // scattered (input order): each thread issues GATHER_BATCH of them before it uses the first, so that
    // enough reads are in flight to cover their latency
    constexpr int GATHER_BATCH = 4;
    for (uint32_t j0 = tid; j0 < tile_n; j0 += GATHER_BATCH * SORT_THREADS) {
        uint32_t dst[GATHER_BATCH], vv[GATHER_BATCH];
        float4 p[GATHER_BATCH];
#pragma unroll
        for (int q = 0; q < GATHER_BATCH; ++q) {
            const uint32_t j = j0 + q * SORT_THREADS;
            if (j < tile_n) {
                const uint32_t kk = s_keys[j];
                const uint32_t dd = (kk >> shift) & DMASK;
                dst[q] = s_base[dd] + j;
                vv[q] = s_vals[j];
                keys_out[dst[q]] = kk;
                vals_out[dst[q]] = vv[q];
                p[q] = xyzr_in[vv[q]];
            }
        }
#pragma unroll
        for (int q = 0; q < GATHER_BATCH; ++q) {
            if (j0 + q * SORT_THREADS < tile_n) {
                float4 A;
                int4 B;
                make_record(p[q], geo, A, B);
                rec_a[REC_STRIDE * (size_t) dst[q]] = A;
                rec_b[REC_STRIDE * (size_t) dst[q]] = B;
                if (xyzr_out)
                    xyzr_out[dst[q]] = p[q];
            }
        }
    }
}

// start[c] = first sorted position whose key is >= c, for c in [0, nbins]. Boundary i of the sorted keys (between
// keys[i-1] and keys[i]) starts the run of cells (keys[i-1], keys[i]]. A warp takes 32 consecutive boundaries, scans the
// lengths of their runs, and its lanes write the cells of all 32 runs together (consecutive lanes, consecutive cells:
// coalesced however long the runs are). A run of more than run_max cells (a sparse grid
// holds runs of millions of empty cells) is queued in chunks of
// at most GAP_CHUNK for cell_gap_fill_kernel. Such runs are disjoint, so the chunks number at most (nbins + 1)
// (1 / GAP_CHUNK + 1 / (run_max + 1)), below the nbins / 64 + 2 entries the list holds (run_max >= 64).
// After a radix sort whose look-back gave up (err), every particle gets the invalid key nbins and the identity order, a
// valid sorted state (an empty grid), so that no later stage indexes with unfinished output; the frame reports
// P2V_ETIMEOUT.
// Uniform 16M (338 M cells, runs of 21): 0.28 ms (5.1 TB/s of stores and keys); with a search over the scanned lengths per
// cell 0.45 ms, bound by issue; a search per cell in a table of every 64th cell's start, as sparse frames took before,
// 1.39 ms.
constexpr uint32_t GAP_CHUNK = 8192;

// Queues a warp's runs [lo, hi] of boundaries base + lane: a lane the chunks of its run, the warp together those of a run of
// many. (One lane writing a million empty cells' chunks held its warp for as long as a hundred others took: a blob of 1 M
// in 512 M cells 1.39 -> 0.57 ms of binning. Not inlined: the registers it would take cost the warps without a queued run
// 10 to 20 %.)
__device__ __noinline__ void queue_runs(bool queued, uint32_t lo, uint32_t hi, uint32_t base, uint32_t lane,
                                        uint4* __restrict__ gaps, uint32_t gap_cap, FrameScalars* __restrict__ fs) {
    constexpr uint32_t MANY = 8;
    const uint32_t nch = queued ? (hi - lo) / GAP_CHUNK + 1u : 0u;
    const uint32_t slot = queued ? atomicAdd(&fs->ngaps, nch) : 0u;
    auto put = [&](uint32_t at, uint32_t q, uint32_t first, uint32_t last, uint32_t i) {
        const uint32_t c0 = first + q * GAP_CHUNK;
        if ((uint64_t) at + q < gap_cap)
            gaps[at + q] = make_uint4(c0, last - c0 < GAP_CHUNK ? last : c0 + (GAP_CHUNK - 1u), i, 0u);
        else
            atomicOr(&fs->error, ERR_GAP_OVERFLOW);
    };
    if (nch < MANY)
        for (uint32_t q = 0; q < nch; ++q)
            put(slot, q, lo, hi, base + lane);
    for (uint32_t m = __ballot_sync(0xffffffffu, nch >= MANY); m; m &= m - 1u) {
        const int l = __ffs(m) - 1;
        const uint32_t first = __shfl_sync(0xffffffffu, lo, l), last = __shfl_sync(0xffffffffu, hi, l);
        const uint32_t at = __shfl_sync(0xffffffffu, slot, l), k = __shfl_sync(0xffffffffu, nch, l);
        for (uint32_t q = lane; q < k; q += 32)
            put(at, q, first, last, base + (uint32_t) l);
    }
}

__global__ void __launch_bounds__(256) boundary_starts_kernel(uint32_t* __restrict__ keys,
    uint32_t* __restrict__ vals, uint32_t n, uint32_t nbins, uint32_t run_max, uint32_t* __restrict__ out,
    uint4* __restrict__ gaps, uint32_t gap_cap, FrameScalars* __restrict__ fs, const FrameScalars* __restrict__ gate) {
    chain_begin();
    if (radix_skipped(gate))
        return;
    const bool failed = (ld_volatile(&fs->error) & ERR_LOOKBACK_TIMEOUT) != 0u;
    __shared__ uint32_t s_owner[256];
    const uint32_t lane = lane_id();
    const uint32_t le_mask = 0xFFFFFFFFu >> (31u - lane);
    const uint64_t wstride = (uint64_t) gridDim.x * blockDim.x;
    for (uint64_t base = (uint64_t) blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base <= n; base += wstride) {
        const uint64_t i64 = base + lane;
        uint32_t lo = 1u, hi = 0u;  // empty run
        if (i64 <= n) {
            const uint32_t i = (uint32_t) i64;
            if (!failed) {
                lo = i == 0 ? 0u : keys[i - 1] + 1u;
                hi = i == n ? nbins : min(keys[i], nbins);
            } else {
                lo = i == 0 ? 0u : nbins + 1u;
                hi = nbins;
                if (i < n) {
                    keys[i] = nbins;
                    vals[i] = i;
                }
            }
        }
        uint32_t len = lo <= hi ? hi - lo + 1u : 0u;
        const bool queued = len > run_max;
        const uint32_t queues = __ballot_sync(0xffffffffu, queued);
        if (queues) {
            queue_runs(queued, lo, hi, (uint32_t) base, lane, gaps, gap_cap, fs);
            if (queued)
                len = 0u;
        }
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t) o)
                incl += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t pre = incl - len;  // first cell slot of this lane's run
        if (!failed && !queues) {
            // the runs of consecutive boundaries follow each other: cell slot j is cell lo(lane 0) + j. Its owner is the
            // last run that has started, by one reduction and a population count.
            const uint32_t cell0 = __shfl_sync(0xffffffffu, lo, 0);
            const uint32_t runs = __ballot_sync(0xffffffffu, len != 0u);
            if (len)
                s_owner[(threadIdx.x & ~31u) | __popc(runs & (le_mask >> 1))] = (uint32_t) i64;
            __syncwarp();
            const uint32_t head = len ? pre : 0xFFFFFFFFu;
            const uint32_t* own = s_owner + (threadIdx.x & ~31u) - 1;
            for (uint32_t j0 = 0; j0 < total; j0 += 32) {
                const uint32_t heads = __reduce_or_sync(0xffffffffu, head - j0 < 32u ? 1u << (head - j0) : 0u);
                if (j0 + lane < total)
                    out[cell0 + j0 + lane] = own[__popc(heads & le_mask)];
                own += __popc(heads);
            }
            __syncwarp();
            continue;
        }
        for (uint32_t j0 = 0; j0 < total; j0 += 32) {
            const uint32_t j = j0 + lane;
            // a queued run among them, or a failed sort: the owner is the last lane whose run starts at or before slot j
            // (lanes with empty runs share the next lane's start and are passed over: the search ends on the last of
            // equal starts)
            uint32_t ow = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t cand = ow + step;
                const uint32_t pc = __shfl_sync(0xffffffffu, pre, cand);
                if (pc <= j)
                    ow = cand;
            }
            const uint32_t olo = __shfl_sync(0xffffffffu, lo, ow);
            const uint32_t opre = __shfl_sync(0xffffffffu, pre, ow);
            if (j < total)
                out[olo + (j - opre)] = (uint32_t) (base + ow);
        }
    }
}

__global__ void __launch_bounds__(256) cell_gap_fill_kernel(const uint4* __restrict__ gaps, uint32_t gap_cap,
    uint32_t* __restrict__ start, const FrameScalars* __restrict__ fs, const FrameScalars* __restrict__ gate) {
    chain_begin();
    if (radix_skipped(gate))
        return;
    const uint32_t ng = min(fs->ngaps, gap_cap);
    for (uint32_t g = blockIdx.x; g < ng; g += gridDim.x) {
        const uint4 e = gaps[g];
        for (uint64_t c = (uint64_t) e.x + threadIdx.x; c <= e.y; c += blockDim.x)  // (e.y may lie near 2^32)
            start[c] = e.z;
    }
}

// ---- counting sort by cell ----
// counts[key] and the arrival ranks in a pass of their own (!counts_in_packing). A rank past BIN_CELL_MAX is not used: one byte.
__global__ void __launch_bounds__(256) count_bins_kernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                         uint32_t* __restrict__ counts, uint8_t* __restrict__ rank) {
    chain_begin();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        __stcs(rank + i, (uint8_t) min(atomicAdd(counts + __ldcs(keys + i), 1u), 255u));
}

constexpr int SCAN_THREADS = 256, SCAN_ITEMS = 16, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// 16 consecutive counts of thread `tid` in tile `tile` (zeros past nb); true when all 16 exist
__device__ __forceinline__ bool load_counts(const uint32_t* __restrict__ counts, uint32_t nb, uint64_t b0,
                                            uint32_t v[SCAN_ITEMS]) {
    const bool full = b0 + SCAN_ITEMS <= nb;
    if (full) {
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q) {
            const uint4 u = reinterpret_cast<const uint4*>(counts + b0)[q];
            v[4 * q] = u.x;
            v[4 * q + 1] = u.y;
            v[4 * q + 2] = u.z;
            v[4 * q + 3] = u.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < SCAN_ITEMS; ++e)
            v[e] = b0 + e < nb ? counts[b0 + e] : 0u;
    }
    return full;
}

// Scan of the cell counts in two steps (tile sums; tile scans, each block adding up the sums before its tile): no
// cross-tile waiting.
// Step 1: the sum of every tile of SCAN_TILE counts, and the largest count (fs->bin_maxcount).
__global__ void __launch_bounds__(SCAN_THREADS) bin_tile_sums_kernel(const uint32_t* __restrict__ counts, uint32_t nb,
    uint32_t* __restrict__ tsum, FrameScalars* __restrict__ fs) {
    chain_begin();
    __shared__ uint32_t s_sum[SCAN_THREADS / 32], s_max[SCAN_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t v[SCAN_ITEMS];
    load_counts(counts, nb, (uint64_t) blockIdx.x * SCAN_TILE + (uint64_t) tid * SCAN_ITEMS, v);
    uint32_t sum = 0, vmax = 0;
#pragma unroll
    for (int e = 0; e < SCAN_ITEMS; ++e) {
        sum += v[e];
        vmax = max(vmax, v[e]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        vmax = max(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if (lane == 0) {
        s_sum[w] = sum;
        s_max[w] = vmax;
    }
    __syncthreads();
    if (tid == 0) {
        for (int k = 1; k < SCAN_THREADS / 32; ++k) {
            sum += s_sum[k];
            vmax = max(vmax, s_max[k]);
        }
        tsum[blockIdx.x] = sum;
        if (vmax > 0)
            atomicMax(&fs->bin_maxcount, vmax);
    }
}

// Step 2: start[c] = the sums of the tiles before + the scan inside the tile, for c in [0, nb).
__global__ void __launch_bounds__(SCAN_THREADS) bin_starts_kernel(const uint32_t* __restrict__ counts, uint32_t nb,
    const uint32_t* __restrict__ tsum, uint32_t* __restrict__ start) {
    chain_begin();
    __shared__ uint32_t s_warp[SCAN_THREADS / 32], s_before[SCAN_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t before = 0;
    for (uint32_t k = tid; k < blockIdx.x; k += SCAN_THREADS)
        before += tsum[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0)
        s_before[w] = before;
    const uint64_t b0 = (uint64_t) blockIdx.x * SCAN_TILE + (uint64_t) tid * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    const bool full = load_counts(counts, nb, b0, v);
    uint32_t sum = 0;
#pragma unroll
    for (int e = 0; e < SCAN_ITEMS; ++e)
        sum += v[e];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += t;
    }
    if (lane == 31)
        s_warp[w] = incl;
    __syncthreads();
    uint32_t wpre = 0;
    for (int k = 0; k < w; ++k)
        wpre += s_warp[k];
    uint32_t run = wpre + incl - sum;
    for (int k = 0; k < SCAN_THREADS / 32; ++k)
        run += s_before[k];
#pragma unroll
    for (int e = 0; e < SCAN_ITEMS; ++e) {
        const uint32_t x = run;
        run += v[e];
        v[e] = x;
    }
    if (full) {
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q)
            reinterpret_cast<uint4*>(start + b0)[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else {
#pragma unroll
        for (int e = 0; e < SCAN_ITEMS; ++e)
            if (b0 + e < nb)
                start[b0 + e] = v[e];
    }
}

// The counting sort moves indices first and particles once. Each particle's index goes to slot start[key] + rank of its
// cell (arrival order; 4 bytes a particle stay in L2 however the particles are ordered), then records_kernel takes the
// slots in order: a particle's place in its cell is the number of smaller indices there, so the result is the stable sort
// by key, and the stores of the records are contiguous. Records scattered in the particles' order, and the cells of two and
// more rewritten in index order after, took 219 + 79 us for 4.4 M particles in no spatial order and 504 + 114 for 8 M; this
// takes 43 + 47 and 78 + 85 (about 60 bytes a particle written and 30 to 50 read); in lattice order (LJ 4M) there is no difference
// beyond the byte-sized ranks. The sorted keys are not written: the cell starts hold them (keys_from_starts_kernel rebuilds
// them for the binning readback).
__global__ void __launch_bounds__(256) scatter_bins_kernel(const uint32_t* __restrict__ keys_in,
    const uint8_t* __restrict__ rank, uint32_t n, const uint32_t* __restrict__ start, uint32_t* __restrict__ arrived,
    const FrameScalars* __restrict__ fs) {
    chain_begin();
    if (fs->bin_maxcount > BIN_CELL_MAX)
        return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        arrived[start[__ldcs(keys_in + i)] + __ldcs(rank + i)] = i;
}

// A frame with a cell of more than BIN_CELL_MAX particles goes to the radix sort instead, and takes its histograms here.
__global__ void __launch_bounds__(256) records_kernel(const uint32_t* __restrict__ keys, SortPlan pl,
    uint32_t* __restrict__ hist, uint32_t* __restrict__ done, uint32_t* __restrict__ status, uint64_t status_words,
    uint32_t hist_blocks, uint32_t n, const uint32_t* __restrict__ arrived, uint32_t* __restrict__ vals,
    const uint32_t* __restrict__ start, const float4* __restrict__ xyzr, float4* __restrict__ rec_a,
    int4* __restrict__ rec_b, float4* __restrict__ xyzr_out, GridGeo geo, const FrameScalars* __restrict__ fs) {
    chain_begin();
    if (fs->bin_maxcount > BIN_CELL_MAX) {
        radix_hist(keys, n, pl, hist, done, status, status_words, hist_blocks);
        return;
    }
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t v = arrived[j];
        const float4 p = xyzr[v];
        uint32_t key;
        int32_t c[3];
        float q[3];
        cell_key(p, geo, key, c, q);
        const uint32_t s = start[key], e = key < geo.nbins ? start[key + 1] : n;
        uint32_t slot = j;
        if (e - s > 1u) {
            slot = s;
            for (uint32_t a = s; a < e; ++a)
                slot += arrived[a] < v ? 1u : 0u;
        }
        vals[slot] = v;
        float4 A;
        int4 B;
        make_record(p, geo, A, B);
        rec_a[REC_STRIDE * (size_t) slot] = A;
        rec_b[REC_STRIDE * (size_t) slot] = B;
        if (xyzr_out)
            xyzr_out[slot] = p;
    }
}

// keys[j] = the cell whose start range holds sorted position j (the counting sort writes no keys)
__global__ void __launch_bounds__(256) keys_from_starts_kernel(const uint32_t* __restrict__ start, uint32_t nbins,
                                                               uint32_t n, uint32_t* __restrict__ keys) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= nbins; k += gridDim.x * blockDim.x) {
        const uint32_t e = k < nbins ? start[k + 1] : n;
        for (uint32_t j = start[k]; j < e; ++j)
            keys[j] = k;
    }
}

// The frame's first kernel: its scalars, the counting sort's cell counts (a multiple of four words) and the radix sort's
// histograms and counters.
__global__ void __launch_bounds__(256) init_frame_kernel(FrameScalars* fs, uint4* __restrict__ counts, uint64_t ncounts4,
                                                         uint32_t* __restrict__ hist, uint32_t hist_words) {
    chain_begin();
    const uint64_t t = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x, step = (uint64_t) gridDim.x * blockDim.x;
    for (uint64_t i = t; i < ncounts4; i += step)
        counts[i] = make_uint4(0u, 0u, 0u, 0u);
    for (uint64_t i = t; i < hist_words; i += step)
        hist[i] = 0u;
    if (t == 0) {
        FrameScalars z{};
        for (int a = 0; a < 3; ++a) {
            z.cmin[a] = INT32_MAX;
            z.cmax[a] = INT32_MIN;
        }
        z.dmin_bits = 0x7f7fffffu;  // FLT_MAX, as the vector aggregator's minDens starts
        *fs = z;
    }
}

__global__ void count_valid_kernel(const uint32_t* __restrict__ start, uint32_t nbins, FrameScalars* fs) {
    chain_begin();
    fs->n_valid = start[nbins];
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------------------------
cudaError_t launch_pack_keys(const ListDesc& L, const GridGeo& g, float4* xyzr, uint32_t* keys, uint32_t* counts,
    uint8_t* rank, FrameScalars* fs, uint32_t empty_flag, cudaStream_t st) {
    if (L.count == 0)
        return cudaSuccess;
    const dim3 block(256);
    // 2 particles per thread (one round) while that is at most eight blocks per SM, then about 8; at most 64 blocks per SM
    const uint64_t one_round = (L.count + 256 * PACK_AHEAD - 1) / (256 * PACK_AHEAD);
    const dim3 grid((unsigned) std::max<uint64_t>(std::min<uint64_t>(one_round, 152ull * 8),
                                                  std::min<uint64_t>((L.count + 2047) / 2048, 152ull * 64)));
    const uintptr_t addr = reinterpret_cast<uintptr_t>(L.data);
    switch (L.type) {
    case 1: {  // FLOAT_XYZ
        bool al = (addr % 4 == 0) && (L.stride % 4 == 0);
        if (al)
            chain(pack_keys_kernel<float, 3, true>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
        else
            chain(pack_keys_kernel<float, 3, false>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
    } break;
    case 2: {  // FLOAT_XYZR
        bool al = (addr % 4 == 0) && (L.stride % 4 == 0);
        if (al)
            chain(pack_keys_kernel<float, 4, true>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
        else
            chain(pack_keys_kernel<float, 4, false>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
    } break;
    case 3: {  // SHORT_XYZ
        bool al = (addr % 2 == 0) && (L.stride % 2 == 0);
        if (al)
            chain(pack_keys_kernel<uint16_t, 3, true>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
        else
            chain(pack_keys_kernel<uint16_t, 3, false>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
    } break;
    case 4: {  // DOUBLE_XYZ
        bool al = (addr % 8 == 0) && (L.stride % 8 == 0);
        if (al)
            chain(pack_keys_kernel<double, 3, true>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
        else
            chain(pack_keys_kernel<double, 3, false>, grid, block, 0, st, L, g, xyzr, keys, counts, rank, fs, empty_flag);
    } break;
    default:
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Below 40 MB of counts (a third of the L2) the packing counts the cells and a pass over the keys is saved; above, the
// packing's streams push the table out of the L2, and a pass that moves only keys and ranks is faster. Packing and
// binning, us, in the packing against apart: 33 MB 207 / 216, 50 MB 323 / 311, 67 MB (LJ 4M) 226 / 209, 69 MB 452 / 397.
bool counts_in_packing(uint32_t nbins) {
    return nbins < (10u << 20);
}

namespace {
size_t status_words_of(const SortPlan& pl, uint32_t n) {  // every pass has its own look-back words
    size_t w = 0;
    for (int p = 0; p < pl.passes; ++p)
        w += (size_t) ceil_div(n, SORT_TILE) << pl.bits[p];
    return w;
}
}  // namespace

size_t sort_status_words(uint32_t n, uint32_t max_key) {
    return std::max(status_words_of(sort_plan(max_key), n), status_words_of(sort_plan(max_key, true), n));
}

size_t sort_hist_words() {
    return HIST_WORDS + 8;
}

int sort_passes(uint32_t max_key) {
    return sort_plan(max_key).passes;
}

uint32_t sort_empty_flag(uint32_t max_key) {
    int nb = 0;
    while (nb < 32 && (max_key >> nb) != 0u)
        ++nb;
    if (nb >= 31)
        return 0u;
    const uint32_t flag = 1u << nb;
    return sort_plan(flag | (flag - 1u)).passes == sort_plan(max_key).passes ? flag : 0u;
}

template<bool GATHER, int BITS>
cudaError_t launch_onesweep_bits(uint32_t tiles, SortBuffers& b, int cur, uint32_t n, int shift, const uint32_t* offs,
                                 uint32_t* counter, uint32_t* status, cudaStream_t st, const FrameScalars* gate) {
    constexpr int RADIX = 1 << BITS;
    const int smem = (int) sizeof(uint32_t) * (2 * SORT_TILE + SORT_WARPS * RADIX + 2 * RADIX);
    const cudaError_t e = cudaFuncSetAttribute(onesweep_kernel<GATHER, BITS>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    chain(onesweep_kernel<GATHER, BITS>, tiles, SORT_THREADS, smem, st, b.keys[cur],
        (cur == 0 && b.implicit_vals0 && b.first_pass) ? nullptr : b.vals[cur], b.keys[cur ^ 1],
        b.vals[cur ^ 1], n, shift, offs, counter, status, b.err, GATHER ? b.xyzr_in : nullptr,
        GATHER ? b.rec_a : nullptr, GATHER ? b.rec_b : nullptr, GATHER ? b.xyzr_out : nullptr, b.geo, gate,
        b.wait_polls ? b.wait_polls : SPIN_LIMIT, b.first_pass ? b.hold_tile : -1);
    return cudaSuccess;
}

template<bool GATHER>
cudaError_t launch_onesweep(int bits, uint32_t tiles, SortBuffers& b, int cur, uint32_t n, int shift,
                            const uint32_t* offs, uint32_t* counter, uint32_t* status, cudaStream_t st,
                            const FrameScalars* gate) {
    return bits == 9 ? launch_onesweep_bits<GATHER, 9>(tiles, b, cur, n, shift, offs, counter, status, st, gate)
                     : launch_onesweep_bits<GATHER, 8>(tiles, b, cur, n, shift, offs, counter, status, st, gate);
}

namespace {
unsigned hist_grid(uint32_t n, int sms) {
    return (unsigned) std::max<uint32_t>(1u, std::min<uint32_t>(ceil_div(n, 256 * 8), (uint32_t) sms * 4));
}

// the radix passes, after their histograms
cudaError_t launch_passes(SortBuffers& b, const SortPlan& pl, uint32_t n, cudaStream_t st, const FrameScalars* gate) {
    const uint32_t tiles = ceil_div(n, SORT_TILE);
    uint32_t* status = b.status;
    int cur = 0;
    for (int p = 0; p < pl.passes; ++p) {
        b.first_pass = p == 0;
        uint32_t* counter = b.hist + HIST_WORDS + p;
        const uint32_t* offs = b.hist + p * MAX_RADIX;
        const cudaError_t e =
            p == pl.passes - 1 && b.xyzr_in != nullptr
                ? launch_onesweep<true>(pl.bits[p], tiles, b, cur, n, pl.shift[p], offs, counter, status, st, gate)
                : launch_onesweep<false>(pl.bits[p], tiles, b, cur, n, pl.shift[p], offs, counter, status, st, gate);
        if (e != cudaSuccess)
            return e;
        status += (size_t) tiles << pl.bits[p];
        cur ^= 1;
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_sort(SortBuffers& b, uint32_t n, uint32_t max_key, int sms, cudaStream_t st) {
    const SortPlan pl = sort_plan(max_key);
    b.result = pl.passes & 1;
    if (n == 0)
        return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(b.hist, 0, sizeof(uint32_t) * sort_hist_words(), st);
    if (e != cudaSuccess)
        return e;
    chain(radix_hist_kernel, hist_grid(n, sms), 256, 0, st, b.keys[0], n, pl, b.hist, b.hist + HIST_WORDS + MAX_PASSES,
                                                         b.status, status_words_of(pl, n));
    return launch_passes(b, pl, n, st, nullptr);
}

cudaError_t launch_init_frame(FrameScalars* fs, uint32_t* counts, uint32_t nbins, uint32_t* hist, int sms,
                              cudaStream_t st) {
    const uint64_t c4 = counts ? ((uint64_t) nbins + 4) / 4 : 0;
    const unsigned grid = (unsigned) std::max<uint64_t>(4, std::min<uint64_t>((c4 + 255) / 256, (uint64_t) sms * 8));
    chain(init_frame_kernel, grid, 256, 0, st, fs, reinterpret_cast<uint4*>(counts), c4, hist, (uint32_t) sort_hist_words());
    return cudaGetLastError();
}

cudaError_t launch_count_valid(const uint32_t* start, uint32_t nbins, FrameScalars* fs, cudaStream_t st) {
    chain(count_valid_kernel, 1, 1, 0, st, start, nbins, fs);
    return cudaGetLastError();
}

cudaError_t launch_keys_from_starts(const uint32_t* start, uint32_t nbins, uint32_t n, uint32_t* keys, int sms,
                                    cudaStream_t st) {
    const unsigned grid = (unsigned) std::max<uint32_t>(1u, std::min<uint32_t>(ceil_div(nbins + 1, 256), (uint32_t) sms * 16));
    keys_from_starts_kernel<<<grid, 256, 0, st>>>(start, nbins, n, keys);
    return cudaGetLastError();
}

size_t bin_scan_words(uint32_t nbins) {
    return (size_t) ceil_div(nbins + 1, SCAN_TILE);
}

namespace {
// The longest run of empty cells that boundary_starts_kernel writes itself. A warp writes its 32 runs one after the other,
// about 0.1 us for 32 cells, while few boundaries leave most of the SMs idle; a queued run takes about 0.7 us of one of
// the fill's 304 blocks. The two are even at runs of n / 25 to n / 40. Binning, all but the shortest runs queued (64) /
// this rule / 8192 always, ms: 300 particles in 0.3 M cells 0.026 / 0.026 / 0.065, 10,000 in 65 M 0.091 / 0.091 / 0.249,
// 30,000 in 16 M 0.089 / 0.075 / 0.072, 300,000 in 126 M 0.62 / 0.15 / 0.15.
uint32_t longest_run(uint32_t n) {
    return std::max<uint32_t>(64u, std::min<uint32_t>(8192u, n / 25));
}
}  // namespace

cudaError_t launch_bin_sort(SortBuffers& b, uint32_t n, const GridGeo& g, uint32_t* counts, uint32_t* start,
                            uint4* gaps, uint32_t gap_cap, FrameScalars* fs, int sms,
                            cudaStream_t st) {
    const uint32_t nb = g.nbins + 1;
    const bool counting = counts != nullptr && n > 0;
    // the radix path: alone, or as the fallback (gated) when a cell holds more than BIN_CELL_MAX particles;
    // with the counting sort its pass count is odd so both leave the sorted keys in buffer 1
    const FrameScalars* gate = counting ? fs : nullptr;
    const uint32_t max_key = b.empty_flag ? (b.empty_flag | (b.empty_flag - 1u)) : g.nbins;
    const SortPlan pl = sort_plan(max_key, counting);
    b.result = pl.passes & 1;
    uint32_t* done = b.hist + HIST_WORDS + MAX_PASSES;
    const uint64_t sw = status_words_of(pl, n);
    if (counting) {
        // counting sort by cell (counts and arrival ranks from the packing): scan (= the cell starts), scatter of the
        // indices, records. Tile sums in the status buffer; the indices in arrival order in keys[1] (the counting sort
        // writes no sorted keys there); ranks in vals[0], the gated radix sort takes the identity as its first pass' values
        const uint32_t ntiles = (uint32_t) bin_scan_words(g.nbins);
        const unsigned pgrid = (unsigned) std::max<uint32_t>(1u, std::min<uint32_t>(ceil_div(n, 256), (uint32_t) sms * 16));
        b.implicit_vals0 = true;
        if (!counts_in_packing(g.nbins))
            chain(count_bins_kernel, pgrid, 256, 0, st, b.keys[0], n, counts, reinterpret_cast<uint8_t*>(b.vals[0]));
        chain(bin_tile_sums_kernel, ntiles, SCAN_THREADS, 0, st, counts, nb, b.status, fs);
        chain(bin_starts_kernel, ntiles, SCAN_THREADS, 0, st, counts, nb, b.status, start);
        chain(scatter_bins_kernel, pgrid, 256, 0, st, b.keys[0], reinterpret_cast<const uint8_t*>(b.vals[0]), n, start,
              b.keys[1], fs);
        chain(records_kernel, pgrid, 256, 0, st, b.keys[0], pl, b.hist, done, b.status, sw, std::min(pgrid, hist_grid(n, sms)),
              n, b.keys[1], b.vals[1], start, b.xyzr_in, b.rec_a, b.rec_b, b.xyzr_out, b.geo, fs);
    } else if (n > 0) {
        chain(radix_hist_kernel, hist_grid(n, sms), 256, 0, st, b.keys[0], n, pl, b.hist, done, b.status, sw);
    }
    if (n > 0) {
        const cudaError_t e = launch_passes(b, pl, n, st, gate);
        if (e != cudaSuccess)
            return e;
    }
    // (gated, the blocks return at once in most frames; else 32 per SM: uniform 16M 1.06 ms of binning against 1.07 with 8)
    const unsigned grid = (unsigned) std::max<uint32_t>(1u, std::min<uint32_t>(ceil_div(n + 1, 256), sms * (gate ? 8 : 32)));
    chain(boundary_starts_kernel, grid, 256, 0, st, b.keys[b.result], b.vals[b.result], n, g.nbins, longest_run(n), start,
          gaps, gap_cap, fs, gate);
    chain(cell_gap_fill_kernel, sms * 2, 256, 0, st, gaps, gap_cap, start, fs, gate);
    return cudaGetLastError();
}

}  // namespace p2v
