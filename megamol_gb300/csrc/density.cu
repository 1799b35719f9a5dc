// Deterministic cell-ordered density gather, its tile statistics, and the grid normalisation.
//
// Reference: ParticlesToDensity::createVolumeCPU (plugins/datatools/src/ParticlesToDensity.cpp:389-747).
// The reference scatters every particle into the (2f+1)^3 nodes of its footprint [c-f, c+f]
// (c = trunc((p-min)/h), f = ceil(r/h), :562-579), wraps node indices with (h+2s)%s in cyclic axes
// while measuring the distance to the unwrapped node (:583-614), and adds rbf(d, sigma*r) (:472-476).
// Here every node gathers instead: a CTA owns a tile of TX*TY*TZ nodes, each thread owns one x-row of
// TX nodes, and the CTA stages the particles of the cell rows around the tile (per cyclic image of the
// tile) in shared memory with coalesced float4 loads. A thread adds its candidates in a fixed order
// (image, cell row (z,y), sorted particle order) with Kahan-compensated FP32 sums, so the result is
// bitwise reproducible. The node set a particle reaches is the reference's footprint intersected with
// the kernel support; nodes outside the support receive exactly zero in the reference as well.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "p2v_common.cuh"
#include "p2v_internal.h"
#include "particle_record.cuh"

namespace p2v {

namespace {

constexpr int GATHER_TX = 8;
constexpr int GATHER_TY = 16;
constexpr int GATHER_TZ = 16;
constexpr int MAX_IMAGES = 8;  // cyclic images per axis a tile may visit

// floor(a / b) for b > 0
__device__ __forceinline__ int floor_div(int a, int b) {
    const int q = a / b;
    return (a % b != 0 && a < 0) ? q - 1 : q;
}

struct Extent {
    int L[3], H[3];     // cell-bin rows [u - L, u + H] can hold candidates of node u
    int klo[3], khi[3]; // cyclic images of the tile to visit
    float eps2_max;
    int ok;
};

// Candidate extents and cyclic images of a tile along axis a (its first node at o3[a]), written to ex: threads 0 to 2 of
// a block take one axis each.
__device__ __forceinline__ void tile_extent(const GridGeo& g, FrameScalars* fs, const int o3[3], const int T3[3], int a,
                                            Extent& ex) {
    const bool bump = g.kernel == 0;
    const float rmax_r = __uint_as_float(fs->rmax_bits);
    const float eps_max = bump ? g.sigma * rmax_r : 3.0f * (g.sigma * rmax_r);
    if (a == 0) {
        ex.ok = rmax_r > 0.0f;
        // enlarged slightly so rounding never prunes a contributing cell row
        ex.eps2_max = eps_max * eps_max * 1.0001f;
    }
    if (!(rmax_r > 0.0f))
        return;
    int E = static_cast<int>(ceilf(eps_max / g.hhi[a] + 1e-3f));
    E = E < 1 ? 1 : E;
    const int F = bump ? static_cast<int>(fminf(ceilf(rmax_r / g.hf[a]), 255.0f)) : E;
    int L = bump ? min(E, F + 1) : E, H = bump ? min(E - 1, F) : E - 1;
    if (L > 100) {  // the Kahan gather keeps staged cell offsets in 8 bits
        atomicOr(&fs->error, ERR_WINDOW_TOO_WIDE);
        L = 100;
        H = min(H, 100);
    }
    int klo = 0, khi = 0;
    if (g.cyc[a]) {
        // images k with [o + k s - L, o + T - 1 + k s + H] meeting the occupied cells
        const int s = g.s[a];
        klo = -floor_div(-(fs->cmin[a] - o3[a] - T3[a] + 1 - H), s);
        khi = floor_div(fs->cmax[a] - o3[a] + L, s);
        if (khi - klo + 1 > MAX_IMAGES) {
            atomicOr(&fs->error, ERR_WINDOW_TOO_WIDE);
            khi = klo + MAX_IMAGES - 1;
        }
    }
    ex.L[a] = L;
    ex.H[a] = H;
    ex.klo[a] = klo;
    ex.khi[a] = khi;
}

// Bound by latency at 14 active lanes per instruction (the nodes' candidate lists differ). Three CTAs per SM (80 registers)
// and the row table's scan by the whole CTA: LJ 864k 0.260 ms, where two CTAs and a one-warp scan took 0.367; four CTAs
// 0.26. How many records it stages: kahan_staged.
template<int TX, int TY, int TZ>
__global__ void __launch_bounds__(TY* TZ, 3) gather_kernel(GridGeo g, const float4* __restrict__ rec_a,
    const int4* __restrict__ rec_b, const uint32_t* __restrict__ start, float* __restrict__ grid,
    TileStats* __restrict__ tiles, FrameScalars* __restrict__ fs, int smax, int rmax) {
    chain_begin();
    constexpr int NT = TY * TZ;
    extern __shared__ __align__(16) unsigned char smem[];
    float* acc_s = reinterpret_cast<float*>(smem);                      // [TX][NT]
    float* acc_c = acc_s + TX * NT;                                      // [TX][NT]
    float4* sp = reinterpret_cast<float4*>(acc_c + TX * NT);             // [smax] phi xyz, support^2
    uint4* sm = reinterpret_cast<uint4*>(sp + smax);                     // [smax] boxes, cells, kernel scale
    uint32_t* row_beg = reinterpret_cast<uint32_t*>(sm + smax);          // [rmax]
    uint32_t* row_off = row_beg + rmax;                                  // [rmax + 1]
    __shared__ double s_dsum[NT / 32];
    __shared__ float s_fmin[NT / 32], s_fmax[NT / 32];
    __shared__ Extent s_ex;
    __shared__ uint32_t s_wsum[NT / 32];

    const int t = threadIdx.x;
    const int ty = t % TY;
    const int tz = t / TY;
    if (blockIdx.x + blockIdx.y + blockIdx.z == 0 && t == 0)
        fs->n_valid = start[g.nbins];
    // tiles cover the slab [zlo, zhi) of the grid (z tile index offset by the slab's first tile)
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = (blockIdx.z + g.zlo / TZ) * TZ;
    const bool row_in = (y0 + ty < g.s[1]) && (z0 + tz >= g.zlo) && (z0 + tz < g.zhi);
    const int T3[3] = {TX, TY, TZ};

#pragma unroll
    for (int k = 0; k < TX; ++k) {
        acc_s[k * NT + t] = 0.0f;
        acc_c[k * NT + t] = 0.0f;
    }

    const bool bump = g.kernel == 0;
    const float E45 = __expf(-4.5f);
    // ---- candidate extents from the largest radius, once per CTA ----
    if (t < 3) {
        const int o3[3] = {x0, y0, z0};
        tile_extent(g, fs, o3, T3, t, s_ex);
    }
    __syncthreads();
    const Extent ex = s_ex;

    if (ex.ok) {
        for (int kz = ex.klo[2]; kz <= ex.khi[2]; ++kz)
            for (int ky = ex.klo[1]; ky <= ex.khi[1]; ++ky)
                for (int kx = ex.klo[0]; kx <= ex.khi[0]; ++kx) {
                    const int u0[3] = {x0 + kx * g.s[0], y0 + ky * g.s[1], z0 + kz * g.s[2]};
                    int wlo[3], whi[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        wlo[a] = min(max(u0[a] - ex.L[a], -1), g.s[a]);
                        whi[a] = max(min(u0[a] + T3[a] - 1 + ex.H[a], g.s[a]), -1);
                    }
                    const int nwy = whi[1] - wlo[1] + 1;
                    const int nwz = whi[2] - wlo[2] + 1;
                    if (nwy > rmax) {
                        if (t == 0)
                            atomicOr(&fs->error, ERR_STAGE_OVERFLOW);
                        continue;
                    }
                    const int planes_per_chunk = rmax / nwy;
                    // This thread's node row (unwrapped) and its candidate cell rows. Each end is first
                    // clamped to the bin range [-1, s]: bins -1 and s hold every particle beyond the box,
                    // so a row range lying wholly outside maps onto them.
                    const int uy = u0[1] + ty, uz = u0[2] + tz;
                    const int ry_lo = max(min(max(uy - ex.L[1], -1), g.s[1]), wlo[1]);
                    const int ry_hi = min(max(min(uy + ex.H[1], g.s[1]), -1), whi[1]);
                    const int rz_lo = max(min(max(uz - ex.L[2], -1), g.s[2]), wlo[2]);
                    const int rz_hi = min(max(min(uz + ex.H[2], g.s[2]), -1), whi[2]);
                    const uint32_t bx_lo = (uint32_t) (wlo[0] + 1), bx_end = (uint32_t) (whi[0] + 2);

                    for (int pz0 = 0; pz0 < nwz; pz0 += planes_per_chunk) {
                        const int pz1 = min(nwz, pz0 + planes_per_chunk);
                        const int nrows = (pz1 - pz0) * nwy;
                        __syncthreads();  // previous users of the row table are done
                        // row table: every cell row's records, and their exclusive scan over the rows, two rows per
                        // thread (rmax <= 2 NT)
                        uint32_t total = 0, cnt[2], sum = 0;
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int r = 2 * t + e;
                            cnt[e] = 0;
                            if (r < nrows) {
                                const int zr = r / nwy;
                                const int zz = wlo[2] + pz0 + zr;
                                const int yy = wlo[1] + r - zr * nwy;
                                const uint32_t rowkey = ((uint32_t) (zz + 1) * g.nb[1] + (uint32_t) (yy + 1)) * g.nb[0];
                                const uint32_t b = start[rowkey + bx_lo];
                                cnt[e] = start[rowkey + bx_end] - b;
                                row_beg[r] = b;
                            }
                            sum += cnt[e];
                        }
                        uint32_t incl = sum;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                            if ((t & 31) >= o)
                                incl += u;
                        }
                        if ((t & 31) == 31)
                            s_wsum[t >> 5] = incl;
                        __syncthreads();
                        uint32_t pre = incl - sum;
#pragma unroll
                        for (int w = 0; w < NT / 32; ++w) {
                            const uint32_t v = s_wsum[w];
                            pre += w < (t >> 5) ? v : 0u;
                            total += v;
                        }
                        if (2 * t < nrows)
                            row_off[2 * t] = pre;
                        if (2 * t + 1 < nrows)
                            row_off[2 * t + 1] = pre + cnt[0];
                        if (t == 0)
                            row_off[nrows] = total;
                        __syncthreads();
                        for (uint32_t cb = 0; cb < total; cb += (uint32_t) smax) {
                            const uint32_t cn = min((uint32_t) smax, total - cb);
                            if (cb > 0)
                                __syncthreads();  // previous chunk fully consumed
                            // ---- stage: coalesced 16-byte loads of the chunk's particle records ----
                            for (uint32_t si = t; si < cn; si += NT) {
                                const uint32_t f = cb + si;
                                int lo = 0, hi = nrows;  // row r with row_off[r] <= f < row_off[r+1]
                                while (hi - lo > 1) {
                                    const int mid = (lo + hi) >> 1;
                                    if (row_off[mid] <= f)
                                        lo = mid;
                                    else
                                        hi = mid;
                                }
                                const uint32_t j = row_beg[lo] + (f - row_off[lo]);
                                const float4 A = rec_a[REC_STRIDE * (size_t) j];
                                const int4 B = rec_b[REC_STRIDE * (size_t) j];
                                const float phi[3] = {A.x, A.y, A.z};
                                const int cf[3] = {B.x, B.y, B.z};
                                const uint32_t meta = (uint32_t) B.w;
                                const float r = A.w;
                                const float eps = bump ? g.sigma * r : 3.0f * (g.sigma * r);
                                int blo[3], bhi[3], crel[3];
                                bool empty = false;
#pragma unroll
                                for (int a = 0; a < 3; ++a) {
                                    const int cr = cf[a] - u0[a];
                                    const float pos = static_cast<float>(cr) + phi[a];
                                    const float eh = eps * g.ihh[a];
                                    // nodes k with |k - pos| < eps / h; a node the rounding drops lies at
                                    // the edge of the support, where the kernel is zero
                                    int lo_a = static_cast<int>(floorf(pos - eh)) + 1;
                                    int hi_a = static_cast<int>(ceilf(pos + eh)) - 1;
                                    if (bump) {
                                        const int f = (int) ((meta >> (8 * a)) & 0xFFu);
                                        const int ctr = cr + (int) ((meta >> (24 + a)) & 1u);
                                        lo_a = max(lo_a, ctr - f);
                                        hi_a = min(hi_a, ctr + f);
                                    }
                                    lo_a = max(lo_a, 0);
                                    hi_a = min(hi_a, T3[a] - 1);
                                    empty = empty || lo_a > hi_a;
                                    blo[a] = lo_a;
                                    bhi[a] = hi_a;
                                    crel[a] = max(min(cr, 120), -120);
                                }
                                uint4 m;
                                if (empty) {
                                    // lo = 127 lies outside every tile, so the y/z box test rejects it
                                    m.x = 0x7Fu | (0x7Fu << 16);
                                    m.y = 0x7Fu;
                                    m.z = 0u;
                                } else {
                                    m.x = (uint32_t) blo[0] | ((uint32_t) (bhi[0] - blo[0]) << 8) |
                                          ((uint32_t) blo[1] << 16) | ((uint32_t) (bhi[1] - blo[1]) << 24);
                                    m.y = (uint32_t) blo[2] | ((uint32_t) (bhi[2] - blo[2]) << 8) |
                                          ((uint32_t) (crel[0] & 0xFF) << 16) | ((uint32_t) (crel[1] & 0xFF) << 24);
                                    m.z = (uint32_t) (crel[2] & 0xFF);
                                }
                                float eps2, inv;
                                if (bump) {
                                    eps2 = eps * eps;
                                    inv = __frcp_rn(eps2);
                                } else {
                                    const float sg = g.sigma * r;
                                    eps2 = 9.0f * sg * sg;
                                    inv = __frcp_rn(2.0f * sg * sg);
                                }
                                m.w = __float_as_uint(inv);
                                sp[si] = make_float4(phi[0], phi[1], phi[2], eps2);
                                sm[si] = m;
                            }
                            __syncthreads();
                            // ---- accumulate: this thread's node row against its candidate rows ----
                            if (row_in) {
                                const int zr_lo = max(rz_lo, wlo[2] + pz0), zr_hi = min(rz_hi, wlo[2] + pz1 - 1);
                                for (int zz = zr_lo; zz <= zr_hi; ++zz) {
                                    // smallest z distance from this node row to cell row zz
                                    const int oz = zz - uz;
                                    const float gz = oz > 0 ? oz * g.hhi[2] : (oz < -1 ? (-oz - 1) * g.hhi[2] : 0.0f);
                                    for (int yy = ry_lo; yy <= ry_hi; ++yy) {
                                        const int oy = yy - uy;
                                        const float gy = oy > 0 ? oy * g.hhi[1] : (oy < -1 ? (-oy - 1) * g.hhi[1] : 0.0f);
                                        // bins -1 and s hold particles from arbitrarily far away: never pruned
                                        if (gy * gy + gz * gz >= ex.eps2_max && yy >= 0 && yy < g.s[1] && zz >= 0 &&
                                            zz < g.s[2])
                                            continue;
                                        const int r = (zz - wlo[2] - pz0) * nwy + (yy - wlo[1]);
                                        uint32_t a0 = row_off[r], a1 = row_off[r + 1];
                                        a0 = max(a0, cb);
                                        a1 = min(a1, cb + cn);
                                        for (uint32_t i = a0; i < a1; ++i) {
                                            const uint32_t li = i - cb;
                                            const uint4 m = sm[li];
                                            const uint32_t ylo = (m.x >> 16) & 0xFFu, yw = m.x >> 24;
                                            const uint32_t zlo = m.y & 0xFFu, zw = (m.y >> 8) & 0xFFu;
                                            if ((uint32_t) (ty - (int) ylo) > yw || (uint32_t) (tz - (int) zlo) > zw)
                                                continue;
                                            const float4 P = sp[li];
                                            const int cy = (int) (int8_t) (m.y >> 24);
                                            const int cz = (int) (int8_t) (m.z & 0xFFu);
                                            const int cx = (int) (int8_t) ((m.y >> 16) & 0xFFu);
                                            const float dy = g.hhi[1] * (static_cast<float>(ty - cy) - P.y);
                                            const float dz = g.hhi[2] * (static_cast<float>(tz - cz) - P.z);
                                            const float dyz = dy * dy + dz * dz;
                                            if (!(dyz < P.w))
                                                continue;
                                            const float inv = __uint_as_float(m.w);
                                            const int xlo = (int) (m.x & 0xFFu);
                                            const int xhi = xlo + (int) ((m.x >> 8) & 0xFFu);
                                            for (int k = xlo; k <= xhi; ++k) {
                                                const float dx = g.hhi[0] * (static_cast<float>(k - cx) - P.x);
                                                const float d2 = __fmaf_rn(dx, dx, dyz);
                                                if (!(d2 < P.w))
                                                    continue;
                                                // __frcp_rn is the correctly rounded reciprocal; __expf's
                                                // relative error stays below 1e-6 over the argument range
                                                // that yields values above 1e-7 of the kernel maximum.
                                                float v;
                                                if (bump) {
                                                    const float w = __fmaf_rn(-d2, inv, 1.0f);
                                                    v = w > 0.0f ? __expf(-__frcp_rn(w)) : 0.0f;
                                                } else {
                                                    v = fmaxf(__expf(-d2 * inv) - E45, 0.0f);
                                                }
                                                float* ps = acc_s + k * NT + t;
                                                float* pcmp = acc_c + k * NT + t;
                                                const float s = *ps;
                                                const float yv = v - *pcmp;
                                                const float tt = s + yv;
                                                *pcmp = (tt - s) - yv;
                                                *ps = tt;
                                            }
                                        }
                                    }
                                }
                            }
                        }
                    }
                }
    }

    // ---- write the tile and its statistics ----
    double dsum = 0.0;
    float vmin = INFINITY, vmax = -INFINITY;
    if (row_in) {
        float* out = grid + ((size_t) (z0 + tz - g.zlo) * g.s[1] + (y0 + ty)) * g.s[0] + x0;
#pragma unroll
        for (int k = 0; k < TX; ++k) {
            if (x0 + k < g.s[0]) {
                const float v = acc_s[k * NT + t] - acc_c[k * NT + t];
                out[k] = v;
                dsum += (double) v;
                vmin = fminf(vmin, v);
                vmax = fmaxf(vmax, v);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
        vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
        vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if ((t & 31) == 0) {
        s_dsum[t >> 5] = dsum;
        s_fmin[t >> 5] = vmin;
        s_fmax[t >> 5] = vmax;
    }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < NT / 32; ++w) {
            dsum += s_dsum[w];
            vmin = fminf(vmin, s_fmin[w]);
            vmax = fmaxf(vmax, s_fmax[w]);
        }
        TileStats ts;
        ts.sum = dsum;
        ts.vmin = vmin;
        ts.vmax = vmax;
        tiles[(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = ts;
    }
}

// ---------------------------------------------------------------------------------------------
// Particle-major gather with exact, order-independent accumulation. A CTA owns a tile of TX*TY*TZ nodes held in
// shared memory; for every cyclic image of the tile it walks the sorted particle records of the surrounding cell
// rows (16-byte loads) and adds each particle's kernel values to the nodes of its footprint that lie in the tile.
//
// ACC selects the accumulation:
//   ACC_EXACT   the density: every contribution (all below 1) is rounded to a multiple of 2^-32 and summed exactly;
//   ACC_FIXED_W the intensity aggregator (ParticlesToDensity.cpp:509-519): contribution = kernel value times
//               the particle's weight w (wts[j * wstride], sorted order), rounded to a multiple of 1 / wscale
//               with wscale = 2^31 / 2^ceil(log2 max|w|) and summed as a signed 64-bit integer (exact, order
//               independent; absolute resolution 2^-31 of the largest weight);
//   ACC_DOUBLE  the vector aggregator's direction and weight sums (:492-508): FP64 shared-memory atomics of
//               the FP32 contributions. Its finish divides two sums, so small sums need relative accuracy
//               (a fixed-point quantum would erase voxels reached only by kernel tails); the sums depend on
//               the arrival order only at the 1e-16 level, below the final rounding to FP32.
// The result is written with stride ostride.
//
// Bound by issue slots, and on sparse frames by the latency of the phases around the walk (row table, output): 68 % of
// the issue slots on LJ 4M. A warp's 32 lanes take 32 (particle, x-row) items at a time; about 11 lanes add a node in an
// average step of the x loop, and an item costs about 35 instructions around it (LJ 4M 0.278 ms, mixed 64M 1.27 ms,
// uniform 16M 3.67 ms, four passes of 500k 0.128 ms). Before: one addition per node whose old value gave the carry, a
// binary search per item, conversions on the special-function unit and whole batches dealt to the warps: 0.369, 1.75,
// 5.73 and 0.249 ms. Skipping the x loop, uniform 16M takes 1.79 ms, of that 0.18 the box set-up, 0.73 the row table,
// 0.59 the output.
constexpr int ACC_EXACT = 0, ACC_FIXED_W = 1, ACC_DOUBLE = 2;

constexpr int GATHER_RES = 1024;  // threads resident per SM (64 registers each; 1280 at 48 spill: mixed 64M +6 %)

// ACC_EXACT: a contribution of q 2^-32 is added as its two 16-bit halves, q >> 16 to the node's high word and q & 65535
// to its low word (node sum = high 2^16 + low, in 64 bits), by two shared-memory additions whose old values nobody
// reads. Neither word overflows below 2^16 contributions. ACC_FIXED_W does the same with a signed high half. A tile that
// one CTA has to walk with more records than that uses `carry` words instead: q to the low word, the carry of the
// addition that wraps it to the high word (node sum = high 2^32 + low); ACC_FIXED_W 64-bit additions.
constexpr uint32_t SPLIT_MAX_RECORDS = 1u << 15;
constexpr float FIX_INV = 2.3283064365386963e-10f;  // 2^-32

// The two halves of rn(v 2^32), v in [0, 1), from fused multiply-adds: t = floor(v 2^16) and u = rn(rest) sit in the low
// mantissa bits above 2^23. (The same integer as __float2uint_rn(v 2^32): every product and 2^23 - 2^16 t are exact, and
// 2^16 t is even. The conversion instruction runs at a quarter of the rate of each of these.)
__device__ __forceinline__ void fixed_halves(float v, uint32_t& hi, uint32_t& lo) {
    const float t = __fmaf_rz(v, 65536.0f, 8388608.0f);
    const float u = __fmaf_rn(v, 4294967296.0f, __fmaf_rn(__fsub_rn(t, 8388608.0f), -65536.0f, 8388608.0f));
    hi = __float_as_uint(t) - 0x4B000000u;
    lo = __float_as_uint(u) - 0x4B000000u;
}

// The float nearest (ties to even) to x 2^-32; q receives the rounded sum (the float times 2^32, an integer). Sums whose
// float lies below 1 take one 32-bit conversion each way, others 32-bit integer operations and one exact conversion (64-bit
// conversions run on the narrow FP64 pipe of this part).
__device__ __forceinline__ float fixed_to_float(unsigned long long x, unsigned long long& q) {
    if (x < 0xFFFFFF80ull) {  // (2^32 - 128 rounds up)
        const float f = __uint2float_rn((uint32_t) x);
        q = __float2uint_rn(f);
        return f * FIX_INV;
    }
    const int sh = 40 - __clzll(x);  // bits below a 24-bit significand
    unsigned long long m = x >> sh;
    const unsigned long long rem = x & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
    m += (rem > half || (rem == half && (m & 1ull))) ? 1ull : 0ull;  // m <= 2^24
    q = m << sh;
    // m * 2^(sh - 32): the significand converts exactly and the scale is a power of two (sh in [8, 40])
    return __uint2float_rn((uint32_t) m) * __int_as_float((95 + sh) << 23);
}

// x < 2^23 as a float, from full-rate operations
__device__ __forceinline__ float small_float(uint32_t x) {
    return __uint_as_float(0x4B000000u | x) - 8388608.0f;
}

// 1 / w within 2^-23 of itself (w is never subnormal: 1 - x of a float x)
__device__ __forceinline__ float rcp_fast(float w) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(w));
    return y;
}

// The kernel at squared distance d2 inside the support. With x = 1 / w (bump) or d2 inv (Gaussian) its relative error
// against exp(-x) grows with x: 2^-23 x from the reciprocal (or the product) and the (2 + 1.173 x) 2^-23 that CUDA
// documents for __expf, 4.4e-6 at x = 16. Against the kernel's peak (e^-1 and 1) it stays below 1e-6 everywhere.
template<bool BUMP>
__device__ __forceinline__ float kernel_value(float d2, float inv, float e45) {
    if (BUMP) {
        const float w = __fmaf_rn(-d2, inv, 1.0f);
        return w > 0.0f ? __expf(-rcp_fast(w)) : 0.0f;
    }
    return fmaxf(__expf(-d2 * inv) - e45, 0.0f);
}

// Adds a kernel value to a node of the CTA's sums (smem: [nn] low and [nn] high words, or [nn] 64-bit sums).
template<int ACC>
__device__ __forceinline__ void add_node(unsigned char* smem, int nn, uint32_t node, float v, float weight, float wscale,
                                         bool carry) {
    if (ACC == ACC_FIXED_W) {
        // |w wscale| <= 2^31 and v < 0.99: the rounded contribution fits 32 bits
        const int q = __float2int_rn(__fmul_rn(__fmul_rn(v, weight), wscale));
        if (!carry) {
            uint32_t* lo = reinterpret_cast<uint32_t*>(smem) + node;
            atomicAdd(lo, (uint32_t) q & 0xFFFFu);
            atomicAdd(lo + nn, (uint32_t) (q >> 16));
        } else {
            atomicAdd(reinterpret_cast<unsigned long long*>(smem) + node, (unsigned long long) (long long) q);
        }
    } else if (ACC == ACC_DOUBLE) {
        const float c = __fmul_rn(v, weight);  // rbf * val, in float
        if (c != 0.0f)
            atomicAdd(reinterpret_cast<double*>(smem) + node, (double) c);
    } else {
        uint32_t* lo = reinterpret_cast<uint32_t*>(smem) + node;
        uint32_t* hi = lo + nn;
        uint32_t qh, ql;
        fixed_halves(v, qh, ql);
        if (!carry) {
            atomicAdd(lo, ql);
            atomicAdd(hi, qh);
        } else {
            const uint32_t q = (qh << 16) + ql;
            const uint32_t old = atomicAdd(lo, q);
            if (old + q < old)
                atomicAdd(hi, 1u);
        }
    }
}

// Sorted position of the f-th staged record: the row r with row_off[r] <= f < row_off[r + 1] holds it.
__device__ __forceinline__ uint32_t locate_record(const uint32_t* row_off, const uint32_t* row_beg, int nrows,
                                                  uint32_t f) {
    int lo = 0, hi = nrows;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (row_off[mid] <= f)
            lo = mid;
        else
            hi = mid;
    }
    return row_beg[lo] + (f - row_off[lo]);
}

// Crowded tiles (a blob trajectory's centres: 250,000 records in one tile, which one CTA walked for 2 ms while the others
// had finished; 32 frames 26.5 -> 18.7 ms). A tile with more than `limit` records is not walked by its own CTA: that CTA counts its records,
// clears a slot of 64-bit sums in `acc` and queues the tile in parts of `chunk` records; gather_heavy_kernel's CTAs
// take the parts, each adds its sums to the slot, and the part that finishes last writes the tile. Integer sums: the
// same result in any order. fs->heavy counts tiles (from bit 40) and parts; a full queue leaves the tile to its own CTA.
template<int TX, int TY, int TZ, int NT>
struct GatherShared {
    double dsum[NT / 32];
    unsigned long long isum[NT / 32], fsum[NT / 32];
    float fmin[NT / 32], fmax[NT / 32];
    uint32_t wsum[NT / 32];
    uint32_t slot;
    Extent ex;
};

enum WalkMode { WALK_ALL, WALK_PART, WALK_COUNT };
constexpr uint32_t WALK_OVER = 0xFFFFFFFFu;

// One CTA's walk of a tile's records (image by image, row by row). WALK_ALL adds every record, WALK_PART those numbered
// [rlo, rhi), WALK_COUNT none. Returns the number of records, or WALK_OVER as soon as there are more than `limit` (the
// sums are then void). Every thread returns the same.
template<int TX, int TY, int TZ, int NT, int ACC, bool BUMP>
__device__ __forceinline__ uint32_t walk_tile(const GridGeo& g, const float4* __restrict__ rec_a,
    const int4* __restrict__ rec_b, const uint32_t* __restrict__ start, FrameScalars* __restrict__ fs, int rmax,
    const float* __restrict__ wts, int wstride, float wscale, const int o3[3], GatherShared<TX, TY, TZ, NT>& sh,
    unsigned char* smem, WalkMode mode, uint32_t rlo, uint32_t rhi, bool carry, uint32_t limit) {
    constexpr int NN = TX * TY * TZ;
    constexpr bool WEIGHTED = ACC != ACC_EXACT;
    float4* part_a = reinterpret_cast<float4*>(smem + 8 * NN);                  // [NT] (box corner - particle) xyz, eps^2
    uint4* part_b = reinterpret_cast<uint4*>(part_a + NT);                      // [NT] kernel scale, corner node, rows, weight
    uint32_t* row_beg = reinterpret_cast<uint32_t*>(part_b + NT);               // [rmax]
    uint32_t* row_off = row_beg + rmax;                                         // [rmax + 1]
    const int t = threadIdx.x;
    const uint32_t lane = t & 31u, warp = t >> 5;
    const uint32_t le_mask = 0xFFFFFFFFu >> (31u - lane);
    const float E45 = __expf(-4.5f);
    const int T3[3] = {TX, TY, TZ};
    const Extent& ex = sh.ex;
    uint32_t seen = 0;
    for (int kz = ex.klo[2]; kz <= ex.khi[2]; ++kz)
        for (int ky = ex.klo[1]; ky <= ex.khi[1]; ++ky)
            for (int kx = ex.klo[0]; kx <= ex.khi[0]; ++kx) {
                const int u0[3] = {o3[0] + kx * g.s[0], o3[1] + ky * g.s[1], o3[2] + kz * g.s[2]};
                int wlo[3], whi[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    wlo[a] = min(max(u0[a] - ex.L[a], -1), g.s[a]);
                    whi[a] = max(min(u0[a] + T3[a] - 1 + ex.H[a], g.s[a]), -1);
                }
                const int nwy = whi[1] - wlo[1] + 1;
                const int nwz = whi[2] - wlo[2] + 1;
                if (nwy > rmax) {
                    if (t == 0)
                        atomicOr(&fs->error, ERR_STAGE_OVERFLOW);
                    continue;
                }
                const int planes_per_chunk = rmax / nwy;
                const uint32_t bx_lo = (uint32_t) (wlo[0] + 1), bx_end = (uint32_t) (whi[0] + 2);
                for (int pz0 = 0; pz0 < nwz; pz0 += planes_per_chunk) {
                    const int pz1 = min(nwz, pz0 + planes_per_chunk);
                    const int nrows = (pz1 - pz0) * nwy;
                    __syncthreads();
                    // row table: every cell row's records, and their exclusive scan over the rows, two rows per thread
                    // (rmax <= 2 NT), all table reads in flight together
                    uint32_t total = 0, cnt[2], sum = 0;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int r = 2 * t + e;
                        cnt[e] = 0;
                        if (r < nrows) {
                            const int zr = r / nwy;
                            const int zz = wlo[2] + pz0 + zr;
                            const int yy = wlo[1] + r - zr * nwy;
                            const uint32_t rowkey = ((uint32_t) (zz + 1) * g.nb[1] + (uint32_t) (yy + 1)) * g.nb[0];
                            const uint32_t b = start[rowkey + bx_lo];
                            cnt[e] = start[rowkey + bx_end] - b;
                            row_beg[r] = b;
                        }
                        sum += cnt[e];
                    }
                    uint32_t incl = sum;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= (uint32_t) o)
                            incl += u;
                    }
                    if (lane == 31)
                        sh.wsum[warp] = incl;
                    __syncthreads();
                    uint32_t pre = incl - sum;
#pragma unroll
                    for (int w = 0; w < NT / 32; ++w) {
                        const uint32_t v = sh.wsum[w];
                        pre += w < (int) warp ? v : 0u;
                        total += v;
                    }
                    if (2 * t < nrows)
                        row_off[2 * t] = pre;
                    if (2 * t + 1 < nrows)
                        row_off[2 * t + 1] = pre + cnt[0];
                    const uint32_t first = seen;
                    seen = seen + total < seen ? WALK_OVER : seen + total;
                    if (seen > limit)
                        return WALK_OVER;
                    if (mode == WALK_COUNT || (mode == WALK_PART && (seen <= rlo || first >= rhi)))
                        continue;
                    if (t == 0)
                        row_off[nrows] = total;
                    __syncthreads();
                    const uint32_t flo = mode == WALK_PART && rlo > first ? rlo - first : 0u;
                    const uint32_t fhi = mode == WALK_PART ? min(total, rhi - first) : total;
                    // The warps take equal shares of the records, in equal batches of at most 32; every lane derives its
                    // particle's node box, then the warp walks the concatenated (particle, x-row) items 32 at a time. The
                    // next batch is located and loaded one iteration ahead (its latency overlaps the current one's nodes).
                    const uint32_t share = (fhi - flo + NT / 32 - 1u) / (NT / 32);
                    const uint32_t wlo_r = min(flo + warp * share, fhi), whi_r = min(wlo_r + share, fhi);
                    const uint32_t nbatch = (share + 31u) / 32u;
                    const uint32_t step = nbatch > 0 ? (share + nbatch - 1u) / nbatch : 1u;
                    uint32_t jn = 0;
                    float4 An = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    int4 Bn = make_int4(0, 0, 0, 0);
                    if (lane < step && wlo_r + lane < whi_r) {
                        jn = locate_record(row_off, row_beg, nrows, wlo_r + lane);
                        An = rec_a[REC_STRIDE * (size_t) jn];
                        Bn = rec_b[REC_STRIDE * (size_t) jn];
                    }
                    for (uint32_t base = wlo_r; base < whi_r; base += step) {
                        const uint32_t f = base + lane;
                        const uint32_t j = jn;
                        const float4 A = An;
                        const int4 B = Bn;
                        if (lane < step && f + step < whi_r) {
                            jn = locate_record(row_off, row_beg, nrows, f + step);
                            An = rec_a[REC_STRIDE * (size_t) jn];
                            Bn = rec_b[REC_STRIDE * (size_t) jn];
                        }
                        uint32_t nb = 0, bx = 0, by = 1, node0 = 0;
                        float d0[3], eps2 = 0.0f, inv = 0.0f;
                        if (lane < step && f < whi_r) {
                            const float phi[3] = {A.x, A.y, A.z};
                            const int cf[3] = {B.x, B.y, B.z};
                            const uint32_t meta = (uint32_t) B.w;
                            const float r = A.w;
                            const float eps = BUMP ? g.sigma * r : 3.0f * (g.sigma * r);
                            int blo[3], bw[3];
                            bool empty = false;
#pragma unroll
                            for (int a = 0; a < 3; ++a) {
                                const int cr = cf[a] - u0[a];
                                const float pos = static_cast<float>(cr) + phi[a];
                                const float eh = eps * g.ihh[a];
                                // nodes k with |k - pos| < eps / h; a node the rounding drops lies at
                                // the edge of the support, where the kernel is zero
                                int lo_a = static_cast<int>(floorf(pos - eh)) + 1;
                                int hi_a = static_cast<int>(ceilf(pos + eh)) - 1;
                                if (BUMP) {
                                    const int fa = (int) ((meta >> (8 * a)) & 0xFFu);
                                    const int ctr = cr + (int) ((meta >> (24 + a)) & 1u);
                                    lo_a = max(lo_a, ctr - fa);
                                    hi_a = min(hi_a, ctr + fa);
                                }
                                lo_a = max(lo_a, 0);
                                hi_a = min(hi_a, T3[a] - 1);
                                empty = empty || lo_a > hi_a;
                                blo[a] = lo_a;
                                bw[a] = hi_a - lo_a + 1;
                                // node offset from the particle, in cells: (k - cr) - phi = (k - lo) + d0
                                d0[a] = static_cast<float>(lo_a - cr) - phi[a];
                            }
                            if (!empty) {
                                bx = (uint32_t) bw[0];
                                by = (uint32_t) bw[1];
                                nb = by * (uint32_t) bw[2];  // x-rows of the box
                                if (BUMP) {
                                    eps2 = eps * eps;
                                    inv = __frcp_rn(eps2);
                                } else {
                                    const float sg = g.sigma * r;
                                    eps2 = 9.0f * sg * sg;
                                    inv = __frcp_rn(2.0f * sg * sg);
                                }
                                // with the scaled reciprocal that splits a row number into z and y
                                const uint32_t m = (uint32_t) __fdividef(4096.0f, static_cast<float>(bw[1])) + 1u;
                                node0 = (uint32_t) ((blo[2] * TY + blo[1]) * TX + blo[0]) | (m << 16);
                            }
                        }
                        // exclusive prefix of the row counts over the warp; the particles with rows take consecutive slots
                        uint32_t rows = nb;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t u = __shfl_up_sync(0xffffffffu, rows, o);
                            if (lane >= (uint32_t) o)
                                rows += u;
                        }
                        const uint32_t wtotal = __shfl_sync(0xffffffffu, rows, 31);
                        if (wtotal == 0)
                            continue;
                        const uint32_t prow = nb ? rows - nb : 0xFFFFu;  // (at most 32 * 256 rows)
                        const uint32_t full = __ballot_sync(0xffffffffu, nb != 0u);
                        if (nb) {
                            const uint32_t at = warp * 32 + __popc(full & (le_mask >> 1));
                            part_a[at] = make_float4(d0[0], d0[1], d0[2], eps2);
                            part_b[at] = make_uint4(__float_as_uint(inv), node0, prow | (bx << 16) | (by << 24),
                                                    WEIGHTED ? __float_as_uint(wts ? __ldg(wts + (size_t) j * wstride) : 1.0f)
                                                             : 0u);
                        }
                        __syncwarp();
                        uint32_t before = warp * 32 - 1u;  // slots whose rows start before the current 32 items, less one
                        for (uint32_t j0 = 0; j0 < wtotal; j0 += 32) {
                            // bit b: a particle's first row is item j0 + b; the item's particle is the last one that has
                            // started (no search: one reduction and a population count)
                            const uint32_t heads =
                                __reduce_or_sync(0xffffffffu, prow - j0 < 32u ? 1u << (prow - j0) : 0u);
                            const uint32_t slot = before + __popc(heads & le_mask);
                            before += __popc(heads);
                            const uint32_t jj = j0 + lane;
                            if (jj < wtotal) {
                                const float4 PA = part_a[slot];
                                const uint4 PB = part_b[slot];
                                const uint32_t pby = PB.z >> 24, pbx = (PB.z >> 16) & 0xFFu;
                                const uint32_t local = jj - (PB.z & 0xFFFFu);
                                const uint32_t zl = (local * (PB.y >> 16)) >> 12;  // local / by: local < 256, by <= 16
                                const uint32_t yl = local - zl * pby;
                                const float dy = g.hhi[1] * (small_float(yl) + PA.y);
                                const float dz = g.hhi[2] * (small_float(zl) + PA.z);
                                const float dyz = __fmaf_rn(dy, dy, dz * dz);
                                const float re2 = PA.w;
                                if (dyz < re2) {
                                    const float rinv = __uint_as_float(PB.x);
                                    const uint32_t row = (PB.y & 0xFFFFu) + (zl * TY + yl) * TX;
                                    const float pw = WEIGHTED ? __uint_as_float(PB.w) : 0.0f;
                                    float xf = 0.0f;
#pragma unroll(BUMP ? 4 : 2)
                                    for (uint32_t xl = 0; xl < pbx; ++xl, xf += 1.0f) {
                                        const float dx = g.hhi[0] * (xf + PA.x);
                                        const float d2 = __fmaf_rn(dx, dx, dyz);
                                        if (d2 < re2)
                                            add_node<ACC>(smem, NN, row + xl, kernel_value<BUMP>(d2, rinv, E45), pw,
                                                          wscale, carry);
                                    }
                                }
                            }
                        }
                        __syncwarp();
                    }
                }
            }
    return seen;
}

// The 64-bit sums of nodes n .. n + 3, n a multiple of 4 (ACC_DOUBLE: their bits).
template<int NN, int ACC>
__device__ __forceinline__ void node_sums(const unsigned char* smem, int n, bool carry, unsigned long long q[4]) {
    if (ACC == ACC_DOUBLE || (ACC == ACC_FIXED_W && carry)) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(reinterpret_cast<const unsigned long long*>(smem) + n);
        const ulonglong2 a = p[0], b = p[1];
        q[0] = a.x;
        q[1] = a.y;
        q[2] = b.x;
        q[3] = b.y;
        return;
    }
    const uint4 lo = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(smem) + n);
    const uint4 hi = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(smem) + NN + n);
    if (ACC == ACC_FIXED_W) {  // signed high words
        q[0] = (unsigned long long) ((long long) (int) hi.x * 65536) + lo.x;
        q[1] = (unsigned long long) ((long long) (int) hi.y * 65536) + lo.y;
        q[2] = (unsigned long long) ((long long) (int) hi.z * 65536) + lo.z;
        q[3] = (unsigned long long) ((long long) (int) hi.w * 65536) + lo.w;
        return;
    }
    const int sh = carry ? 32 : 16;
    q[0] = ((unsigned long long) hi.x << sh) + lo.x;
    q[1] = ((unsigned long long) hi.y << sh) + lo.y;
    q[2] = ((unsigned long long) hi.z << sh) + lo.z;
    q[3] = ((unsigned long long) hi.w << sh) + lo.w;
}

// Float bits as integers in the floats' order (no NaN), for integer warp reductions, and back.
__device__ __forceinline__ int order_bits(float v) {
    const int b = __float_as_int(v);
    return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float unorder(int b) {
    return __int_as_float(b ^ ((b >> 31) & 0x7FFFFFFF));
}

// Writes a tile (x fastest, coalesced) and its statistics. sums: the tile's slot of 64-bit sums, or null: the CTA's own.
// The density's tile sum is the exact sum of the floats written, in integers (no node pays an FP64 addition: the FP64 pipe
// of this part is 1/64 of the FP32 rate).
template<int TX, int TY, int TZ, int NT, int ACC>
__device__ __forceinline__ void write_tile(const GridGeo& g, const int o3[3], GatherShared<TX, TY, TZ, NT>& sh,
    const unsigned char* smem, const unsigned long long* sums, bool carry, float winv, float* __restrict__ grid, int ostride,
    TileStats* __restrict__ ts_out) {
    constexpr int NN = TX * TY * TZ;
    const int t = threadIdx.x;
    double dsum = 0.0;
    unsigned long long isum = 0ull, fsum = 0ull;  // whole and fractional parts (each below 2^44 for a tile)
    float vmin = INFINITY, vmax = -INFINITY;
    // four nodes along x per thread and round
#pragma unroll 2
    for (int n = 4 * t; n < NN; n += 4 * NT) {
        const int x = o3[0] + n % TX, y = o3[1] + (n / TX) % TY, z = o3[2] + n / (TX * TY);
        if (x >= g.s[0] || y >= g.s[1] || z < g.zlo || z >= g.zhi)
            continue;
        float* out = grid + (((size_t) (z - g.zlo) * g.s[1] + y) * g.s[0] + x) * (size_t) ostride;
        unsigned long long q[4];
        if (sums) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                q[e] = __ldcg(sums + n + e);
        } else {
            node_sums<NN, ACC>(smem, n, carry, q);
        }
        const int m = min(4, g.s[0] - x);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e >= m)
                break;
            float v;
            if (ACC == ACC_EXACT) {
                unsigned long long r;
                v = fixed_to_float(q[e], r);
                isum += r >> 32;
                fsum += r & 0xFFFFFFFFull;
            } else {
                v = ACC == ACC_FIXED_W ? __ll2float_rn((long long) q[e]) * winv
                                       : __double2float_rn(__longlong_as_double((long long) q[e]));
                dsum += (double) v;
            }
            out[e * ostride] = v;
            vmin = fminf(vmin, v);
            vmax = fmaxf(vmax, v);
        }
    }
    if (!ts_out)  // (uniform)
        return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (ACC == ACC_EXACT) {
            isum += __shfl_xor_sync(0xffffffffu, isum, o);
            fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
        } else {
            dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
        }
    }
    vmin = unorder(__reduce_min_sync(0xffffffffu, order_bits(vmin)));
    vmax = unorder(__reduce_max_sync(0xffffffffu, order_bits(vmax)));
    if ((t & 31) == 0) {
        sh.dsum[t >> 5] = dsum;
        sh.isum[t >> 5] = isum;
        sh.fsum[t >> 5] = fsum;
        sh.fmin[t >> 5] = vmin;
        sh.fmax[t >> 5] = vmax;
    }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < NT / 32; ++w) {
            dsum += sh.dsum[w];
            isum += sh.isum[w];
            fsum += sh.fsum[w];
            vmin = fminf(vmin, sh.fmin[w]);
            vmax = fmaxf(vmax, sh.fmax[w]);
        }
        if (ACC == ACC_EXACT)
            dsum = (double) isum + (double) fsum * 2.3283064365386963e-10;
        TileStats ts;
        ts.sum = dsum;
        ts.vmin = vmin;
        ts.vmax = vmax;
        *ts_out = ts;
    }
}

// 2^31 / 2^ceil(log2 max|w|) of the frame's weights, and its inverse (ACC_FIXED_W)
__device__ __forceinline__ void weight_scale(const FrameScalars* fs, float& wscale, float& winv) {
    wscale = winv = 1.0f;
    const float wmax = __uint_as_float(fs->wmax_bits);
    if (wmax > 0.0f) {
        int e;
        frexpf(wmax, &e);  // wmax <= 2^e
        e = max(e, -90);
        wscale = ldexpf(1.0f, 31 - e);
        winv = ldexpf(1.0f, e - 31);
    }
}

template<int NN, int NT>
__device__ __forceinline__ void clear_sums(unsigned char* smem) {
    for (int n = threadIdx.x; n < NN / 2; n += NT)
        reinterpret_cast<uint4*>(smem)[n] = make_uint4(0u, 0u, 0u, 0u);
}

template<int TX, int TY, int TZ, int NT, int ACC, bool BUMP>
__global__ void __launch_bounds__(NT, GATHER_RES / NT) gather_fixed_kernel(const __grid_constant__ GridGeo g,
    const float4* __restrict__ rec_a, const int4* __restrict__ rec_b, const uint32_t* __restrict__ start,
    const __grid_constant__ GatherPasses ps, TileStats* __restrict__ tiles, FrameScalars* __restrict__ fs, int rmax,
    const GatherHeavy hv, uint32_t tiles_z) {
    chain_begin();
    constexpr int NN = TX * TY * TZ;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ GatherShared<TX, TY, TZ, NT> sh;
    const int t = threadIdx.x;
    if (blockIdx.x + blockIdx.y + blockIdx.z == 0 && t == 0)
        fs->n_valid = start[g.nbins];
    // tiles cover the slab [zlo, zhi) of the grid (z tile index offset by the slab's first tile)
    const uint32_t pass = blockIdx.z / tiles_z, bz = blockIdx.z - pass * tiles_z;
    const uint32_t tile = (bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const int o3[3] = {(int) blockIdx.x * TX, (int) blockIdx.y * TY, (int) (bz + g.zlo / TZ) * TZ};
    clear_sums<NN, NT>(smem);
    if (t < 3) {
        const int T3[3] = {TX, TY, TZ};
        tile_extent(g, fs, o3, T3, t, sh.ex);
    }
    float wscale = 1.0f, winv = 1.0f;
    if (ACC == ACC_FIXED_W)
        weight_scale(fs, wscale, winv);
    __syncthreads();
    bool carry = false;
    if (sh.ex.ok) {
        uint32_t seen = walk_tile<TX, TY, TZ, NT, ACC, BUMP>(g, rec_a, rec_b, start, fs, rmax, ps.w[pass], ps.wstride, wscale, o3,
                                                       sh, smem, WALK_ALL, 0u, 0u, false, hv.limit);
        if (seen == WALK_OVER) {
            uint32_t slot = 0xFFFFFFFFu;
            if (hv.cap > 0) {
                seen = walk_tile<TX, TY, TZ, NT, ACC, BUMP>(g, rec_a, rec_b, start, fs, rmax, nullptr, 1, wscale, o3, sh, smem,
                                                      WALK_COUNT, 0u, 0u, false, WALK_OVER - 1u);
                if (t == 0) {
                    sh.slot = slot;
                    if (seen != WALK_OVER) {
                        const uint32_t parts = (seen + hv.chunk - 1u) / hv.chunk;
                        const unsigned long long at = atomicAdd(&fs->heavy, (1ull << 40) | parts);
                        if ((uint32_t) (at >> 40) < hv.cap) {
                            sh.slot = (uint32_t) (at >> 40);
                            hv.tiles[sh.slot] = HeavyTile{tile, pass, (uint32_t) at, parts};
                            hv.done[sh.slot] = 0u;
                        }
                    }
                }
                __syncthreads();
                slot = sh.slot;
            }
            if (slot != 0xFFFFFFFFu) {
                for (int n = t; n < NN; n += NT)
                    hv.sums[(size_t) slot * NN + n] = 0ull;
                return;
            }
            // no slot: this CTA walks the tile, however many records it has
            carry = true;
            clear_sums<NN, NT>(smem);
            walk_tile<TX, TY, TZ, NT, ACC, BUMP>(g, rec_a, rec_b, start, fs, rmax, ps.w[pass], ps.wstride, wscale, o3, sh, smem,
                                           WALK_ALL, 0u, 0u, true, WALK_OVER);
        }
    }
    __syncthreads();
    write_tile<TX, TY, TZ, NT, ACC>(g, o3, sh, smem, nullptr, carry, winv, ps.out[pass], ps.ostride[pass],
                                    pass == 0 ? tiles + tile : nullptr);
}

// The queued parts of crowded tiles: returns at once when there are none.
template<int TX, int TY, int TZ, int NT, int ACC, bool BUMP>
__global__ void __launch_bounds__(NT, GATHER_RES / NT) gather_heavy_kernel(const __grid_constant__ GridGeo g,
    const float4* __restrict__ rec_a, const int4* __restrict__ rec_b, const uint32_t* __restrict__ start,
    const __grid_constant__ GatherPasses ps, TileStats* __restrict__ tiles, FrameScalars* __restrict__ fs, int rmax,
    const GatherHeavy hv, uint32_t tiles_x, uint32_t tiles_y) {
    chain_begin();
    constexpr int NN = TX * TY * TZ;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ GatherShared<TX, TY, TZ, NT> sh;
    const int t = threadIdx.x;
    const unsigned long long queued = fs->heavy;
    const uint32_t items = (uint32_t) queued, ntiles = min((uint32_t) (queued >> 40), hv.cap);
    if (items == 0u || ntiles == 0u)
        return;
    float wscale = 1.0f, winv = 1.0f;
    if (ACC == ACC_FIXED_W)
        weight_scale(fs, wscale, winv);
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
        uint32_t lo = 0, hi = ntiles;  // the last tile whose first part is at or before `it`
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (hv.tiles[mid].first <= it)
                lo = mid;
            else
                hi = mid;
        }
        const HeavyTile ht = hv.tiles[lo];
        if (it < ht.first || it - ht.first >= ht.parts)
            continue;  // parts of a tile that found the queue full
        const uint32_t part = it - ht.first;
        const uint32_t bx = ht.tile % tiles_x, by = (ht.tile / tiles_x) % tiles_y, bz = ht.tile / (tiles_x * tiles_y);
        const int o3[3] = {(int) bx * TX, (int) by * TY, (int) (bz + g.zlo / TZ) * TZ};
        __syncthreads();  // the previous item's sums and flags are read
        clear_sums<NN, NT>(smem);
        if (t < 3) {
            const int T3[3] = {TX, TY, TZ};
            tile_extent(g, fs, o3, T3, t, sh.ex);
        }
        __syncthreads();
        walk_tile<TX, TY, TZ, NT, ACC, BUMP>(g, rec_a, rec_b, start, fs, rmax, ps.w[ht.pass], ps.wstride, wscale, o3, sh, smem,
                                       WALK_PART, part * hv.chunk, part * hv.chunk + hv.chunk, false, WALK_OVER);
        __syncthreads();
        unsigned long long* sums = hv.sums + (size_t) lo * NN;
        for (int n = 4 * t; n < NN; n += 4 * NT) {
            unsigned long long q[4];
            node_sums<NN, ACC>(smem, n, false, q);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (q[e] == 0ull)
                    continue;
                if (ACC == ACC_DOUBLE)
                    atomicAdd(reinterpret_cast<double*>(sums) + n + e, __longlong_as_double((long long) q[e]));
                else
                    atomicAdd(sums + n + e, q[e]);
            }
        }
        __threadfence();  // this part's sums before its count
        __syncthreads();
        if (t == 0)
            sh.slot = atomicAdd(hv.done + lo, 1u);
        __syncthreads();
        if (sh.slot == ht.parts - 1u) {  // every part has added its sums
            __threadfence();
            write_tile<TX, TY, TZ, NT, ACC>(g, o3, sh, smem, sums, false, winv, ps.out[ht.pass], ps.ostride[ht.pass],
                                            ht.pass == 0 ? tiles + ht.tile : nullptr);
        }
    }
}

// Fixed-order reduction of the tile statistics (one block) and the normalisation constants.
__global__ void __launch_bounds__(1024) finalize_kernel(const TileStats* __restrict__ tiles, uint32_t ntiles,
    FrameScalars* __restrict__ fs, int mass_normalize, int minmax_normalize, double voxel_volume) {
    chain_begin();
    __shared__ double s_sum[32];
    __shared__ float s_min[32], s_max[32];
    double sum = 0.0;
    float mn = INFINITY, mx = -INFINITY;
    // a thread's tiles in order, eight loads in flight (85,184 tiles: 45 -> 32 us)
    constexpr uint32_t AHEAD = 8;
    for (uint32_t i0 = threadIdx.x; i0 < ntiles; i0 += AHEAD * blockDim.x) {
        TileStats ts[AHEAD];
#pragma unroll
        for (uint32_t u = 0; u < AHEAD; ++u) {
            const uint32_t i = i0 + u * blockDim.x;
            ts[u] = i < ntiles ? tiles[i] : TileStats{0.0, INFINITY, -INFINITY};
        }
#pragma unroll
        for (uint32_t u = 0; u < AHEAD; ++u) {
            if (i0 + u * blockDim.x < ntiles) {
                sum += ts[u].sum;
                mn = fminf(mn, ts[u].vmin);
                mx = fmaxf(mx, ts[u].vmax);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_sum[threadIdx.x >> 5] = sum;
        s_min[threadIdx.x >> 5] = mn;
        s_max[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (int) min(blockDim.x >> 5, (ntiles + 31u) >> 5);  // the warps that had tiles (27 tiles: 10 -> 8 us)
        for (int w = 1; w < nw; ++w) {
            sum += s_sum[w];
            mn = fminf(mn, s_min[w]);
            mx = fmaxf(mx, s_max[w]);
        }
        fs->mass = sum;
        fs->vmin = mn;
        fs->vmax = mx;
        double ms = 1.0;
        if (mass_normalize && sum > 0.0)
            ms = (double) fs->n_valid / (sum * voxel_volume);
        fs->mass_scale = ms;
        float lo = mn, hi = mx;
        if (mass_normalize) {
            lo = (float) (mn * ms);
            hi = (float) (mx * ms);
        }
        if (minmax_normalize) {
            // ParticlesToDensity.cpp:676-682: rcp = 1 / (max - min); v = (v - min) * rcp
            fs->offset = lo;
            fs->scale = 1.0f / (hi - lo);
            fs->out_min = 0.0f;
            fs->out_max = 1.0f;
        } else {
            fs->offset = 0.0f;
            fs->scale = 1.0f;
            fs->out_min = lo;
            fs->out_max = hi;
        }
    }
}

__global__ void __launch_bounds__(256) normalize_scalar_kernel(float* __restrict__ grid, uint64_t n,
    const FrameScalars* __restrict__ fs, int mass_normalize, int minmax_normalize) {
    chain_begin();
    const float ms = (float) fs->mass_scale;
    const float off = fs->offset, sc = fs->scale;
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
        grid[i] = normalize_one(grid[i], ms, off, sc, mass_normalize, minmax_normalize);
}

// Streams the grid in 16-byte vectors, four per thread per round (many loads in flight); the tail past
// the last whole vector is done element-wise.
__global__ void __launch_bounds__(256) normalize_kernel(float* __restrict__ grid, uint64_t n,
    const FrameScalars* __restrict__ fs, int mass_normalize, int minmax_normalize) {
    chain_begin();
    const float ms = (float) fs->mass_scale;
    const float off = fs->offset, sc = fs->scale;
    float4* g4 = reinterpret_cast<float4*>(grid);
    const uint64_t n4 = n / 4;
    const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = g4[i + u * stride];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            v[u].x = normalize_one(v[u].x, ms, off, sc, mass_normalize, minmax_normalize);
            v[u].y = normalize_one(v[u].y, ms, off, sc, mass_normalize, minmax_normalize);
            v[u].z = normalize_one(v[u].z, ms, off, sc, mass_normalize, minmax_normalize);
            v[u].w = normalize_one(v[u].w, ms, off, sc, mass_normalize, minmax_normalize);
            g4[i + u * stride] = v[u];
        }
    }
    for (; i < n4; i += stride) {
        float4 v = g4[i];
        v.x = normalize_one(v.x, ms, off, sc, mass_normalize, minmax_normalize);
        v.y = normalize_one(v.y, ms, off, sc, mass_normalize, minmax_normalize);
        v.z = normalize_one(v.z, ms, off, sc, mass_normalize, minmax_normalize);
        v.w = normalize_one(v.w, ms, off, sc, mass_normalize, minmax_normalize);
        g4[i] = v;
    }
    const uint64_t t = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x;
    if (t < n - 4 * n4)
        grid[4 * n4 + t] = normalize_one(grid[4 * n4 + t], ms, off, sc, mass_normalize, minmax_normalize);
}

}  // namespace

// z tiles of the slab [zlo, zhi): from the tile holding plane zlo to the one holding plane zhi - 1
uint32_t gather_tiles_z(const GatherConfig& c, const GridGeo& g) {
    return ceil_div((uint32_t) g.zhi, (uint32_t) c.tz) - (uint32_t) (g.zlo / c.tz);
}

uint32_t gather_tile_count(const GatherConfig& c, const GridGeo& g) {
    return ceil_div(g.s[0], c.tx) * ceil_div(g.s[1], c.ty) * gather_tiles_z(c, g);
}

// A chunk of staged records occupies only the threads whose rows it holds, so a crowded tile goes as fast as its chunks are
// large: as many records as fit beside the tile's sums for the CTAs that an SM gets. Density, ms, 1024 records always / this
// rule: 20k particles in 12 tiles of a 17^3 grid 4.51 / 1.10, 100k in 54 tiles 0.60 / 0.19, 500k in 250 tiles 0.44 / 0.25, a
// blob of 500k in 1024 tiles 1.42 / 1.02, LJ 864k (940 records a tile: one chunk) 0.256 / 0.260. 2048 for two CTAs: LJ 0.342.
int kahan_staged(uint32_t tiles, int sms) {
    return tiles <= (uint32_t) sms ? 6400 : tiles <= 2u * (uint32_t) sms ? 2816 : 1728;
}

GatherHeavy gather_heavy_plan(const GatherConfig& c, uint32_t n, int sms, size_t* bytes) {
    GatherHeavy h{};
    *bytes = 0;
    // A part is a quarter of an SM's even share of the records, and a tile is split from one share on: below that, the parts'
    // second row table and their additions to the slot cost more than the tail they take away (a limit of a quarter share:
    // 4.4 M particles with clusters 0.258 against 0.174 ms, 8 M 0.494 against 0.358; the trajectory is the same).
    h.chunk = std::max<uint32_t>(2048u, std::min<uint32_t>(SPLIT_MAX_RECORDS / 4, n / (uint32_t) (sms * 4)));
    h.limit = std::max<uint32_t>(4096u, std::min<uint32_t>(SPLIT_MAX_RECORDS, n / (uint32_t) sms));
    if (c.mode != GATHER_EXACT || n <= SPLIT_MAX_RECORDS) {
        h.limit = SPLIT_MAX_RECORDS;
        return h;
    }
    h.cap = (uint32_t) std::min<uint64_t>(2048, 4ull * n / h.limit + 16);
    *bytes = (size_t) h.cap * ((size_t) c.tx * c.ty * c.tz * sizeof(unsigned long long) + sizeof(HeavyTile) + sizeof(uint32_t));
    return h;
}

namespace {
template<int TX, int TY, int TZ, int NT, int ACC, bool BUMP>
cudaError_t launch_tiles(const GatherConfig& c, const GridGeo& g, cudaStream_t st, const float4* rec_a,
    const int4* rec_b, const uint32_t* start, const GatherPasses& ps, TileStats* tiles, FrameScalars* fs, GatherHeavy hv,
    void* hbuf, int sms) {
    auto kern = gather_fixed_kernel<TX, TY, TZ, NT, ACC, BUMP>;
    // 64-bit sums, 32 bytes of staged particle per thread, the row table
    const size_t smem = (size_t) TX * TY * TZ * sizeof(unsigned long long) + NT * 32 + (size_t) (2 * c.rmax + 1) * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess)
        return e;
    if (hv.cap) {
        hv.sums = static_cast<unsigned long long*>(hbuf);
        hv.tiles = reinterpret_cast<HeavyTile*>(hv.sums + (size_t) hv.cap * TX * TY * TZ);
        hv.done = reinterpret_cast<uint32_t*>(hv.tiles + hv.cap);
    }
    const uint32_t gx = ceil_div(g.s[0], TX), gy = ceil_div(g.s[1], TY), gz = gather_tiles_z(c, g);
    chain(kern, dim3(gx, gy, gz * (uint32_t) ps.count), NT, smem, st, g, rec_a, rec_b, start, ps, tiles, fs, c.rmax, hv, gz);
    if (hv.cap) {
        auto heavy = gather_heavy_kernel<TX, TY, TZ, NT, ACC, BUMP>;
        if ((e = cudaFuncSetAttribute(heavy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)) != cudaSuccess)
            return e;
        chain(heavy, sms * (GATHER_RES / NT), NT, smem, st, g, rec_a, rec_b, start, ps, tiles, fs, c.rmax, hv, gx, gy);
    }
    return cudaGetLastError();
}

template<int ACC, bool BUMP>
cudaError_t launch_exact(const GatherConfig& c, const GridGeo& g, cudaStream_t st, const float4* rec_a,
    const int4* rec_b, const uint32_t* start, const GatherPasses& ps, TileStats* tiles, FrameScalars* fs,
    const GatherHeavy& hv, void* hbuf, int sms) {
    if (c.tx == 16 && c.ty == 16 && c.tz == 16) {
        // 512 threads per tile where the tiles leave SMs idle (20k, 27 tiles: 13.0 against 15.0 us) and for the FP64
        // sums, whose atomics wait longest (vector 500k 0.128 against 0.140 ms); else 256, four CTAs per SM out of step
        // with one another (LJ 4M 0.268 against 0.333 ms)
        if constexpr (ACC != ACC_DOUBLE)
            if (gather_tile_count(c, g) * (uint32_t) ps.count > (uint32_t) sms)
                return launch_tiles<16, 16, 16, 256, ACC, BUMP>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms);
        return launch_tiles<16, 16, 16, 512, ACC, BUMP>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms);
    }
    if (c.tx == 16 && c.ty == 8 && c.tz == 8)
        return launch_tiles<16, 8, 8, 256, ACC, BUMP>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms);
    if (c.tx == 32 && c.ty == 16 && c.tz == 8)
        return launch_tiles<32, 16, 8, 512, ACC, BUMP>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t launch_gather(const GatherConfig& c, const GridGeo& g, const float4* rec_a, const int4* rec_b,
    const uint32_t* start, const GatherPasses& ps, TileStats* tiles, FrameScalars* fs, const GatherHeavy& hv, void* hbuf,
    int sms, cudaStream_t st) {
    if (c.mode == GATHER_EXACT) {
        const bool bump = g.kernel == 0;
        auto run = [&](auto acc) {
            constexpr int ACC = decltype(acc)::value;
            return bump ? launch_exact<ACC, true>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms)
                        : launch_exact<ACC, false>(c, g, st, rec_a, rec_b, start, ps, tiles, fs, hv, hbuf, sms);
        };
        if (ps.mode == GatherPasses::DOUBLE)
            return run(std::integral_constant<int, ACC_DOUBLE>{});
        if (ps.mode == GatherPasses::FIXED)
            return run(std::integral_constant<int, ACC_FIXED_W>{});
        return run(std::integral_constant<int, ACC_EXACT>{});
    }
    if (ps.mode != GatherPasses::DENSITY)
        return cudaErrorInvalidValue;  // the weighted aggregators use the particle-major gather
    if (c.tx != GATHER_TX || c.ty != GATHER_TY || c.tz != GATHER_TZ)
        return cudaErrorInvalidValue;
    auto kern = gather_kernel<GATHER_TX, GATHER_TY, GATHER_TZ>;
    const size_t smem = (size_t) 2 * c.tx * c.ty * c.tz * sizeof(float) + (size_t) c.smax * (sizeof(float4) + sizeof(uint4)) +
                        (size_t) (2 * c.rmax + 1) * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess)
        return e;
    dim3 grd(ceil_div(g.s[0], c.tx), ceil_div(g.s[1], c.ty), gather_tiles_z(c, g));
    chain(kern, grd, c.ty * c.tz, smem, st, g, rec_a, rec_b, start, ps.out[0], tiles, fs, c.smax, c.rmax);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const TileStats* tiles, uint32_t ntiles, FrameScalars* fs, int mass_normalize,
    int minmax_normalize, double, double voxel_volume, cudaStream_t st) {
    chain(finalize_kernel, 1, 1024, 0, st, tiles, ntiles, fs, mass_normalize, minmax_normalize, voxel_volume);
    return cudaGetLastError();
}

cudaError_t launch_normalize_modes(float* grid, uint64_t nvox, const FrameScalars* fs, int mass_normalize,
    int minmax_normalize, int sms, cudaStream_t st) {
    if (!mass_normalize && !minmax_normalize)
        return cudaSuccess;
    // the grid starts 16-byte aligned (cudaMalloc, or a caller's device buffer checked below)
    if (reinterpret_cast<uintptr_t>(grid) % 16 != 0) {
        const unsigned g1 = (unsigned) std::max<uint64_t>(1, std::min<uint64_t>((nvox + 255) / 256, (uint64_t) sms * 16));
        chain(normalize_scalar_kernel, g1, 256, 0, st, grid, nvox, fs, mass_normalize, minmax_normalize);
        return cudaGetLastError();
    }
    const unsigned grd = (unsigned) std::max<uint64_t>(1, std::min<uint64_t>((nvox / 4 + 255) / 256, (uint64_t) sms * 8));
    chain(normalize_kernel, grd, 256, 0, st, grid, nvox, fs, mass_normalize, minmax_normalize);
    return cudaGetLastError();
}

}  // namespace p2v
