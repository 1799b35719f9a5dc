// The plain cone march (mdao_deferred_fragment_ambocc.inc.glsl:9-60) on corner blocks: the eight texels around a
// trilinear sample of a mip level lie together in memory, so a sample is one 32-byte load. The same operations in the
// same order as cone_march.cuh's march: the same bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "ao_internal.h"
#include "cone_device.cuh"
#include "cone_march.cuh"

namespace p2v {
namespace {

constexpr int MARCH_THREADS = 128;

__device__ __forceinline__ void load_block(const float* p, float v[8]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}

__device__ __forceinline__ void store_block(float* p, const float v[8]) {
    asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                 "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(p)
                 : "memory");
}

// Corner blocks of every blocked level in one launch (block 0: zeros). Block (x, y, z) of a level, 0 <= x <= d[0]
// and so on, holds the texels x - 1 .. x, y - 1 .. y, z - 1 .. z (x fastest) as the march reads them: 0 outside the
// level, level 0 saturated. Bound by its 32-byte stores (levels of 129^3 + 65^3 blocks: 24 us, 77 MB).
__global__ void __launch_bounds__(256) corner_blocks_kernel(const __grid_constant__ ConeParams cp,
                                                            const __grid_constant__ ConeBlocks cb,
                                                            float* __restrict__ blocks) {
    chain_begin();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cb.nblocks; i += gridDim.x * blockDim.x) {
        float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        int l = -1;
        for (int k = 0; k < cp.nlevels; ++k)  // levels lie in order; those without blocks are passed over
            if (cb.lv[k].sxy != 0u && i >= cb.lv[k].first)
                l = k;
        if (l >= 0) {
            const uint32_t j = i - cb.lv[l].first;
            const uint32_t z = j / cb.lv[l].sxy, r = j - z * cb.lv[l].sxy;
            const uint32_t y = r / cb.lv[l].sx, x = r - y * cb.lv[l].sx;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                v[c] = tex_fetch<true>(cp.lv[l], (int) x - 1 + (c & 1), (int) y - 1 + ((c >> 1) & 1),
                                       (int) z - 1 + (c >> 2), 0, l == 0 ? cp.sat : 0.0f);
        }
        store_block(blocks + (size_t) 8 * i, v);
    }
}

// floor(c) of |c| < 2^22 from one add rounded down: t = c + 1.5 * 2^23 holds it in its low mantissa bits, t - 1.5 *
// 2^23 is it as a float. Anything else fails the range test of block_sample.
constexpr float FLOOR_MAGIC = 12582912.0f;
constexpr uint32_t FLOOR_BITS = 0x4B400000u;

// trilinear() of level l at normalised point u, bit for bit, from its corner block. A sample outside the level (no
// texel within reach) takes block 0 instead of a branch.
__device__ __forceinline__ float block_sample(const ConeParams& cp, const ConeBlocks& cb, int l, float ux, float uy,
                                              float uz) {
    const ConeBlocks::Level& L = cb.lv[l];
    if (L.sxy == 0u)  // uniform: a level with more texels than samples
        return trilinear<true>(cp.lv[l], ux, uy, uz, cp.border, l == 0 ? cp.sat : 0.0f);
    const float cx = __fmaf_rn(ux, L.fx, -0.5f), cy = __fmaf_rn(uy, L.fy, -0.5f), cz = __fmaf_rn(uz, L.fz, -0.5f);
    const float tx = __fadd_rd(cx, FLOOR_MAGIC), ty = __fadd_rd(cy, FLOOR_MAGIC), tz = __fadd_rd(cz, FLOOR_MAGIC);
    const float wx = __fsub_rn(cx, __fsub_rn(tx, FLOOR_MAGIC)), wy = __fsub_rn(cy, __fsub_rn(ty, FLOOR_MAGIC));
    const float wz = __fsub_rn(cz, __fsub_rn(tz, FLOOR_MAGIC));
    const bool in = cx >= -1.0f && cx < L.fx && cy >= -1.0f && cy < L.fy && cz >= -1.0f && cz < L.fz;
    const uint32_t i = in ? __float_as_uint(tz) * L.sxy + __float_as_uint(ty) * L.sx + (__float_as_uint(tx) + L.off) : 0u;
    float v[8];
    load_block(cb.blocks + (size_t) 8 * i, v);
    const float c00 = lerp_rn(v[0], v[1], wx), c10 = lerp_rn(v[2], v[3], wx);
    const float c01 = lerp_rn(v[4], v[5], wx), c11 = lerp_rn(v[6], v[7], wx);
    return lerp_rn(lerp_rn(c00, c10, wy), lerp_rn(c01, c11, wy), wz);
}

// The plain march (the bits of cone_ao_at): SPLIT one thread per (particle, cone), the particle's cones added in cone
// order by its first thread; else one thread per particle.
// Bound by the load unit: a 32-byte block load takes one data wavefront per lane that does not share its 128-byte
// line. LJ 4M (737 M samples, 8 cones x 32 steps): 2.50 ms, 2.3 ms of it wavefronts; eight 4-byte loads with their
// border checks took 7.77 ms. Lanes keep to one (cone, step) although cones end at different steps (14 of 32 lanes
// busy): letting every lane run on to its next cone (24 busy) needs the step and level tables per lane, and their
// shared-memory reads take the load unit's wavefronts (3.5 ms). 40 registers for twelve blocks per SM: 2.50 ms, 64
// registers 2.68 ms. SPLIT fills the SMs when the particles do not: uniform 100k 0.136 against 0.187 ms; at 4M it costs
// 2 % more (2.72 against 2.68 ms).
// A cone that has left the volume (widened by the coarsest level's border reach) samples only zeros from there on,
// which leave its sum as it is: it ends there. (Not so an infinite sum, which they turn into NaN: levels whose texels may
// lie outside [0, 1] get no walls.)
template<bool SPLIT>
__global__ void __launch_bounds__(MARCH_THREADS, 12) cone_blocks_kernel(const __grid_constant__ ConeParams cp,
    const __grid_constant__ ConeBlocks cb, const float4* __restrict__ xyzr, const float4* __restrict__ nrm, uint32_t n,
    const uint32_t* __restrict__ out_order, float* __restrict__ ao) {
    chain_begin();
    __shared__ float s_acc[SPLIT ? MARCH_THREADS : 1];
    const uint32_t t = threadIdx.x, nc = (uint32_t) cp.ncones;
    uint32_t i, c = 0;
    bool live;
    if (SPLIT) {
        const uint32_t per = MARCH_THREADS / nc, q = t / nc;
        c = t - q * nc;
        i = blockIdx.x * per + q;
        live = q < per && i < n;
    } else {
        i = blockIdx.x * MARCH_THREADS + t;
        live = i < n;
    }
    float x[3], nn[3];
    bool normal = false;
    float ambient = 0.0f;
    if (live)
        normal = surface_point(xyzr[i], nrm[i], x, nn);
    if (normal) {
        float u[3], ex[3], ez[3];
        cone_frame(cp, x, nn, u, ex, ez);
        for (uint32_t cc = c; cc < nc; ++cc) {
            float dir[3], acc = 0.0f, tmax = INFINITY;
            cone_dir(cp, (int) cc, ex, nn, ez, dir);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                // the distance to the wall ahead (an axis the cone does not move along: +-infinity, inside or outside)
                const float gap = dir[a] > 0.0f ? cb.whi - u[a] : u[a] - cb.wlo;
                tmax = fminf(tmax, __fdividef(gap, fabsf(dir[a])) * 1.0001f);
            }
            for (int k = 0; k < cp.nsteps; ++k) {
                const float d = cp.t[k], lod = cp.lod[k];
                if (d > tmax)
                    break;
                const int l0 = min((int) lod, cp.nlevels - 1);
                const float fr = __fsub_rn(lod, (float) l0);
                const float qx = __fmaf_rn(d, dir[0], u[0]), qy = __fmaf_rn(d, dir[1], u[1]);
                const float qz = __fmaf_rn(d, dir[2], u[2]);
                float vis = block_sample(cp, cb, l0, qx, qy, qz);
                if (fr > 0.0f && l0 + 1 < cp.nlevels)
                    vis = __fmaf_rn(fr, block_sample(cp, cb, l0 + 1, qx, qy, qz),
                                    __fmul_rn(__fsub_rn(1.0f, fr), vis));
                acc = __fmaf_rn(__fsub_rn(1.0f, acc), vis, acc);
                if (cp.early_exit && acc > 0.99f)
                    break;
            }
            ambient = __fadd_rn(ambient, acc);
            if (SPLIT)
                break;
        }
        if (SPLIT)
            s_acc[t] = ambient;
    }
    if (SPLIT) {
        __syncthreads();
        ambient = 0.0f;
        if (live && c == 0 && normal)
            for (uint32_t k = 0; k < nc; ++k)
                ambient = __fadd_rn(ambient, s_acc[t + k]);
    }
    if (live && (!SPLIT || c == 0))
        ao[out_order ? out_order[i] : i] = normal ? cone_combine(cp, ambient) : 1.0f;
}

}  // namespace

// Which levels get blocks, for n particles. A level's blocks cost about 10 ps per texel to build and save about 7 ps
// per sample of it, and early exit leaves about half of a cone's samples: blocks from 2.5 samples per texel on (the
// bound is flat: 0.1 to 20 change the uniform 100k frame by 6 %, LJ 4M and the blob trajectory by under 1 %), and at
// most 2^25 blocks (1 GB) a level. None for n = 0.
ConeBlocks cone_block_plan(const ConeParams& cp, bool unit_texels, uint32_t n) {
    ConeBlocks cb{};
    uint32_t samples[MAX_LEVELS] = {};
    for (int k = 0; k < cp.nsteps; ++k) {
        const int l0 = std::min((int) cp.lod[k], cp.nlevels - 1);
        ++samples[l0];
        if (cp.lod[k] - (float) l0 > 0.0f && l0 + 1 < cp.nlevels)
            ++samples[l0 + 1];
    }
    uint64_t off = 1;
    float dmin = INFINITY;
    for (int l = 0; l < cp.nlevels; ++l) {
        ConeBlocks::Level& b = cb.lv[l];
        for (int a = 0; a < 3; ++a)
            dmin = std::min(dmin, cp.lv[l].fd[a]);
        const uint64_t sx = (uint64_t) cp.lv[l].d[0] + 1, sxy = sx * ((uint64_t) cp.lv[l].d[1] + 1);
        const uint64_t nb = sxy * ((uint64_t) cp.lv[l].d[2] + 1);
        if (cp.border != 0 || nb > (1ull << 25) || (double) n * cp.ncones * samples[l] < 2.5 * (double) nb)
            continue;
        b.fx = cp.lv[l].fd[0];
        b.fy = cp.lv[l].fd[1];
        b.fz = cp.lv[l].fd[2];
        b.first = (uint32_t) off;
        b.sx = (uint32_t) sx;
        b.sxy = (uint32_t) sxy;
        // block index of texel floor (x, y, z): first + (z + 1) sxy + (y + 1) sx + x + 1, with the three floors as
        // FLOOR_BITS + floor (32-bit wrap-around)
        b.off = b.first + (1u - FLOOR_BITS) * (b.sxy + b.sx + 1u);
        off += nb;
    }
    cb.nblocks = (uint32_t) off;
    // a level's samples are zero past half a texel outside it; 0.501: the rounding of the sample position and of its
    // texel coordinate, below 0.0005 texels at 4096 texels per axis
    cb.wlo = -0.501f / dmin;
    cb.whi = 1.0f + 0.501f / dmin;
    // no walls where distances do not grow (a cone length below the offset), or where a sum may overflow
    bool walls = unit_texels;
    for (int k = 0; k < cp.nsteps; ++k)
        walls = walls && cp.t[k] >= (k > 0 ? cp.t[k - 1] : 0.0f);
    if (!walls) {
        cb.wlo = -INFINITY;
        cb.whi = INFINITY;
    }
    return cb;
}

cudaError_t launch_cone_blocks(const ConeParams& cp, ConeBlocks cb, float* blocks, const float4* xyzr, const float4* nrm,
                               uint32_t n, const uint32_t* out_order, float* ao, int sms, cudaStream_t st) {
    if (n == 0)
        return cudaSuccess;
    cb.blocks = blocks;
    const unsigned bgrid = (unsigned) std::min<uint32_t>(ceil_div(cb.nblocks, 256), (uint32_t) sms * 32);
    chain(corner_blocks_kernel, bgrid, 256, 0, st, cp, cb, blocks);
    // fewer particles than the SMs hold threads: one thread per (particle, cone)
    if ((uint64_t) n < (uint64_t) sms * 2048) {
        const uint32_t per = (uint32_t) MARCH_THREADS / (uint32_t) cp.ncones;
        chain(cone_blocks_kernel<true>, ceil_div(n, per), MARCH_THREADS, 0, st, cp, cb, xyzr, nrm, n, out_order, ao);
    } else {
        chain(cone_blocks_kernel<false>, ceil_div(n, MARCH_THREADS), MARCH_THREADS, 0, st, cp, cb, xyzr, nrm, n, out_order,
                                                                                        ao);
    }
    return cudaGetLastError();
}

}  // namespace p2v
