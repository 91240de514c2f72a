// Deformed-structure synthesis on the device: the periodic Voronoi label fill of the synthetic
// domains (host_generate.cpp) as a CUDA kernel, bit for bit the host's labels.
//
// The host's search (nearest_exact here) labels a cell with its nearest seed (ties to the lowest id): shells of
// Chebyshev radius r around the cell's home bucket, visited until the nearest distance found is within the
// lower bound r bw / scale of every unvisited bucket, in FP64 (periodic |dx|, division by the metric scale,
// square, sum; no contraction into FMA: this file is compiled with -fmad=false).
// Bound by the FP64 pipe (1/64 rate; 30 to 125 candidates of 16 operations a cell: 256^3 cells, 2,500 seeds
// 92 ms), so a block takes the cells of one bucket, gathers the seeds of the buckets around it into shared
// memory, and FP32 finds each cell's nearest seed and everything as near within the rounding; only those, when
// there is more than one, are compared in FP64, with the host's operations.  A seed that FP32 leaves out is
// farther than the nearest by more than the rounding, so every label is the host's; an exact tie goes
// through the host's search itself.  The seeds, orientations, densities and nuclei stay on the host's random
// stream; the fill consumes no random numbers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/score_gb300.h"
#include "host_generate.h"

namespace {

struct VoronoiDev {
    uint32_t n[3], nb[3];
    double scale[3], bw[3];
    int unit_scale;                 // every scale is 1: the division is skipped (x / 1.0 == x)
    const double* pos;
    const uint32_t* start;
    const uint32_t* items;
};

__device__ __forceinline__ double seed_d2(const VoronoiDev& v, uint32_t s, const double c[3]) {
    double r = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double d = fabs(__dsub_rn(c[a], __ldg(&v.pos[3 * s + a])));
        const double e = __dsub_rn((double)v.n[a], d);
        if (e < d) d = e;
        if (!v.unit_scale) d = __ddiv_rn(d, v.scale[a]);
        r = __dadd_rn(r, __dmul_rn(d, d));
    }
    return r;
}

// the host's search for one cell
__device__ __noinline__ uint32_t nearest_exact(const VoronoiDev& v, uint32_t x, uint32_t y, uint32_t z) {
    const int nbx = (int)v.nb[0], nby = (int)v.nb[1], nbz = (int)v.nb[2];
    const int maxr = max(nbx, max(nby, nbz));
    const double c[3] = {x + 0.5, y + 0.5, z + 0.5};
    int home[3] = {(int)__ddiv_rn(c[0], v.bw[0]), (int)__ddiv_rn(c[1], v.bw[1]), (int)__ddiv_rn(c[2], v.bw[2])};
    if (home[0] >= nbx) home[0] = nbx - 1;
    if (home[1] >= nby) home[1] = nby - 1;
    if (home[2] >= nbz) home[2] = nbz - 1;
    double best = 1e300;
    uint32_t arg = 0xFFFFFFFFu;
    for (int r = 0; r <= maxr; ++r) {
        for (int dz = -r; dz <= r; ++dz)
            for (int dy = -r; dy <= r; ++dy)
                for (int dx = -r; dx <= r; ++dx) {
                    if (max(abs(dx), max(abs(dy), abs(dz))) != r) continue;
                    const int bx = ((home[0] + dx) % nbx + nbx) % nbx;
                    const int by = ((home[1] + dy) % nby + nby) % nby;
                    const int bz = ((home[2] + dz) % nbz + nbz) % nbz;
                    const uint32_t b = (uint32_t)bx + v.nb[0] * ((uint32_t)by + v.nb[1] * (uint32_t)bz);
                    const uint32_t e = __ldg(&v.start[b + 1]);
                    for (uint32_t k = __ldg(&v.start[b]); k < e; ++k) {
                        const uint32_t s = __ldg(&v.items[k]);
                        const double d = seed_d2(v, s, c);
                        if (d < best || (d == best && s < arg)) { best = d; arg = s; }
                    }
                }
        double lb = 1e300;
#pragma unroll
        for (int a = 0; a < 3; ++a) lb = fmin(lb, __ddiv_rn(__dmul_rn((double)r, v.bw[a]), v.scale[a]));
        if (arg != 0xFFFFFFFFu && best <= __dmul_rn(lb, lb)) break;
    }
    return arg;
}

constexpr uint32_t kSeedCap = 1024;  // seeds in shared memory

// first cell of bucket b along an axis of n cells (every cell belongs to one bucket; where rounding puts a cell
// on a boundary does not matter: the bounds below are taken from the cell itself)
__device__ __forceinline__ uint32_t bucket_cell(uint32_t b, uint32_t nb, uint32_t n, double bw) {
    if (b >= nb) return n;
    const double c = ceil((double)b * bw - 0.5);
    return c <= 0.0 ? 0u : min(n, (uint32_t)c);
}

// Block (bucket, part): the part's share of the bucket's cells, 256 at a time.  Distances in FP32 are in units of the finest
// axis' scale, so that their squares stay in range whatever the scales.  Error of a squared distance D^2: a
// seed's position relative to the bucket is rounded once (2^-24 of its size, at most the domain's largest
// edge), the cell's twice and the difference once, so a component is off by at most e = 4 u, u = 2^-24 edge, D^2 by
// 2 sqrt(3) e D + 3 e^2 + 6e-7 D^2; `tol` is above that.
__global__ void __launch_bounds__(256) k_voronoi_fill(VoronoiDev v, uint32_t parts, uint32_t* grid) {
    __shared__ float4 s_seed[kSeedCap];  // position relative to the bucket's first cell, id
    __shared__ uint32_t s_n;
    __shared__ float s_below[3], s_above[3];  // from the bucket's first cell to the ends of the slab of buckets
    uint32_t b[3], lo[3], w[3];
    b[0] = blockIdx.x % v.nb[0];
    b[1] = (blockIdx.x / v.nb[0]) % v.nb[1];
    b[2] = blockIdx.x / (v.nb[0] * v.nb[1]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = bucket_cell(b[a], v.nb[a], v.n[a], v.bw[a]);
        w[a] = bucket_cell(b[a] + 1, v.nb[a], v.n[a], v.bw[a]) - lo[a];
    }
    const uint64_t M = (uint64_t)w[0] * w[1] * w[2];
    const uint64_t m_end = M * (blockIdx.y + 1) / parts;
    const double fine = fmin(v.scale[0], fmin(v.scale[1], v.scale[2]));
    const float inv[3] = {(float)(fine / v.scale[0]), (float)(fine / v.scale[1]), (float)(fine / v.scale[2])};
    const float edge = (float)max(v.n[0], max(v.n[1], v.n[2]));
    const float u = 5.9604645e-8f * edge, tol0 = 64.0f * u * u, tol1 = 16.0f * u, tol2 = 1.5e-6f;
    int have = 0;  // radius of the seeds in shared memory
    for (uint64_t m0 = M * blockIdx.y / parts; m0 < m_end; m0 += 256) {
        const uint64_t m = m0 + threadIdx.x;
        const bool cell = m < m_end;
        const uint32_t mm = cell ? (uint32_t)m : 0u;  // a bucket has fewer than 2^32 cells
        const uint32_t lx = mm % w[0], ly = (mm / w[0]) % w[1], lz = mm / (w[0] * w[1]);
        const float c[3] = {lx + 0.5f, ly + 0.5f, lz + 0.5f};
        bool done = !cell;
        uint32_t arg = 0xFFFFFFFFu;
        for (int r = 1;; ++r) {
            // buckets b - r .. b + r along each axis, or all of them
            uint32_t cnt[3], from[3];
            bool all = true;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const bool whole = 2u * (uint32_t)r + 1u >= v.nb[a];
                cnt[a] = whole ? v.nb[a] : 2u * (uint32_t)r + 1u;
                from[a] = whole ? 0u : (b[a] + v.nb[a] - (uint32_t)r) % v.nb[a];
                all = all && whole;
            }
            if (have != r) {
                __syncthreads();
                if (threadIdx.x == 0) s_n = 0u;
                if (threadIdx.x < 3) {
                    const int a = (int)threadIdx.x;
                    const double first = (double)(a == 0 ? lo[0] : a == 1 ? lo[1] : lo[2]), g = v.bw[a];
                    const double at = (double)(a == 0 ? b[0] : a == 1 ? b[1] : b[2]);
                    s_below[a] = (float)(first - (at - (double)r) * g);
                    s_above[a] = (float)((at + (double)(r + 1)) * g - first);
                }
                __syncthreads();
                const uint32_t nbk = cnt[0] * cnt[1] * cnt[2];
                for (uint32_t k = threadIdx.x; k < nbk; k += 256) {
                    const uint32_t kx = (from[0] + k % cnt[0]) % v.nb[0], ky = (from[1] + (k / cnt[0]) % cnt[1]) % v.nb[1],
                                   kz = (from[2] + k / (cnt[0] * cnt[1])) % v.nb[2];
                    const uint32_t q = kx + v.nb[0] * (ky + v.nb[1] * kz), i0 = __ldg(&v.start[q]), i1 = __ldg(&v.start[q + 1]);
                    const uint32_t at = i1 > i0 ? atomicAdd(&s_n, i1 - i0) : 0u;
                    for (uint32_t i = i0; i < i1 && at + (i - i0) < kSeedCap; ++i) {
                        const uint32_t id = __ldg(&v.items[i]);
                        float p[3];
#pragma unroll
                        for (int a = 0; a < 3; ++a) {  // the image nearest to the bucket
                            double d = __ldg(&v.pos[3 * id + a]) - (double)lo[a];
                            const double n = (double)v.n[a], mid = 0.5 * (double)w[a];
                            if (d - mid > 0.5 * n) d -= n;
                            if (d - mid < -0.5 * n) d += n;
                            p[a] = (float)d;
                        }
                        s_seed[at + (i - i0)] = make_float4(p[0], p[1], p[2], __uint_as_float(id));
                    }
                }
                __syncthreads();
                have = r;
            }
            const uint32_t n = s_n;
            if (n > kSeedCap) {  // more seeds than fit: the host's search (also the end of an unlucky growth of r)
                if (!done) arg = nearest_exact(v, lo[0] + lx, lo[1] + ly, lo[2] + lz);
                have = 0;
                break;
            }
            if (!done) {
                // a cell's distance to a seed by the other image can be the smaller one: min over both
                float best = 3.0e38f, second = 3.0e38f;
                uint32_t at = 0;
                for (uint32_t k = 0; k < n; ++k) {
                    const float4 q = s_seed[k];
                    float dx = fabsf(c[0] - q.x), dy = fabsf(c[1] - q.y), dz = fabsf(c[2] - q.z);
                    dx = fminf(dx, fabsf((float)v.n[0] - dx)) * inv[0];
                    dy = fminf(dy, fabsf((float)v.n[1] - dy)) * inv[1];
                    dz = fminf(dz, fabsf((float)v.n[2] - dz)) * inv[2];
                    const float d = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
                    if (d < best) { second = best; best = d; at = k; }
                    else second = fminf(second, d);
                }
                const float tol = tol0 + tol1 * sqrtf(best) + tol2 * best;
                // every seed not in the list lies beyond the slab of buckets along some axis
                float lb = 3.0e38f;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if (cnt[a] == v.nb[a]) continue;
                    lb = fminf(lb, fmaxf(0.0f, fminf(s_below[a] + c[a], s_above[a] - c[a])) * inv[a]);
                }
                if (n && (all || (best + tol) * 1.00001f <= lb * lb)) {
                    done = true;
                    if (second > best + 2.0f * tol) {
                        arg = __float_as_uint(s_seed[at].w);
                    } else {  // the seeds that FP32 cannot tell apart, in FP64
                        const double x[3] = {lo[0] + lx + 0.5, lo[1] + ly + 0.5, lo[2] + lz + 0.5};
                        double d64 = 1e300;
                        bool tie = false;
                        for (uint32_t k = 0; k < n; ++k) {
                            const float4 q = s_seed[k];
                            float dx = fabsf(c[0] - q.x), dy = fabsf(c[1] - q.y), dz = fabsf(c[2] - q.z);
                            dx = fminf(dx, fabsf((float)v.n[0] - dx)) * inv[0];
                            dy = fminf(dy, fabsf((float)v.n[1] - dy)) * inv[1];
                            dz = fminf(dz, fabsf((float)v.n[2] - dz)) * inv[2];
                            if (__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)) > best + 2.0f * tol) continue;
                            const uint32_t id = __float_as_uint(q.w);
                            const double d = seed_d2(v, id, x);
                            if (d == d64) tie = true;
                            if (d < d64) { d64 = d; arg = id; tie = false; }
                        }
                        if (tie) arg = nearest_exact(v, lo[0] + lx, lo[1] + ly, lo[2] + lz);
                    }
                }
            }
            if (!__syncthreads_or(done ? 0 : 1)) break;
        }
        if (cell) grid[(uint64_t)(lo[0] + lx) + (uint64_t)v.n[0] * ((lo[1] + ly) + (uint64_t)v.n[1] * (lo[2] + lz))] = arg;
    }
}

// The device fill behind score_generate_domain_gpu; the labels go back to the host grid.
int fill_voronoi_device(const score::VoronoiGrid& vg, uint32_t* grid, int device, std::string& err) {
    const uint64_t N = (uint64_t)vg.n[0] * vg.n[1] * vg.n[2];
    const size_t S = vg.pos.size() / 3, NB = vg.start.size();
    cudaError_t e = cudaSetDevice(device);
    int sms = 1;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    char* blk = nullptr;
    const size_t b_pos = ((S * 3 * 8) + 255) & ~(size_t)255, b_st = ((NB * 4) + 255) & ~(size_t)255, b_it = ((S * 4) + 255) & ~(size_t)255;
    if (e == cudaSuccess) e = cudaMalloc((void**)&blk, b_pos + b_st + b_it + N * 4);
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return SCORE_ERR_NOMEM; }
    VoronoiDev v{};
    for (int a = 0; a < 3; ++a) { v.n[a] = vg.n[a]; v.nb[a] = vg.nb[a]; v.scale[a] = vg.scale[a]; v.bw[a] = vg.bw[a]; }
    v.unit_scale = vg.scale[0] == 1.0 && vg.scale[1] == 1.0 && vg.scale[2] == 1.0;
    v.pos = (const double*)blk;
    v.start = (const uint32_t*)(blk + b_pos);
    v.items = (const uint32_t*)(blk + b_pos + b_st);
    uint32_t* d_grid = (uint32_t*)(blk + b_pos + b_st + b_it);
    e = cudaMemcpy((void*)v.pos, vg.pos.data(), S * 3 * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy((void*)v.start, vg.start.data(), NB * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy((void*)v.items, vg.items.data(), S * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        // a block a bucket, and parts of buckets until the GPU has several blocks an SM (few, large grains)
        const uint64_t buckets = (uint64_t)v.nb[0] * v.nb[1] * v.nb[2];
        const uint64_t cells = (N + buckets - 1) / buckets, want = ((uint64_t)sms * 16 + buckets - 1) / buckets;
        const uint32_t parts = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({want, (cells + 255) / 256, 65535}));
        k_voronoi_fill<<<dim3((unsigned)buckets, parts), 256>>>(v, parts, d_grid);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(grid, d_grid, N * 4, cudaMemcpyDeviceToHost);
    cudaFree(blk);
    if (e != cudaSuccess) { err = cudaGetErrorString(e); return SCORE_ERR_CUDA; }
    return SCORE_OK;
}

}  // namespace

extern "C" int score_generate_domain_gpu(const score_gen_params* g, uint32_t* grid, double* defg_quat, double* defg_rho0,
                                         double* rxg_quat, uint32_t* rxg_site, double* rxg_tincub, int device) {
    if (!g) return SCORE_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return SCORE_ERR_NOT_BUILT; }
    if (device < 0 || device >= ndev) return SCORE_ERR_ARG;
    std::string err;
    return score::generate_domain_with(g, grid, defg_quat, defg_rho0, rxg_quat, rxg_site, rxg_tincub,
                                       [&](const score::VoronoiGrid& vg, uint32_t* out) { return fill_voronoi_device(vg, out, device, err); });
}
