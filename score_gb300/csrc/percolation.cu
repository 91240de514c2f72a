// Percolation analysis on the device: the clusters of recrystallized and infected cells
// (caHdl::log_PERCOLATION, SCORE_OnTheFlyCharacterization.cpp:777-875, and its percAnalyzer,
// SCORE_PercAnalyzer.cpp), as a parallel union-find instead of the reference's sequential
// Hoshen-Kopelman scan.
//
// The scan's union-find ends with the connected components of the links it makes, and every link
// is decided by the cell and its three lower neighbours alone (hk3d_core_nonperiodic, :161-226): a
// cell links to each lower neighbour (-x, -y, -z) that is a 1-cell other than the origin (labels are
// cell indices and 0 means "not recrystallized", so the origin never joins a cluster), except that
// with all three present it links to the lower y and z neighbours only (:218-225).  So the
// reference's clusters are found exactly by linking those pairs in any order (SCORE_PERC_REFERENCE);
// SCORE_PERC_CONNECTED links all present lower neighbours: the true 6-connected clusters.
//
// The 1-cells are packed into 32-bit words along y, whose links every mode makes, so that the links along y inside a
// word are bits, not unions: a cell belongs to the head of its run, only heads have a parent, and a link along x
// or z is made once for each pair of runs that touch instead of once a cell (one union-find entry and up to three
// unions a cell, in seven passes over N-word arrays: 0.84 ms at 256^3, 15 % recrystallized; runs along x, which the
// reference's scan leaves unlinked inside a cluster: 0.75 ms).
// Kernels: bits (from the device's bricks), runs (links along y, heads), link (lock-free union: the larger root
// is attached to the smaller with atomicCAS, path halving in find), flatten (every head's root, clusters' sizes and
// face bits for percolates (:500-615), a run at a time, one bit a root in cell order), then the compaction of
// compactify (:334-390): clusters numbered in the order of their first cell, which is the root (the smallest index
// of a cluster) order, by a count / scan / assign pass over the root bits; then the labels.  The size distribution
// (:617-656) is sorted on the host.
#include "percolation.h"

#include <algorithm>
#include <vector>

namespace score {
namespace {

constexpr uint32_t kPercTile = 256;           // words per count / assign tile
constexpr uint32_t kFindLimit = 1u << 24;     // bounded pointer chasing: a longer chain flags an error
constexpr uint32_t kUniteLimit = 1u << 20;    // bounded link retries

// word (x, v, z), at (z V + v) nx + x, holds cells (x, 32 v .. 32 v + 31, z)
struct PercArgs {
    uint32_t nx, ny, nz, V, words;
    const uint32_t* ones;      // 1-cells
    uint32_t* parent;          // of run heads: cell index
    uint32_t* size;            // of roots: cells, then the compact label
    uint32_t* face;            // of roots: touched faces
    uint32_t* roots;           // a bit a cell, in cell order
    uint32_t rootwords;
};
// cell index of bit 0 of a word; x, v, z of it
__device__ __forceinline__ uint32_t word_cell(const PercArgs& a, uint32_t i, uint32_t& x, uint32_t& v, uint32_t& z) {
    const uint32_t q = i / a.nx;
    x = i - q * a.nx;
    z = q / a.V;
    v = q - z * a.V;
    return x + a.nx * (32u * v + a.ny * z);
}

__device__ __forceinline__ uint32_t find_root(uint32_t* parent, uint32_t x, uint32_t* err) {
    for (uint32_t k = 0; k < kFindLimit; ++k) {
        const uint32_t p = parent[x];
        if (p == x) return x;
        const uint32_t g = parent[p];
        if (g != p) parent[x] = g;  // path halving: g is an ancestor of x, any interleaving keeps the forest
        x = p;
    }
    atomicOr(err, 1u);
    return x;
}

__device__ __forceinline__ void unite(uint32_t* parent, uint32_t a, uint32_t b, uint32_t* err) {
    for (uint32_t k = 0; k < kUniteLimit; ++k) {
        a = find_root(parent, a, err);
        b = find_root(parent, b, err);
        if (a == b) return;
        if (a < b) { const uint32_t t = a; a = b; b = t; }
        const uint32_t old = atomicCAS(&parent[a], a, b);  // attach the larger root below the smaller
        if (old == a) return;
        a = old;  // a was attached elsewhere meanwhile: retry from its new parent
    }
    atomicOr(err, 2u);
}

// first bit of the run of bit p inside its word: the highest bit at or below p whose lower neighbour is not set
__device__ __forceinline__ uint32_t run_head(uint32_t ones, uint32_t p) {
    return 31u - (uint32_t)__clz(~(ones << 1) & (0xFFFFFFFFu >> (31u - p)));
}

// A warp packs 32 x 32 cells of a z layer: rows along x by ballots, then the transpose of the bits; two layers a block, so
// that a brick's sector is read from L1 by the other layer and row.
__global__ void __launch_bounds__(256) k_perc_bits(const uint32_t* grid, uint32_t gbx, uint32_t gby, uint32_t nx, uint32_t ny, uint32_t nz,
                                                   uint32_t ndefg, uint32_t V, uint32_t* ones) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t bx = (nx + 31) / 32, pairs = (nz + 1) / 2, jobs = bx * V * pairs;
    for (uint32_t j = blockIdx.x * 4u + (warp >> 1); j < jobs; j += gridDim.x * 4u) {
        const uint32_t x = 32u * (j % bx) + lane, v = (j / bx) % V, z = 2u * (j / (bx * V)) + (warp & 1u);
        if (z >= nz) continue;  // uniform over the warp
        uint32_t mine = 0;  // row `lane`, bits along x
#pragma unroll 8
        for (uint32_t r = 0; r < 32; ++r) {
            const uint32_t y = 32u * v + r;
            bool one = false;
            if (x < nx && y < ny && (x | y | z))
                one = grid[(((z >> 1) * gby + (y >> 1)) * gbx + (x >> 1)) * 8u + ((z & 1u) << 2 | (y & 1u) << 1 | (x & 1u))] >= ndefg;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, one);
            if (lane == r) mine = m;
        }
        uint32_t out = 0;
#pragma unroll
        for (uint32_t k = 0; k < 32; ++k) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (mine >> k) & 1u);
            if (lane == k) out = m;
        }
        if (x < nx) ones[((uint64_t)z * V + v) * nx + x] = out;
    }
}

// run heads start as their own roots
__global__ void __launch_bounds__(256) k_perc_runs(PercArgs a) {
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < a.words; i += gridDim.x * 256u) {
        const uint32_t o = a.ones[i];
        if (!o) continue;
        uint32_t x, v, z;
        const uint32_t cell0 = word_cell(a, i, x, v, z);
        for (uint32_t h = o & ~(o << 1); h; h &= h - 1u) {
            const uint32_t c = cell0 + a.nx * (uint32_t)(__ffs(h) - 1);
            a.parent[c] = c;
            a.size[c] = 0u;
            a.face[c] = 0u;
        }
    }
}

// The links between runs: to the word before along y, and to the lower neighbours in z and x, once for each pair of runs
// that touch (where the cell before along y made the link and both cells are linked to the ones before them, it is
// there already).  The reference's scan makes the link along x only where a lower neighbour in y or z is missing.
__global__ void __launch_bounds__(256) k_perc_link(PercArgs a, int mode, uint32_t* err) {
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < a.words; i += gridDim.x * 256u) {
        const uint32_t o = a.ones[i];
        if (!o) continue;
        uint32_t x, v, z;
        const uint32_t cell0 = word_cell(a, i, x, v, z);
        const uint32_t before = v ? a.ones[i - a.nx] : 0u, oz = z ? a.ones[i - a.nx * a.V] : 0u, ox = x ? a.ones[i - 1] : 0u;
        const uint32_t oy = (o << 1) | (before >> 31);  // the lower neighbour along y is a 1-cell
        if (o & oy & 1u) unite(a.parent, cell0, cell0 - a.nx * (32u - run_head(before, 31u)), err);
        const uint32_t pz = o & oz;
        for (uint32_t m = pz & ~((o & oz & pz) << 1); m; m &= m - 1u) {
            const uint32_t p = (uint32_t)(__ffs(m) - 1);
            unite(a.parent, cell0 + a.nx * run_head(o, p), cell0 - a.nx * a.ny + a.nx * run_head(oz, p), err);
        }
        uint32_t px = o & ox;
        if (mode == SCORE_PERC_REFERENCE) px &= ~(oy & oz);
        for (uint32_t m = px & ~((o & ox & px) << 1); m; m &= m - 1u) {
            const uint32_t p = (uint32_t)(__ffs(m) - 1);
            unite(a.parent, cell0 + a.nx * run_head(o, p), cell0 - 1u + a.nx * run_head(ox, p), err);
        }
    }
}

// Every head's root, a bit for each root, and the clusters' sizes and faces a run at a time; a warp's last clusters add
// together, so that a cluster over most of the domain gets one atomic a warp.  The walk only reads: path halving
// here could overwrite the root another thread just stored for its own head with an older ancestor.
__global__ void __launch_bounds__(256) k_perc_flatten(PercArgs a, uint32_t* err) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    uint32_t cur = 0xFFFFFFFFu, sum = 0, bits = 0;
    const uint32_t o = i < a.words ? a.ones[i] : 0u;
    if (o) {
        uint32_t x, v, z;
        const uint32_t cell0 = word_cell(a, i, x, v, z);
        const uint32_t xz = (x == 0 ? 1u : 0u) | (x == a.nx - 1 ? 2u : 0u) | (z == 0 ? 16u : 0u) | (z == a.nz - 1 ? 32u : 0u);
        for (uint32_t h = o & ~(o << 1); h; h &= h - 1u) {
            const uint32_t p = (uint32_t)(__ffs(h) - 1), c = cell0 + a.nx * p;
            uint32_t r = a.parent[c], k = 0;
            for (uint32_t q = a.parent[r]; q != r && k < kFindLimit; q = a.parent[r], ++k) r = q;
            if (k == kFindLimit) atomicOr(err, 1u);
            if (r == c) atomicOr(&a.roots[c >> 5], 1u << (c & 31u));
            else a.parent[c] = r;
            const uint32_t run = o >> p, len = run == 0xFFFFFFFFu ? 32u : (uint32_t)(__ffs(~run) - 1);
            const uint32_t f = xz | (v == 0 && p == 0 ? 4u : 0u) | (32u * v + p + len == a.ny ? 8u : 0u);
            if (r != cur) {
                if (sum) { atomicAdd(&a.size[cur], sum); if (bits) atomicOr(&a.face[cur], bits); }
                cur = r; sum = 0; bits = 0;
            }
            sum += len;
            bits |= f;
        }
    }
    const uint32_t m = __match_any_sync(0xFFFFFFFFu, cur);
    sum = __reduce_add_sync(m, sum);
    bits = __reduce_or_sync(m, bits);
    if (cur != 0xFFFFFFFFu && (__ffs(m) - 1) == (int)(threadIdx.x & 31)) {
        atomicAdd(&a.size[cur], sum);
        if (bits) atomicOr(&a.face[cur], bits);
    }
}

// roots per tile of kPercTile words of root bits
__global__ void __launch_bounds__(kPercTile) k_perc_count(PercArgs a, uint32_t* tilecnt) {
    __shared__ uint32_t s_w[kPercTile / 32];
    const uint32_t i = blockIdx.x * kPercTile + threadIdx.x;
    const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, i < a.rootwords ? (uint32_t)__popc(a.roots[i]) : 0u);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (uint32_t k = 0; k < kPercTile / 32; ++k) t += s_w[k];
        tilecnt[blockIdx.x] = t;
    }
}

// exclusive scan of the tile counts by one block; total in *total
__global__ void __launch_bounds__(1024) k_perc_scan(uint32_t* tilecnt, uint32_t ntiles, uint32_t* total) {
    __shared__ uint32_t s_w[32], s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < ntiles; base += 1024) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < ntiles ? tilecnt[i] : 0u;
        uint32_t inc = v;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, w, o);
                if (lane >= o) w += x;
            }
            s_w[lane] = w;
        }
        __syncthreads();
        if (i < ntiles) tilecnt[i] = s_carry + (warp ? s_w[warp - 1] : 0u) + inc - v;
        __syncthreads();
        if (threadIdx.x == 0) s_carry += s_w[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = s_carry;
}

// compact label of every root: 1 + roots before it (the reference's order of first appearance); its size and faces in
// that order, the label in the place of the size
__global__ void __launch_bounds__(kPercTile) k_perc_assign(PercArgs a, const uint32_t* tilebase, uint32_t* csize, uint8_t* cface) {
    __shared__ uint32_t s_w[kPercTile / 32];
    const uint32_t i = blockIdx.x * kPercTile + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t roots = i < a.rootwords ? a.roots[i] : 0u;
    const uint32_t n = (uint32_t)__popc(roots);
    uint32_t inc = n;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, k);
        if (lane >= k) inc += x;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    uint32_t at = tilebase[blockIdx.x] + inc - n;
    for (int w = 0; w < warp; ++w) at += s_w[w];
    for (; roots; roots &= roots - 1u, ++at) {
        const uint32_t c = 32u * i + (uint32_t)(__ffs(roots) - 1);
        csize[at] = a.size[c];
        cface[at] = (uint8_t)a.face[c];
        a.size[c] = at + 1u;
    }
}

// every cell's compact label: a warp takes 32 cells along x, their words and runs are neighbours
__global__ void __launch_bounds__(256) k_perc_label(PercArgs a, uint32_t* label) {
    const uint32_t bx = (a.nx + 31) / 32, lane = threadIdx.x & 31u, jobs = bx * a.ny * a.nz;  // below 2^31: at most N
    for (uint32_t j = (blockIdx.x * 256u + threadIdx.x) >> 5; j < jobs; j += gridDim.x * 8u) {
        const uint32_t row = j / bx, x = 32u * (j - row * bx) + lane, z = row / a.ny, y = row - z * a.ny;
        if (x >= a.nx) continue;
        const uint32_t o = a.ones[(z * a.V + (y >> 5)) * a.nx + x], p = y & 31u;
        uint32_t l = 0;
        if ((o >> p) & 1u) l = a.size[a.parent[x + a.nx * ((y & ~31u) + run_head(o, p) + a.ny * z)]];
        label[x + a.nx * row] = l;
    }
}

}  // namespace

namespace {
uint64_t perc_words(uint32_t nx, uint32_t ny, uint32_t nz) { return (uint64_t)nx * ((ny + 31) / 32) * nz; }
}  // namespace

size_t percolation_scratch(uint32_t nx, uint32_t ny, uint32_t nz) {
    const uint64_t rw = ((uint64_t)nx * ny * nz + 31) / 32, tiles = (rw + kPercTile - 1) / kPercTile;
    return (perc_words(nx, ny, nz) + rw + tiles + 2) * 4;
}

int percolation_analyze(const PercBuffers& b, uint32_t gbx, uint32_t gby, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t ndefg, int mode,
                        cudaStream_t st, int sms, score_perc_result* out, uint32_t* sizes, uint32_t sizes_cap, uint32_t* labels,
                        std::string& err) {
    if (mode != SCORE_PERC_REFERENCE && mode != SCORE_PERC_CONNECTED) { err = "unknown percolation mode"; return SCORE_ERR_ARG; }
    const uint64_t N = (uint64_t)nx * ny * nz;
    PercArgs a{};
    a.nx = nx; a.ny = ny; a.nz = nz;
    a.V = (ny + 31) / 32;
    a.words = (uint32_t)perc_words(nx, ny, nz);  // at most N
    a.rootwords = (uint32_t)((N + 31) / 32);
    const uint32_t ntiles = (a.rootwords + kPercTile - 1) / kPercTile, wtiles = (a.words + 255) / 256;
    uint32_t* const ones = (uint32_t*)b.scratch;
    a.roots = ones + a.words;
    uint32_t* const misc = a.roots + a.rootwords;  // [0] total, [1] error flags; cleared with the root bits
    uint32_t* const tile = misc + 2;
    a.ones = ones;
    a.parent = b.parent; a.size = b.size; a.face = b.label;
    // at most every other cell of a 6-connected structure starts a cluster: sizes, then face bytes, in N words
    uint32_t* const csize = b.compact;
    uint8_t* const cface = (uint8_t*)(csize + N / 2 + 1);
    cudaError_t e = cudaMemsetAsync(a.roots, 0, ((size_t)a.rootwords + 2) * 4, st);
    if (e == cudaSuccess) {
        const uint32_t g = std::min<uint32_t>(wtiles, (uint32_t)sms * 8);
        const uint64_t packs = (uint64_t)((nx + 31) / 32) * a.V * ((nz + 1) / 2), rows = (uint64_t)((nx + 31) / 32) * ny * nz;
        k_perc_bits<<<(uint32_t)std::min<uint64_t>((packs + 3) / 4, (uint64_t)sms * 8), 256, 0, st>>>(b.grid, gbx, gby, nx, ny, nz, ndefg, a.V, ones);
        k_perc_runs<<<g, 256, 0, st>>>(a);
        k_perc_link<<<g, 256, 0, st>>>(a, mode, misc + 1);
        k_perc_flatten<<<wtiles, 256, 0, st>>>(a, misc + 1);
        k_perc_count<<<ntiles, kPercTile, 0, st>>>(a, tile);
        k_perc_scan<<<1, 1024, 0, st>>>(tile, ntiles, misc);
        k_perc_assign<<<ntiles, kPercTile, 0, st>>>(a, tile, csize, cface);
        if (labels) k_perc_label<<<(uint32_t)std::min<uint64_t>((rows + 7) / 8, (uint64_t)sms * 16), 256, 0, st>>>(a, b.label);
        e = cudaGetLastError();
    }
    uint32_t hm[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(hm, misc, 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    std::vector<uint32_t> hs;
    std::vector<uint8_t> hf;
    if (e == cudaSuccess && hm[1] == 0) {
        hs.resize(hm[0]);
        hf.resize(hm[0]);
        if (hm[0]) e = cudaMemcpyAsync(hs.data(), csize, (size_t)hm[0] * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && hm[0]) e = cudaMemcpyAsync(hf.data(), cface, (size_t)hm[0], cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && labels) e = cudaMemcpyAsync(labels, b.label, N * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) { err = std::string("percolation: ") + cudaGetErrorString(e); return SCORE_ERR_CUDA; }
    if (hm[1]) { err = "percolation: a bounded union-find loop gave up"; return SCORE_ERR_TIMEOUT; }
    score_perc_result r{};
    r.n_clusters = hm[0];
    for (uint32_t k = 0; k < hm[0]; ++k) {
        r.largest = std::max(r.largest, hs[k]);
        if ((hf[k] & 3u) == 3u) r.spans |= 1u;
        if ((hf[k] & 12u) == 12u) r.spans |= 2u;
        if ((hf[k] & 48u) == 48u) r.spans |= 4u;
    }
    r.percolates = r.spans != 0;
    r.PL = N ? (double)r.largest / (double)N : 0.0;
    if (out) *out = r;
    if (sizes) {
        std::sort(hs.begin(), hs.end());
        std::copy(hs.begin(), hs.begin() + std::min<size_t>(hs.size(), sizes_cap), sizes);
    }
    return SCORE_OK;
}

}  // namespace score
