// score_gb300 growth context: device memory layout, the per-step launch sequence
// and the host FP64 master-thread work (dt, physics, P on first use).
//
// HBM layout of one domain (N cells; list capacities cap_I = N, cap_B = N or the
// reference's 2(xy+xz+yz) Border limit):
//   grid   u32[N]   deformed id < ndefg | CURRENTLY_INFECTED | ndefg + rxg
//   claim  u32[N]   attempt ordinal of the first infection of this step (0xFFFFFFFF free)
//   front list L (SoA, slot-indexed): fill f64|f32, [comp f32], vel f64|f32, defg u32,
//          rxg u32, xyz u32, dir u8
//   full_L u32[cap_L], recyc_L u32[reccap_L]                 (rebuilt every step)
//   fmask_L, imask_L u32[cap_L/32], tcnt_L u32[2 cap_L/2048]  grow bit masks, tile counts
//   amask, tobm u32[N], ctcnt u32[2 N/256]                    per-full-cell attempt/win masks
//   ptab   u64[nrxg*ndefg] mobility weights P(rxg,defg), filled on first use
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <limits>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/score_gb300.h"
#include "device_common.cuh"
#include "growth_kernels.cuh"
#include "fused_step.cuh"
#include "host_model.h"
#include "percolation.h"

using namespace score;

namespace {

static_assert(offsetof(DevState, nfull) == kStepFieldsOffset, "per-step fields must start at kStepFieldsOffset");

// ------------------------------------------------------------------ small kernels
__global__ void k_gather_u32(const uint32_t* src, const uint32_t* idx, uint32_t n, uint32_t* out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = src[idx[i]];
}

struct NucRec { uint32_t list, slot, site, rxg, defg, pad; double P; };

// nucleus: fill 1.0 (ALMOST_FULLY_INFECTED), infector 26 (f_geo 1.0)
template <bool FP32>
__global__ void k_place_nuclei(DomainArgs a, const NucRec* rec, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const NucRec r = rec[i];
        const DFront& f = a.f[r.list];
        const double mo = mobility(a, r.P);
        const double v = velocity_from_mobility(a, mo, r.defg, 26);
        f.mob[r.slot] = mo;
        if (!FP32) { ((double*)f.fill)[r.slot] = 1.0; ((double*)f.vel)[r.slot] = v; }
        else { ((float*)f.fill)[r.slot] = 1.0f; f.comp[r.slot] = 0.0f; ((float*)f.vel)[r.slot] = (float)v; }
        f.dir[r.slot] = 26 | kStale;
        f.defg[r.slot] = r.defg;
        f.rxg[r.slot] = r.rxg;
        f.xyz[r.slot] = r.site;
        a.grid[r.site] = kCurrentlyInfected;
    }
}

// Nuclei due during the run, placed on the device so that the host needs no round trip:
// candidates in rxg order with the deformed grain of their site and P (computed by the
// host from the loaded grid: a site that is still deformed has its loaded grain).  A
// candidate is placed when its site is still deformed and no earlier candidate of the
// batch has the same site, exactly as the host placement decides; placed nuclei take
// the next slots of their list in candidate order.
struct NucDue { uint32_t site, rxg, defg, list; double P; };
constexpr uint32_t kDueMax = 1024;  // candidates per launch (one block)

template <bool FP32>
__global__ void __launch_bounds__(kDueMax) k_place_due(DomainArgs a, const NucDue* rec, uint32_t n) {
    __shared__ uint32_t s_site[kDueMax];
    __shared__ uint32_t s_wc[2][kDueMax / 32];
    __shared__ uint32_t s_base[2];
    const uint32_t i = threadIdx.x;
    const int warp = (int)(i >> 5), lane = (int)(i & 31);
    NucDue r{};
    if (i < n) { r = rec[i]; s_site[i] = r.site; }
    if (i == 0) { s_base[0] = a.st->next_never[0]; s_base[1] = a.st->next_never[1]; }
    __syncthreads();
    bool ok = false;
    if (i < n && r.site < a.ncells && r.list < 2) {
        ok = a.grid[r.site] < a.ndefg;
        for (uint32_t j = 0; j < i && ok; ++j) if (s_site[j] == r.site) ok = false;
    }
    const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, ok && r.list == 0), b1 = __ballot_sync(0xFFFFFFFFu, ok && r.list == 1);
    if (lane == 0) { s_wc[0][warp] = __popc(b0); s_wc[1][warp] = __popc(b1); }
    __syncthreads();
    const int L = r.list == 1 ? 1 : 0;
    uint32_t rank = __popc((L ? b1 : b0) & lanemask_lt());
    for (int w = 0; w < warp; ++w) rank += s_wc[L][w];
    if (ok) {
        const uint32_t slot = s_base[L] + rank;
        const DFront& f = a.f[L];
        if (slot >= f.cap) {
            atomicOr(&a.st->err, kErrCapacity);
        } else if (L == 1 && a.border_policy == 0 && slot >= a.border_ref_cap) {
            atomicOr(&a.st->err, kErrBorderRef);
        } else {
            const double mo = mobility(a, r.P);
            const double v = velocity_from_mobility(a, mo, r.defg, 26);
            f.mob[slot] = mo;
            if (!FP32) { ((double*)f.fill)[slot] = 1.0; ((double*)f.vel)[slot] = v; }
            else { ((float*)f.fill)[slot] = 1.0f; f.comp[slot] = 0.0f; ((float*)f.vel)[slot] = (float)v; }
            f.dir[slot] = 26 | kStale;
            f.defg[slot] = r.defg;
            f.rxg[slot] = r.rxg;
            f.xyz[slot] = r.site;
            a.grid[r.site] = kCurrentlyInfected;
            a.ptab[(unsigned long long)r.rxg * a.ndefg + r.defg] = (unsigned long long)__double_as_longlong(r.P);
            if (r.P >= 0.0) atomicMax(&a.st->pmax_bits, (unsigned long long)__double_as_longlong(r.P));
        }
    }
    if (i == 0) {
        uint32_t t0 = 0, t1 = 0;
        for (int w = 0; w < (int)(kDueMax / 32); ++w) { t0 += s_wc[0][w]; t1 += s_wc[1][w]; }
        a.st->next_never[0] = s_base[0] + t0;
        a.st->next_never[1] = s_base[1] + t1;
        a.st->nnuc += t0 + t1;
    }
}

__global__ void k_clear_ptab(unsigned long long* ptab, const unsigned long long* idx, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) ptab[idx[i]] = kPtabEmpty;
}

__global__ void k_fill_ptab(unsigned long long* ptab, const unsigned long long* idx, const double* val, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        ptab[idx[i]] = (unsigned long long)__double_as_longlong(val[i]);
}

// labels of the front's cells by the clarify rule (half filled: the rx grain) into the linear map
template <bool FP32>
__global__ void k_labels_front(DomainArgs a, int L, uint32_t n, uint32_t* lab) {
    const DFront& f = a.f[L];
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        if (f.dir[s] == kInactive) continue;
        bool rx;
        if (!FP32) rx = !(((const double*)f.fill)[s] < 0.5);
        else rx = !((((const float*)f.fill)[s] - f.comp[s]) < 0.5f);
        int x, y, z;
        decode(a, f.xyz[s], x, y, z);
        lab[linear_of(a, x, y, z)] = rx ? a.ndefg + f.rxg[s] : f.defg[s];
    }
}

// the grid between the linear order of the C interface and the device's bricks (gindex); the
// padding words of odd extents hold kPadCell, which no attempt can claim
constexpr uint32_t kPadCell = 0xFFFFFFFFu;

// The loaded grid into bricks, and its cells per deformed grain (ids >= ndefg set kErrBounds).  A warp's 32
// grid words are an 8 x 2 x 2 box that lies in one or two grains, so its cells are counted by one atomic a grain:
// one atomic a cell, in a pass of its own, was bound by same-address atomics (422 grains, 56 M cells: load of
// 12.7 ms, now 2.1; 20,000 grains, 134 M cells: 7.2 and 5.7, of which the host copy takes most).  Four boxes a warp in flight; a grain's count stays with the warp while it lasts.
__global__ void __launch_bounds__(kBlock) k_brick(DomainArgs a, const uint32_t* lin, uint32_t* g, uint32_t* cnt) {
    const int lane = threadIdx.x & 31;
    const uint32_t end = (a.ncells + 31u) & ~31u, stride = gridDim.x * blockDim.x;
    uint32_t held = kPadCell, n = 0;  // the grain of the warp's last whole box, and its cells not yet added
    bool bad = false;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < end; i0 += 4u * stride) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = i0 + (uint32_t)k * stride;
            v[k] = kPadCell;
            if (i0 + (uint64_t)k * stride < a.ncells) {
                int x, y, z;
                decode(a, i, x, y, z);
                if (x < (int)a.nx && y < (int)a.ny && z < (int)a.nz) {
                    v[k] = lin[linear_of(a, x, y, z)];
                    bad |= v[k] >= a.ndefg;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i0 + (uint64_t)k * stride < a.ncells) g[i0 + (uint32_t)k * stride] = v[k];
            const uint32_t v0 = __shfl_sync(0xFFFFFFFFu, v[k], 0);
            if (__all_sync(0xFFFFFFFFu, v[k] == v0)) {
                if (v0 != held) {
                    if (lane == 0 && held < a.ndefg) atomicAdd(&cnt[held], n);
                    held = v0; n = 0;
                }
                n += 32;
            } else {
                const uint32_t m = __match_any_sync(0xFFFFFFFFu, v[k]);
                if ((__ffs(m) - 1) == lane && v[k] < a.ndefg) atomicAdd(&cnt[v[k]], (uint32_t)__popc(m));
            }
        }
    }
    if (lane == 0 && held < a.ndefg) atomicAdd(&cnt[held], n);
    if (bad) atomicOr(&a.st->err, kErrBounds);
}
__global__ void k_unbrick(DomainArgs a, const uint32_t* g, uint32_t* lin) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.ncells; i += gridDim.x * blockDim.x) {
        int x, y, z;
        decode(a, i, x, y, z);
        if (x < (int)a.nx && y < (int)a.ny && z < (int)a.nz) lin[linear_of(a, x, y, z)] = g[i];
    }
}

// stable compaction of ACTIVE slots of list L into scratch arrays (ompshar_defragmentation,
// SCORE_Kernel.cpp:3877-3937), in three passes over tiles of kGrowTile slots like the
// grow step: count, one-block scan (k_scan_defrag), move.  Uses the list's tile counts.
__global__ void __launch_bounds__(kBlock) k_defrag_count(DomainArgs a, int L, uint32_t n) {
    const DFront fr = a.f[L];
    const uint32_t ntiles = (n + kGrowTile - 1) / kGrowTile;
    __shared__ uint32_t s_c[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint32_t c = 0;
        for (int k = 0; k < kGrowItems; ++k) {
            const uint32_t s = tile * kGrowTile + (uint32_t)(k * kBlock) + threadIdx.x;
            c += __popc(__ballot_sync(0xFFFFFFFFu, s < n && fr.dir[s] != kInactive));
        }
        if (lane == 0) s_c[warp] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int w = 0; w < kWarps; ++w) t += s_c[w];
            fr.tcnt[2 * tile] = t;
            fr.tcnt[2 * tile + 1] = 0;
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(1024) k_scan_defrag(DomainArgs a, int L, uint32_t n, uint32_t* out_count) {
    uint32_t tA, tB;
    scan_pairs_block(a.f[L].tcnt, (n + kGrowTile - 1) / kGrowTile, tA, tB);
    if (threadIdx.x == 0) *out_count = tA;
}
template <bool FP32>
__global__ void __launch_bounds__(kBlock) k_defrag_compact(DomainArgs a, int L, uint32_t n, DFront scratch) {
    constexpr int ITEMS = kGrowItems;
    const DFront fr = a.f[L];
    const uint32_t ntiles = (n + kGrowTile - 1) / kGrowTile;
    __shared__ uint32_t s_cntA[ITEMS * kWarps], s_cntB[ITEMS * kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = lanemask_lt();
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t base = tile * kGrowTile;
        uint32_t am[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t s = base + (uint32_t)(k * kBlock) + threadIdx.x;
            am[k] = __ballot_sync(0xFFFFFFFFu, s < n && fr.dir[s] != kInactive);
            if (lane == 0) { s_cntA[k * kWarps + warp] = __popc(am[k]); s_cntB[k * kWarps + warp] = 0; }
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t tA, tB;
            scan64_pair(s_cntA, s_cntB, tA, tB);
        }
        __syncthreads();
        const uint32_t ex = fr.tcnt[2 * tile];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            if (!((am[k] >> lane) & 1u)) continue;
            const uint32_t s = base + (uint32_t)(k * kBlock) + threadIdx.x;
            const uint32_t r = ex + s_cntA[k * kWarps + warp] + __popc(am[k] & lt);
            if (!FP32) {
                ((double*)scratch.fill)[r] = ((const double*)fr.fill)[s];
                ((double*)scratch.vel)[r] = ((const double*)fr.vel)[s];
                scratch.inc[r] = fr.inc[s];
                scratch.mob[r] = fr.mob[s];
            } else {
                ((float*)scratch.fill)[r] = ((const float*)fr.fill)[s];
                scratch.comp[r] = fr.comp[s];
                ((float*)scratch.vel)[r] = ((const float*)fr.vel)[s];
                scratch.mob[r] = fr.mob[s];
            }
            scratch.defg[r] = fr.defg[s]; scratch.rxg[r] = fr.rxg[s]; scratch.xyz[r] = fr.xyz[s]; scratch.dir[r] = fr.dir[s];
        }
        __syncthreads();
    }
}

// ---- on-the-fly characterization: RX area profile (log_rxareaprofile(threshold),
// SCORE_OnTheFlyCharacterization.cpp:274-384) over a label map, slices [z0, z1) ----
// section of every rx grain in every slice: hist[(z - z0) nrxg + rxg]; cells of one warp that
// carry the same label add together (a row of cells mostly belongs to one grain)
__global__ void k_area_hist(const uint32_t* lab, uint32_t nxy, uint32_t z0, uint32_t z1, uint32_t ndefg, uint32_t nrxg,
                            uint32_t* hist) {
    // cells and keys of a chunk fit 32 bits: N < 2^31 and the chunk's slices x nrxg <= N
    const uint64_t lo = (uint64_t)z0 * nxy;
    const uint32_t n = (z1 - z0) * nxy, stride = gridDim.x * blockDim.x;
    const uint32_t end = (n + 31u) & ~31u;  // whole warps, so that every lane takes part in the match
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < end; i += stride) {
        uint32_t key = 0xFFFFFFFFu;
        if (i < n) {
            const uint32_t r = lab[lo + i] - ndefg;  // wraps for deformed ids
            if (r < nrxg) key = (i / nxy) * nrxg + r;
        }
        const uint32_t m = __match_any_sync(0xFFFFFFFFu, key);
        if (key != 0xFFFFFFFFu && (__ffs(m) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&hist[key], (uint32_t)__popc(m));
    }
}
// one block per slice: cells of the rx grains whose section reaches the threshold, and the rest;
// clears the slice's histogram for the next use
__global__ void __launch_bounds__(kBlock) k_area_sum(uint32_t* hist, uint32_t nrxg, uint32_t nxy, uint32_t thr, uint32_t* out) {
    __shared__ uint32_t s_w[kWarps];
    uint32_t* h = hist + (uint64_t)blockIdx.x * nrxg;
    uint32_t rx = 0;
    for (uint32_t r = threadIdx.x; r < nrxg; r += blockDim.x) {
        const uint32_t v = h[r];
        if (v >= thr) rx += v;
        h[r] = 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rx += __shfl_xor_sync(0xFFFFFFFFu, rx, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = rx;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kWarps; ++w) t += s_w[w];
        out[2 * blockIdx.x] = t;
        out[2 * blockIdx.x + 1] = nxy - t;
    }
}

// ---- ensemble post-processing (SCORE_SolitaryUnitAveraging.cpp) of the grain-evolution logs ----
// caHdl::get_interpCellCount (SCORE_SolitaryUnitAveraging.cpp:1304-1365) of a grain at time `when`: its final count at
// or after the end of the run, its first count at or before the first snapshot, its last after the last one, else
//   c1 + ((when - t1) * ((c2 - c1) / (t2 - t1)))
// between the snapshots around it.  The slope belongs to the grain and the interval, not to the time: k_rediscr_rows
// makes (c1, slope) once a grain and interval, and a time slot costs a product and a sum on the FP64 pipe (1/64
// rate), where the division made it ten.  A row with slope 0 is the count itself.
struct EvoDev {
    const double* t;              // snapshot times
    const uint32_t* counts;       // nsnap x (ndefg + nrxg)
    const uint32_t* fin_defg;     // counts at the end of the run
    const uint32_t* fin_rxg;
    const uint32_t* order;        // grains by class, in grain order within a class (macrotexture), or null: 0, 1, ...
    const uint32_t* first;        // first place of each class in that order, nclass + 1
    double2* rows;                // (nsnap + 2) x ngr: before the first snapshot, each interval, after the last, the end
    uint32_t ndefg, nrxg, nsnap, ngr;
    double tsimend, nboxvol;
};
__global__ void __launch_bounds__(256) k_rediscr_rows(const EvoDev* doms) {
    const EvoDev e = doms[blockIdx.y];
    const uint32_t G = e.ndefg + e.nrxg;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < e.ngr; q += gridDim.x * blockDim.x) {
        const uint32_t id = e.order ? e.order[q] : q;
        double c1 = (double)e.counts[id], t1 = e.t[0];
        e.rows[q] = make_double2(c1, 0.0);
        for (uint32_t i = 1; i < e.nsnap; ++i) {
            const double c2 = (double)e.counts[(uint64_t)i * G + id], t2 = e.t[i];
            // equal counts: the quotient is 0 (times ascend), no division
            e.rows[(uint64_t)i * e.ngr + q] = make_double2(c1, c2 == c1 ? 0.0 : __ddiv_rn(__dsub_rn(c2, c1), __dsub_rn(t2, t1)));
            c1 = c2; t1 = t2;
        }
        e.rows[(uint64_t)e.nsnap * e.ngr + q] = make_double2(c1, 0.0);
        e.rows[(uint64_t)(e.nsnap + 1) * e.ngr + q] = make_double2((double)(id < e.ndefg ? e.fin_defg[id] : e.fin_rxg[id - e.ndefg]), 0.0);
    }
}
// One thread per (domain, class, time slot), a warp's slots neighbours in time, so that they mostly read the same row:
// the class's grains summed in order (postprocess_rediscr_kinetics, :546-600: one class, the deformed grains, as
// box volume minus the sum; postprocess_rediscr_macrotexture, :673-747).  What bounds it is the FP64 pipe and the
// chain of sums: 16 grains' rows are in flight at a time, and a grain that is not there in the interval costs no
// FP64 operation (x + 0 is x for the sums here, which are never -0).
constexpr uint32_t kMaxClasses = 32;
__global__ void __launch_bounds__(32) k_rediscr_sum(const EvoDev* doms, const double* when, uint32_t nslots, uint32_t nclass, int kinetics,
                                                    double* per_dom) {
    const EvoDev e = doms[blockIdx.z];
    const uint32_t c = blockIdx.y, n = blockIdx.x * 32u + threadIdx.x;
    if (n >= nslots) return;
    const double w = when[n];
    uint32_t r = 0;
    while (r < e.nsnap && e.t[r] < w) ++r;  // the first snapshot at or after it
    double dt = 0.0;
    if (r > 0 && r < e.nsnap) dt = __dsub_rn(w, e.t[r - 1]);
    if (w >= e.tsimend) { r = e.nsnap + 1; dt = 0.0; }
    const uint32_t lo = kinetics ? 0u : e.first[c], hi = kinetics ? e.ndefg : e.first[c + 1];
    const double2* row = e.rows + (uint64_t)r * e.ngr;
    constexpr uint32_t U = 16;
    double acc = 0.0;
    for (uint32_t g = lo; g < hi; g += U) {
        double2 v[U];
#pragma unroll
        for (uint32_t k = 0; k < U; ++k) v[k] = g + k < hi ? __ldg(&row[g + k]) : make_double2(0.0, 0.0);
#pragma unroll
        for (uint32_t k = 0; k < U; ++k) {
            if (__double_as_longlong(v[k].y) != 0) acc = __dadd_rn(acc, __dadd_rn(v[k].x, __dmul_rn(dt, v[k].y)));
            else if (__double_as_longlong(v[k].x) != 0) acc = __dadd_rn(acc, v[k].x);
        }
    }
    per_dom[((uint64_t)blockIdx.z * nslots + n) * nclass + c] = kinetics ? __dsub_rn(e.nboxvol, acc) : acc;
}
// ensemble sums over the domains in order, one thread per output value
__global__ void k_rediscr_ensemble(const double* per_dom, uint32_t ndom, uint32_t m, double* out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    double v = 0.0;
    for (uint32_t d = 0; d < ndom; ++d) v = __dadd_rn(v, per_dom[(uint64_t)d * m + k]);
    out[k] = v;
}

__global__ void k_first_inactive(const uint8_t* dir, uint32_t lo, uint32_t hi, uint32_t* out) {
    for (uint32_t s = lo + blockIdx.x * blockDim.x + threadIdx.x; s < hi; s += gridDim.x * blockDim.x)
        if (dir[s] == kInactive) atomicMin(out, s);
}

inline uint32_t blocks_for(uint64_t work, int sms, int per_sm = 8) {
    uint64_t b = (work + kBlock - 1) / kBlock;
    uint64_t cap = (uint64_t)sms * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (uint32_t)b;
}

template <typename T>
cudaError_t dalloc(T** p, size_t count) {
    return cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T));
}

}  // namespace

// ------------------------------------------------------------------ context
struct Engine;

struct score_ctx {
    score_params prm{};
    int device = 0;
    int sms = 1;
    cudaStream_t stream = nullptr;
    std::string err;
    Physics ph;

    uint32_t nx = 0, ny = 0, nz = 0;
    uint64_t N = 0;
    uint64_t ncells = 0;               // grid words on the device (2x2x2 bricks over the extents rounded up to even)
    uint32_t ndefg = 0, nrxg = 0;
    bool loaded = false, fp32 = false, failed = false;
    int refresh = 0;                   // next step: 1 full refresh from P, 2 from cached mobilities
    std::vector<double> defg_q, rxg_q, rho0, rho, tincub;
    std::vector<uint32_t> site;        // nucleus sites, linear index (x + nx (y + ny z))
    std::vector<uint32_t> gsite;       // the same sites as grid words (brick index)
    std::vector<uint32_t> site_defg;   // deformed grain of each nucleus site in the loaded grid
    std::vector<uint8_t> placed;
    std::vector<uint32_t> nuc_order;   // rxg ids sorted by (tincub, id)
    size_t nuc_pos = 0;                // nuc_order[0, nuc_pos) already considered
    std::vector<uint32_t> defg_cnt_host, defg_cnt_init_host;
    std::vector<double> user_ptab;
    std::vector<double> pforce_host;
    double mob_host[4] = {0, 0, 0, 0};  // mobilities the front's vel factors were computed with
    double dt_cached = -1.0;             // dt the front's cached fill increments were computed with
    double pf_sig[2] = {0, 0};           // Gb^2/2 and drag the driving-force table was computed with
    uint64_t rho_version = 0, pf_rho_version = ~0ull, rhomax_version = ~0ull;
    std::vector<uint32_t> rho_order;   // deformed grains by descending rho0 (rho max while rho == rho0)
    size_t rho_cursor = 0;             // rho_order[0, cursor) have no cells left
    std::vector<double> rho_next;      // rho at the end of the running step (computed while it runs)
    bool ahead = false;                // physics_ahead ran for the running step

    DomainArgs a{};
    DevState* d_state = nullptr;
    DevState* h_state = nullptr;       // pinned host copy of the device scalars (load checks)
    HostBox* h_box = nullptr;          // pinned, device-mapped step mailbox
    HostBox* d_box = nullptr;          // its device address
    double* d_pforce = nullptr;
    double* h_pforce = nullptr;            // pinned staging of the driving forces: two buffers of ndefg, in turn
    int pf_buf = 0;                        // the buffer with the newest
    bool pf_pending = false;               // not on the device yet
    // stepping inside one launch (k_steps_fused)
    uint32_t fuse_seq = 1;                 // number of the next command
    bool fuse_live = false;                // a launch steps this domain: driving forces go by its commands
    bool pre_done = false;                 // pre_step ran for a step that no launch has taken yet
    uint32_t pre_newnuc = 0;
    uint32_t fuse_replay = 0;              // flags of a command that its launch left without seeing (kCmdReplay set)
    FusePay fuse_sent{};                   // the payload the running launch has
    NucDue* h_due = nullptr;               // pinned staging of nuclei due during the run
    NucDue* d_due = nullptr;
    uint32_t* d_grid_init = nullptr;       // the loaded deformed grid (restart source)
    uint32_t* d_defg_cnt_init = nullptr;   // its per-grain cell counts
    uint32_t* d_u32tmp = nullptr;
    void* d_stage = nullptr;
    size_t stage_cap = 0;
    DFront scratch{};
    uint32_t scratch_cap = 0;
    size_t scnt_words[2] = {0, 0}, csct_words = 0;  // supertile counter arrays (zeroed on reset)

    double Xcells = 0.0;
    uint32_t step = 0, defrag_cnt = 0, n_nuclei = 0;
    uint32_t next_never[2] = {0, 0}, high_water[2] = {0, 0};
    score_step_stats last{};

    Engine* eng = nullptr;             // launches this domain's steps (its own, or a batch's)
    bool own_eng = false;
    bool running = false;              // steps in the next batched step
    double weights_ms = 0.0;           // host time in requested weights (summed into the engine's timing)
    bool ans_ready = false;            // the engine computed this step's requested weights already
    std::vector<unsigned long long> ans_idx;  // weights computed for the last step's requests
    std::vector<double> ans_val;
    uint64_t launches = 0;             // kernels launched outside the step sequence
    std::vector<score_step_stats> trace;  // per-step stats of the last batched run
    // on-the-fly characterization: the grain-evolution log at the SingleGrainVolOverTime logpoints
    double t_step = 0.0;               // t at the start of the running step (the log records it)
    std::vector<double> log_cells;     // logpoint X times N: the reference's output_atthisX
    uint32_t log_next = 0;             // next logpoint
    std::vector<score_grainevo_info> log_info;
    uint32_t* d_log_counts = nullptr;  // log_cap x (ndefg + nrxg) cell counts
    uint32_t* d_log_area = nullptr;    // log_cap x 2 nz RX area profile
    uint32_t log_cap = 0;
    // P-table entries the runs since the last reset wrote (requests, nuclei): a reset clears these
    // instead of the whole table, unless the table is fresh or was loaded from the caller
    std::vector<unsigned long long> ptab_touched;
    uint32_t ntouch = 0;               // entries the device settled itself (a.touched)
    bool ptab_dirty_all = true;

    ~score_ctx() { release_domain(); release_stream(); }
    void release_domain();
    void release_stream();
    int fail(int code, const std::string& msg) { err = msg; return code; }
    int cuda_fail(cudaError_t e, const char* what) {
        err = std::string(what) + ": " + cudaGetErrorString(e);
        return SCORE_ERR_CUDA;
    }
    bool stage(size_t bytes);
    void unstage() {
        if (d_stage) cudaFree(d_stage);
        d_stage = nullptr; stage_cap = 0;
    }
};

void score_ctx::release_domain() {
    if (device >= 0) cudaSetDevice(device);
    void* ptrs[] = {a.fuse, a.touched, (void*)a.rxq, (void*)a.dfq, a.f[0].inc, a.f[1].inc, scratch.inc, a.f[0].mob, a.f[1].mob, scratch.mob, a.f[0].fill, a.f[0].comp, a.f[0].vel, a.f[0].defg, a.f[0].rxg, a.f[0].xyz, a.f[0].dir, a.f[0].full, a.f[0].recyc,
                    a.f[1].fill, a.f[1].comp, a.f[1].vel, a.f[1].defg, a.f[1].rxg, a.f[1].xyz, a.f[1].dir, a.f[1].full, a.f[1].recyc,
                    a.grid, a.claim, a.amask, a.ptab, a.defg_cnt, a.rxg_cnt, a.depleted, a.miss, a.tobm, a.ctcnt, a.fcell,
                    a.f[0].fmask, a.f[0].imask, a.f[0].tcnt, a.f[1].fmask, a.f[1].imask, a.f[1].tcnt,
                    a.f[0].scnt, a.f[1].scnt, a.csct,
                    d_state, d_pforce, d_u32tmp, d_stage, d_grid_init, d_defg_cnt_init, d_due, d_log_counts, d_log_area,
                    scratch.fill, scratch.comp, scratch.vel, scratch.defg, scratch.rxg, scratch.xyz, scratch.dir};
    for (void* p : ptrs) if (p) cudaFree(p);
    if (h_pforce) cudaFreeHost(h_pforce);
    h_pforce = nullptr;
    if (h_due) cudaFreeHost(h_due);
    h_due = nullptr; d_due = nullptr;
    a = DomainArgs{};
    scratch = DFront{};
    d_state = nullptr; d_pforce = nullptr; d_u32tmp = nullptr; d_stage = nullptr;
    d_grid_init = nullptr; d_defg_cnt_init = nullptr;
    d_log_counts = nullptr; d_log_area = nullptr; log_cap = 0;
    stage_cap = 0; scratch_cap = 0;
    loaded = false;
}


// ------------------------------------------------------------------ step engine
// Launches one growth step of every running domain of a set (one domain, or a batch of
// independent domains) as one sequence of kernels over all of them, on one stream:
// the per-domain argument blocks go to the device in one copy, the sequence runs as
// a CUDA graph (captured once per domain count and tile configuration) or as direct
// launches, and the step ends with one stream synchronization.
struct TuneCfg {
    int items = 8;          // grow tile = kBlock * items slots
    int fill_bpsm = 16;     // k_grow_fill blocks per SM
    int claim_bpsm = 4;     // k_claim blocks per SM: what fits at 64 registers
    int commit_bpsm = 8;    // k_resolve / k_commit blocks per SM (autotuner's choice on the 512^3 workload)
    int spec_pct = 30;      // every slot's data loaded with its infector byte up to this INACTIVE share [%]
    int timing_every = 8;   // phase events on every k-th step of a run (0 never): each event costs
                            // microseconds of device time, so the steps in between run without
    bool operator==(const TuneCfg& o) const {
        return items == o.items && fill_bpsm == o.fill_bpsm && claim_bpsm == o.claim_bpsm && commit_bpsm == o.commit_bpsm;
    }
};

// Slots of the constant-memory argument array c_args, per device: each engine holds a
// contiguous range for as long as it lives.
std::mutex g_slot_mu;
uint64_t g_slots_used[64] = {};

int alloc_slots(int device, int n, int* base) {
    if (device < 0 || device >= 64 || n < 1 || n > kMaxDomains) return SCORE_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_slot_mu);
    for (int b = 0; b + n <= kMaxDomains; ++b) {
        const uint64_t m = (n == 64 ? ~0ull : ((1ull << n) - 1)) << b;
        if (!(g_slots_used[device] & m)) {
            g_slots_used[device] |= m;
            *base = b;
            return SCORE_OK;
        }
    }
    return SCORE_ERR_CAPACITY;
}

void free_slots(int device, int base, int n) {
    if (base < 0 || n < 1) return;
    std::lock_guard<std::mutex> lock(g_slot_mu);
    g_slots_used[device] &= ~((n == 64 ? ~0ull : ((1ull << n) - 1)) << base);
}

// Persistent worker threads for the per-domain host work of a batched step.
// Host worker threads for the per-domain and per-grain work between GPU steps.  A step's
// host work comes in short rounds a few hundred microseconds apart, so an idle worker spins
// (yielding) for up to kSpin before it sleeps: a round then starts and ends in about a
// microsecond instead of the tens of microseconds of a condition-variable wake-up.
// Jobs are handed out as tickets (round << 32 | index): a worker still finishing an older
// round can never take, or lose, a job of a newer one.
class WorkerPool {
public:
    explicit WorkerPool(unsigned n) {
        for (unsigned i = 0; i < n; ++i) th_.emplace_back([this] { loop(); });
    }
    ~WorkerPool() {
        {
            std::lock_guard<std::mutex> l(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (auto& t : th_) t.join();
    }
    size_t size() const { return th_.size(); }
    // run f(0..n-1) on the workers and the calling thread; returns when all are done
    void run(int n, const std::function<void(int)>& f) {
        const uint64_t g = ++round_;
        ticket_.store(g << 32);  // first: tickets of the last round stop working
        job_.store(&f);
        njobs_.store((uint32_t)n);
        pending_.store(n);
        {
            std::lock_guard<std::mutex> l(mu_);
            gen_.store(g);
        }
        if (sleepers_.load() > 0) cv_.notify_all();
        work(g);
        while (pending_.load() > 0) std::this_thread::yield();
    }

private:
    static constexpr std::chrono::microseconds kSpin{2000};
    void work(uint64_t g) {
        for (;;) {
            uint64_t t = ticket_.load();
            for (;;) {
                if ((t >> 32) != g || (uint32_t)t >= njobs_.load()) return;
                if (ticket_.compare_exchange_weak(t, t + 1)) break;
            }
            (*job_.load())((int)(uint32_t)t);
            pending_.fetch_sub(1);
        }
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            const auto t0 = std::chrono::steady_clock::now();
            while (gen_.load() == seen && !stop_.load()) {
                if (std::chrono::steady_clock::now() - t0 < kSpin) {
                    std::this_thread::yield();
                    continue;
                }
                std::unique_lock<std::mutex> l(mu_);
                sleepers_.fetch_add(1);
                cv_.wait(l, [&] { return stop_.load() || gen_.load() != seen; });
                sleepers_.fetch_sub(1);
            }
            if (stop_.load()) return;
            seen = gen_.load();
            work(seen);
        }
    }
    std::vector<std::thread> th_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::atomic<const std::function<void(int)>*> job_{nullptr};
    std::atomic<uint64_t> ticket_{0}, gen_{0};
    std::atomic<uint32_t> njobs_{0};
    std::atomic<int> pending_{0}, sleepers_{0};
    std::atomic<bool> stop_{false};
    uint64_t round_ = 0;  // only the calling thread starts rounds
};

// Slots of a domain's front up to which its steps run inside one launch.  A fused step saves the separate
// kernels' fixed cost (about 50 us) but streams a large front with half their loads in flight.  Measured per run,
// limits of 2 / 4 / 8 / 14 M slots: FP64 384^3 rolled sheet 67.9 / 68.1 / 63.5 / 63.6 ms, the same with few cells in
// motion for 2,000 steps 235 / 236 / 171 / 171, FP64 512^3 104.3 / 103.7 / 103.6 / 105.9, FP32 384^3 with recovery
// 160 / 132 / 131 / 131 (211 with none).
constexpr uint64_t kFuseSlots = 8ull << 20;
// Slots a block of all the launch's domains: a batch's blocks are shared out to its domains, and beyond this the separate
// kernels, which put every SM on every domain, gain more than their launches cost.  64 domains in two groups (22 M
// slots a group on 76 blocks at the end): 284 ms a run without this limit, 249 at 193 K a block, 253 at 221 K, 261 at
// 248 K; 48 in one group (31 M slots on 152 blocks): 174 without, 185 at 166 K.
constexpr uint64_t kFuseBlockSlots = 200ull << 10;
// Slots a block from which a thread takes 4 slots a tile instead of 2: fewer, wider accesses (16-domain batch: fill
// 42 us a step with 2, 23 with 4), but half the tiles to spread over the blocks.
constexpr uint64_t kFuseWide = 4096;

// A launch's turn, after which its groups leave so that other work of the device gets its own.
constexpr int64_t kFuseTurnUs = 2000;

// The limits of an engine's fused steps and staging.  Results do not depend on them: tests lower them, so that small domains
// take every path (score_internal_step_limits), never raise them.
struct StepLimits {
    uint32_t host_polls = kFuseHostSpin, group_polls = kFuseSpin;
    uint32_t wide = (uint32_t)kFuseWide, block_slots = (uint32_t)kFuseBlockSlots;
    uint64_t slots = kFuseSlots;
    uint32_t number = 0;               // of the next command (1 to kCmdSeqMask; 0: as it is)
    uint32_t refuse_after = ~0u;       // cooperative launches until one is answered as refused (~0: never)
    uint64_t stage = ~0ull;            // bytes beyond which a staging buffer is refused
};

struct Engine {
    int device = 0, sms = 1;
    cudaStream_t stream = nullptr;
    bool fp32 = false;
    std::vector<score_ctx*> dom;
    int base = -1, nslots = 0;         // this engine's slots of c_args
    DomainArgs* d_args = nullptr;      // device address of c_args[base]
    DomainArgs* h_args = nullptr;      // pinned staging of the argument blocks
    std::vector<DomainArgs> h_args_dev;  // what the device's slots hold
    bool args_dirty = true;
    TuneCfg cfg;
    bool use_graph = true;
    bool capturing = false;
    bool events = false;               // the sequence being launched records the phase events
    int fill_mode = kFillAny;          // ... and the grow mode of every stepping domain (kFillAny: per domain)
    // the step without / with phase events, with the general / the refresh-only grow kernel
    // the step graphs: with or without phase events, times the fill mode (0..4, 5 for a batch of
    // cached increments, or per domain)
    static constexpr int kGraphs = 14;
    cudaGraphExec_t gexec[kGraphs] = {};
    TuneCfg gcfg[kGraphs];
    int gndom[kGraphs] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    bool gfp32[kGraphs] = {};
    uint64_t run_steps = 0;            // steps since the run started (phase sampling)
    // 0 start, 1 end of fill, 2 end of lists, 3 end of claim, 4 end of step, 5/6 run span
    cudaEvent_t ev[7] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    score_timing tm{};
    uint64_t launches = 0;
    std::string err;
    std::unique_ptr<WorkerPool> pool;  // batches of several domains
    unsigned pool_threads = 0;         // workers of the pool (0: the caller's default)
    WorkerPool& workers(unsigned dflt) {
        if (!pool) pool.reset(new WorkerPool(std::max(1u, pool_threads ? pool_threads : std::min(dflt, std::thread::hardware_concurrency() - 1))));
        return *pool;
    }
    // the host's weights for all domains' requests, in pinned device-mapped memory: the
    // few cells that wait for them read them directly (no copy before the step)
    unsigned long long* h_ans_i = nullptr; double* h_ans_v = nullptr;
    unsigned long long* d_ans_i = nullptr; double* d_ans_v = nullptr;
    size_t ans_cap = 0, ans_total = 0;
    int stage_answers();

    ~Engine() { release(); }
    int init(int dev, int ndom) {
        device = dev;
        int s = alloc_slots(dev, ndom, &base);
        if (s != SCORE_OK) return s;
        nslots = ndom;
        cudaError_t e = cudaSetDevice(dev);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        for (auto& x : ev) if (e == cudaSuccess) e = cudaEventCreate(&x);
        void* sym = nullptr;
        if (e == cudaSuccess) e = cudaGetSymbolAddress(&sym, c_args);
        if (e == cudaSuccess) d_args = (DomainArgs*)sym + base;
        if (e == cudaSuccess) e = cudaMallocHost((void**)&h_args, (size_t)ndom * sizeof(DomainArgs));
        h_args_dev.assign((size_t)ndom, DomainArgs{});
        args_dirty = true;
        int coop = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        for (const void* k : {(const void*)k_steps_fused<false, 2>, (const void*)k_steps_fused<true, 2>, (const void*)k_steps_fused<false, 4>,
                              (const void*)k_steps_fused<true, 4>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(FuseShared));
        fuse = e == cudaSuccess && coop != 0;
        fuse_sms = sms;
        return e == cudaSuccess ? SCORE_OK : SCORE_ERR_CUDA;
    }
    void drop_graph() {
        for (int k = 0; k < kGraphs; ++k) {
            if (gexec[k]) cudaGraphExecDestroy(gexec[k]);
            gexec[k] = nullptr;
            gndom[k] = -1;
        }
    }
    void release() {
        cudaSetDevice(device);
        drop_graph();
        if (h_ans_i) cudaFreeHost(h_ans_i);
        if (h_ans_v) cudaFreeHost(h_ans_v);
        h_ans_i = nullptr; h_ans_v = nullptr; d_ans_i = nullptr; d_ans_v = nullptr;
        ans_cap = ans_total = 0;
        if (h_args) cudaFreeHost(h_args);
        d_args = nullptr; h_args = nullptr;
        free_slots(device, base, nslots);
        base = -1; nslots = 0;
        for (auto& x : ev) if (x) { cudaEventDestroy(x); x = nullptr; }
        if (stream) cudaStreamDestroy(stream);
        stream = nullptr;
    }
    int fail(int code, const std::string& m) { err = m; return code; }
    void launch_sequence(int n);
    cudaError_t enqueue_step(int n, bool timed, int mode);
    int step(bool timed);
    bool fused_ok() const;
    int fused_session(double x_target, uint32_t max_steps, bool one, std::vector<uint32_t>& done);
    void balance_weights();
    int run_until(double x_target, uint32_t max_steps, uint32_t* steps_done);
    int autotune(double x_target, uint32_t max_steps, score_tune* out);
    void get_tune(score_tune* out) const;
    int set_tune(const score_tune* t);
    void mark_run_start() { cudaEventRecord(ev[5], stream); run_steps = 0; }
    StepLimits lim;
    bool fuse = false;                 // cooperative launches of k_steps_fused are possible
    int fuse_sms = 1;                  // blocks of one of them (batches share the SMs between their engines)
    bool sample_step() const { return cfg.timing_every > 0 && run_steps % (uint64_t)cfg.timing_every == 0; }
    int mark_run_end();
};

namespace {
template <class Body>
void for_grains(score_ctx* c, Body body) {
    const size_t n = c->ndefg;
    Engine& E = *c->eng;
    if (n < 8192 || E.dom.size() != 1) { body(0, n); return; }
    E.workers(15);
    constexpr int kChunks = 16;
    E.pool->run(kChunks, [&](int k) { body(n * (size_t)k / kChunks, n * (size_t)(k + 1) / kChunks); });
}
}  // namespace

bool score_ctx::stage(size_t bytes) {
    if (bytes <= stage_cap) return true;
    if (bytes > eng->lim.stage) return false;
    unstage();
    if (cudaMalloc(&d_stage, bytes) != cudaSuccess) {
        cudaGetLastError();  // the caller may go on without
        d_stage = nullptr;
        return false;
    }
    stage_cap = bytes;
    return true;
}

// (after Engine is complete: deleting it runs its destructor, which returns its
// argument slots, stream, events and pinned buffers)
void score_ctx::release_stream() {
    if (device >= 0) cudaSetDevice(device);
    if (h_state) cudaFreeHost(h_state);
    h_state = nullptr;
    if (h_box) cudaFreeHost(h_box);
    h_box = nullptr; d_box = nullptr;
    if (own_eng) delete eng;
    eng = nullptr;
    stream = nullptr;  // owned by the engine
}

// ------------------------------------------------------------------ helpers
namespace {

// Per-grain host loop over [0, ndefg): split over the engine's worker threads for a
// single domain with many grains (a batch already runs its domains in parallel).
template <class Body>
void for_grains(score_ctx* c, Body body);

// newest driving forces to the device, in stream order
int flush_pforce(score_ctx* c) {
    if (!c->pf_pending) return SCORE_OK;
    const cudaError_t e = cudaMemcpyAsync(c->d_pforce, c->h_pforce + (size_t)c->pf_buf * c->ndefg, (size_t)c->ndefg * 8,
                                          cudaMemcpyHostToDevice, c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "upload driving force");
    c->pf_pending = false;
    return SCORE_OK;
}

// Driving force per deformed grain, the grow step's p (SCORE_Kernel.cpp:4082), from `rho`
// (whose version is `rho_ver`).  When it or the mobilities change, the front's velocity
// factors are recomputed in the next grow.  The copy is stream-ordered after every launch
// already enqueued, so a step in flight still reads the previous values.
int upload_physics(score_ctx* c, const double* rho, uint64_t rho_ver) {
    const double mob[4] = {c->ph.mLAGB, c->ph.mHAGB, c->ph.mGS, c->ph.mRHHAGB};
    const bool mob_same = memcmp(mob, c->mob_host, sizeof mob) == 0;
    // p depends on Gb^2/2, the drag and rho only: skip the per-grain pass when none changed
    const double sig[2] = {c->ph.Gbhalfsq, c->ph.zener()};
    if (mob_same && !c->pforce_host.empty() && memcmp(sig, c->pf_sig, sizeof sig) == 0 && c->pf_rho_version == rho_ver)
        return SCORE_OK;
    memcpy(c->pf_sig, sig, sizeof sig);
    c->pf_rho_version = rho_ver;
    // new p per grain, straight into the pinned staging buffer that the device does not read (the last
    // copy out of it finished before the step that just ended), noting whether any value changed
    double* const h_new = c->h_pforce + (size_t)(c->pf_buf ^ 1) * c->ndefg;
    if (c->pforce_host.size() != c->ndefg) c->pforce_host.assign(c->ndefg, std::numeric_limits<double>::quiet_NaN());
    std::atomic<bool> pf_changed{false};
    for_grains(c, [&](size_t lo, size_t hi) {
        bool ch = false;
        for (size_t g = lo; g < hi; ++g) {
            const double v = c->ph.driving_force(rho[g]);
            h_new[g] = v;
            if (v != c->pforce_host[g]) { c->pforce_host[g] = v; ch = true; }
        }
        if (ch) pf_changed.store(true);
    });
    if (!pf_changed.load() && mob_same) return SCORE_OK;
    c->refresh = (c->refresh == 1 || !mob_same) ? 1 : 2;  // new mobilities need P again
    memcpy(c->mob_host, mob, sizeof mob);
    if (!pf_changed.load()) return SCORE_OK;
    c->pf_buf ^= 1;
    c->pf_pending = true;
    return c->fuse_live ? SCORE_OK : flush_pforce(c);
}

void set_step_args(score_ctx* c) {
    c->a.mLAGB = c->ph.mLAGB; c->a.mHAGB = c->ph.mHAGB; c->a.mGS = c->ph.mGS; c->a.mRH = c->ph.mRHHAGB;
    c->a.dt = c->ph.dt; c->a.cinv = (1.0 / c->prm.cellsize);
    c->a.dtc32 = (float)(c->ph.dt * (1.0 / c->prm.cellsize));
}

double weight_of(score_ctx* c, uint32_t r, uint32_t g) {
    if (!c->user_ptab.empty()) return c->user_ptab[(size_t)r * c->ndefg + g];
    return mobility_weight(c->prm, &c->rxg_q[4 * (size_t)r], &c->defg_q[4 * (size_t)g]);
}

// thresholds of the FP32 classification (weight_class)
WeightClass make_weight_class(const score_params& p) {
    double fac = 0, lagb = 0, maxdev = 0, m40[4], sat = 0;
    weight_constants(p, &fac, &lagb, &maxdev, m40, &sat);
    WeightClass w{};
    w.model = p.mobility_model;
    const double deg40 = 2.0 * kPi / 9.0;
    w.cos_lagb = (float)std::cos(0.5 * lagb);
    w.cos_lo = (float)std::cos(0.5 * (deg40 - maxdev));
    w.cos_hi = (float)std::cos(0.5 * (deg40 + maxdev));
    w.cos_dev = (float)std::cos(0.5 * maxdev);
    w.cos_sat = sat < kPi ? (float)std::cos(0.5 * sat) : -2.0f;
    for (int i = 0; i < 4; ++i) w.m40[i] = (float)m40[i];
    return w;
}

// compute P for a list of table indices on the host, in parallel for large batches
// (`alone`: no other domain of a batch uses the engine's workers meanwhile)
void resolve_weights(score_ctx* c, const std::vector<unsigned long long>& idx, std::vector<double>& val, bool alone = false) {
    val.resize(idx.size());
    auto work = [&](size_t lo, size_t hi) {
        for (size_t i = lo; i < hi; ++i)  // a void slot (lost race) keeps 0, which no cell reads
            val[i] = idx[i] == kMissVoid ? 0.0 : weight_of(c, (uint32_t)(idx[i] / c->ndefg), (uint32_t)(idx[i] % c->ndefg));
    };
    size_t n = idx.size();
    Engine& E = *c->eng;
    if (n >= (alone ? 256u : 16u) && (alone || E.dom.size() == 1)) {  // one domain: the engine's workers (a batch runs its domains in parallel)
        E.workers(15);
        const int chunks = (int)std::min<size_t>(64, n / 8);
        E.pool->run(chunks, [&](int k) { work(n * (size_t)k / chunks, n * (size_t)(k + 1) / chunks); });
        return;
    }
    // a batch computes its domains' weights on the engine's workers already: no nested threads
    unsigned nth = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
    if (n < 4096 || nth == 1 || E.dom.size() > 1) { work(0, n); return; }
    std::vector<std::thread> th;
    for (unsigned t = 0; t < nth; ++t) th.emplace_back(work, n * t / nth, n * (t + 1) / nth);
    for (auto& t : th) t.join();
}

int check_device_errors(score_ctx* c, uint32_t flags) {
    if (!flags) return SCORE_OK;
    if (flags & kErrTimeout)
        return c->fail(SCORE_ERR_TIMEOUT, "a bounded device wait gave up (at " + std::to_string(c->h_box->snap.err_info >> 28) + ", block " +
                                              std::to_string((c->h_box->snap.err_info >> 16) & 0xFFFu) + ")");
    if (flags & kErrKeyLimit) return c->fail(SCORE_ERR_KEYLIMIT, "more than 2^32-1 infection attempts in one step");
    if (flags & kErrBorderRef) return c->fail(SCORE_ERR_BORDER_CAPACITY, "Border list exceeded 2(xy+xz+yz) slots (the reference writes out of bounds here)");
    if (flags & kErrCapacity) return c->fail(SCORE_ERR_CAPACITY, "front list capacity exceeded");
    if (flags & kErrMissCap) return c->fail(SCORE_ERR_CAPACITY, "mobility-weight request list capacity exceeded");
    return c->fail(SCORE_ERR_STATE, "device bounds check failed (corrupt domain?)");
}

// site-saturated placement of nuclei with tincub <= t, rxg order
// (ompshar_sim_myCA_sitesaturatedNucleation / infect_JuvenileNucleation, SCORE_GrowthMachine.cpp:50-189)
// With `on_device`, up to kDueMax candidates are placed by k_place_due in stream order
// before the step (no host round trip); the placed count, the slots and the P max reach
// the host in the step's mailbox.  Otherwise the host reads the site values, decides and
// uploads the nuclei (two synchronizations).
int place_nuclei_upto(score_ctx* c, double tnow, uint32_t* nplaced, bool on_device) {
    std::vector<uint32_t> cand;
    while (c->nuc_pos < c->nuc_order.size() && c->tincub[c->nuc_order[c->nuc_pos]] <= tnow) cand.push_back(c->nuc_order[c->nuc_pos++]);
    std::sort(cand.begin(), cand.end());  // the reference places nuclei in rxg order
    if (nplaced) *nplaced = 0;
    if (cand.empty()) return SCORE_OK;
    const uint32_t n = (uint32_t)cand.size();
    if (on_device && n <= kDueMax) {
        const uint32_t nx = c->nx, ny = c->ny, nxy = nx * ny;
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t r = cand[i], s = c->site[r], g = c->site_defg[r];
            const uint32_t z = s / nxy, y = (s - z * nxy) / nx, x = s - z * nxy - y * nx;
            const bool inside = x > 0 && x < nx - 1 && y > 0 && y < ny - 1 && z > 0 && z < c->nz - 1;
            c->placed[r] = 1;
            c->h_due[i] = NucDue{c->gsite[r], r, g, inside ? 0u : 1u, weight_of(c, r, g)};
            c->ptab_touched.push_back((unsigned long long)r * c->ndefg + g);
        }
        const cudaError_t e = cudaMemcpyAsync(c->d_due, c->h_due, (size_t)n * sizeof(NucDue), cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return c->cuda_fail(e, "upload due nuclei");
        set_step_args(c);
        if (c->fp32) k_place_due<true><<<1, kDueMax, 0, c->stream>>>(c->a, c->d_due, n);
        else k_place_due<false><<<1, kDueMax, 0, c->stream>>>(c->a, c->d_due, n);
        c->launches++;
        return SCORE_OK;
    }
    std::vector<uint32_t> sites(n), gsites(n), gval(n);
    for (uint32_t i = 0; i < n; ++i) { sites[i] = c->site[cand[i]]; gsites[i] = c->gsite[cand[i]]; }
    if (!c->stage((size_t)n * 8)) return c->fail(SCORE_ERR_NOMEM, "staging buffer");
    uint32_t* d_idx = (uint32_t*)c->d_stage;
    uint32_t* d_out = d_idx + n;
    cudaError_t e = cudaMemcpyAsync(d_idx, gsites.data(), (size_t)n * 4, cudaMemcpyHostToDevice, c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "upload nucleus sites");
    k_gather_u32<<<blocks_for(n, c->sms), kBlock, 0, c->stream>>>(c->a.grid, d_idx, n, d_out);
    c->launches++;
    e = cudaMemcpyAsync(gval.data(), d_out, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "gather nucleus sites");

    std::vector<NucRec> recs;
    // sites taken by earlier nuclei, open addressing (N < 2^31: no site is ~0)
    uint32_t slots = 64;
    while (slots < 2 * n) slots *= 2;
    std::vector<uint32_t> taken(slots, 0xFFFFFFFFu);
    auto at = [&](uint32_t site) {
        uint32_t h = (site * 2654435769u) & (slots - 1);
        while (taken[h] != 0xFFFFFFFFu && taken[h] != site) h = (h + 1) & (slots - 1);
        return h;
    };
    std::vector<unsigned long long> pidx;
    std::vector<double> pval;
    const uint32_t nx = c->nx, ny = c->ny, nxy = nx * ny;
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t r = cand[i];
        c->placed[r] = 1;
        uint32_t g = gval[i];
        const uint32_t h = at(sites[i]);
        if (taken[h] == sites[i]) g = kCurrentlyInfected;
        if (g >= c->ndefg) continue;  // site already infected or recrystallized: nucleus not placeable
        const uint32_t s = sites[i];
        const uint32_t z = s / nxy, y = (s - z * nxy) / nx, x = s - z * nxy - y * nx;
        const bool inside = x > 0 && x < nx - 1 && y > 0 && y < ny - 1 && z > 0 && z < c->nz - 1;
        const int L = inside ? 0 : 1;
        const uint32_t slot = c->next_never[L];
        if (slot >= c->a.f[L].cap) return c->fail(SCORE_ERR_CAPACITY, "front list capacity exceeded while placing nuclei");
        if (L == 1 && c->prm.border_policy == SCORE_BORDER_REFERENCE_LIMIT && slot >= c->a.border_ref_cap)
            return c->fail(SCORE_ERR_BORDER_CAPACITY, "Border list exceeded 2(xy+xz+yz) slots while placing nuclei");
        c->next_never[L]++;
        NucRec q{};
        q.list = (uint32_t)L; q.slot = slot; q.site = gsites[i]; q.rxg = r; q.defg = g;
        recs.push_back(q);
        taken[h] = s;
        pidx.push_back((unsigned long long)r * c->ndefg + g);
        c->ptab_touched.push_back(pidx.back());
        c->n_nuclei++;
        if (nplaced) (*nplaced)++;
    }
    if (recs.empty()) return SCORE_OK;
    // the weights on the workers (50,000 nuclei: 14.4 ms with one weight after another and a node-based set of
    // sites, 3.1 now)
    resolve_weights(c, pidx, pval, true);
    for (size_t i = 0; i < recs.size(); ++i) {
        recs[i].P = pval[i];
        if (pval[i] >= c->ph.Pmax) c->ph.Pmax = pval[i];  // reg_myMobilityWeightMax, then the master's max
    }
    const size_t nr = recs.size();
    const size_t bytes = nr * sizeof(NucRec) + nr * 16;
    if (!c->stage(bytes)) return c->fail(SCORE_ERR_NOMEM, "staging buffer");
    NucRec* d_rec = (NucRec*)c->d_stage;
    unsigned long long* d_pi = (unsigned long long*)(d_rec + nr);
    double* d_pv = (double*)(d_pi + nr);
    e = cudaMemcpyAsync(d_rec, recs.data(), nr * sizeof(NucRec), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_pi, pidx.data(), nr * 8, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_pv, pval.data(), nr * 8, cudaMemcpyHostToDevice, c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "upload nuclei");
    set_step_args(c);
    if (c->fp32) k_place_nuclei<true><<<blocks_for(nr, c->sms), kBlock, 0, c->stream>>>(c->a, d_rec, (uint32_t)nr);
    else k_place_nuclei<false><<<blocks_for(nr, c->sms), kBlock, 0, c->stream>>>(c->a, d_rec, (uint32_t)nr);
    k_fill_ptab<<<blocks_for(nr, c->sms), kBlock, 0, c->stream>>>(c->a.ptab, d_pi, d_pv, (uint32_t)nr);
    c->launches += 2;
    e = cudaMemcpyAsync((char*)c->d_state + offsetof(DevState, next_never), c->next_never, 8, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "place nuclei");
    for (int L = 0; L < 2; ++L) c->high_water[L] = std::max(c->high_water[L], c->next_never[L]);
    return SCORE_OK;
}

// ompshar_defragmentation, SCORE_Kernel.cpp:3877-3937, for one list
int defragment(score_ctx* c, int L) {
    const uint32_t n = c->next_never[L];
    if (n == 0) return SCORE_OK;
    DFront& fr = c->a.f[L];
    if (c->scratch_cap < n) {
        void* ptrs[] = {c->scratch.inc, c->scratch.mob, c->scratch.fill, c->scratch.comp, c->scratch.vel, c->scratch.defg, c->scratch.rxg, c->scratch.xyz, c->scratch.dir};
        for (void* p : ptrs) if (p) cudaFree(p);
        c->scratch = DFront{};
        const size_t fb = c->fp32 ? 4 : 8;
        cudaError_t e = cudaMalloc(&c->scratch.fill, (size_t)n * fb);
        if (e == cudaSuccess && c->fp32) e = cudaMalloc((void**)&c->scratch.comp, (size_t)n * 4);
        if (e == cudaSuccess) e = cudaMalloc(&c->scratch.vel, (size_t)n * fb);
        if (e == cudaSuccess && !c->fp32) e = dalloc(&c->scratch.inc, n);
        if (e == cudaSuccess) e = dalloc(&c->scratch.mob, n);
        if (e == cudaSuccess) e = dalloc(&c->scratch.defg, n);
        if (e == cudaSuccess) e = dalloc(&c->scratch.rxg, n);
        if (e == cudaSuccess) e = dalloc(&c->scratch.xyz, n);
        if (e == cudaSuccess) e = dalloc(&c->scratch.dir, n);
        if (e != cudaSuccess) return c->fail(SCORE_ERR_NOMEM, "defragmentation scratch");
        c->scratch_cap = n;
    }
    uint32_t* d_cnt = c->d_u32tmp;
    const uint32_t ntiles = (n + kGrowTile - 1) / kGrowTile;
    const uint32_t grid = std::min<uint32_t>(ntiles, (uint32_t)c->sms * 8);
    k_defrag_count<<<grid, kBlock, 0, c->stream>>>(c->a, L, n);
    k_scan_defrag<<<1, 1024, 0, c->stream>>>(c->a, L, n, d_cnt);
    if (c->fp32) k_defrag_compact<true><<<grid, kBlock, 0, c->stream>>>(c->a, L, n, c->scratch);
    else k_defrag_compact<false><<<grid, kBlock, 0, c->stream>>>(c->a, L, n, c->scratch);
    c->launches += 3;
    uint32_t active = 0;
    cudaError_t e = cudaMemcpyAsync(&active, d_cnt, 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "defragment");
    if (active == n) {
        // no INACTIVE slot below next_never: the reference's scan for the first INACTIVE
        // continues into slots left behind by earlier compactions
        uint32_t first = c->high_water[L];
        if (c->high_water[L] > n) {
            e = cudaMemcpyAsync(d_cnt, &first, 4, cudaMemcpyHostToDevice, c->stream);
            k_first_inactive<<<blocks_for(c->high_water[L] - n, c->sms), kBlock, 0, c->stream>>>(fr.dir, n, c->high_water[L], d_cnt);
            c->launches++;
            if (e == cudaSuccess) e = cudaMemcpyAsync(&first, d_cnt, 4, cudaMemcpyDeviceToHost, c->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
            if (e != cudaSuccess) return c->cuda_fail(e, "defragment");
        }
        c->next_never[L] = std::max(n, first);
    } else {
        const size_t fb = c->fp32 ? 4 : 8;
        e = cudaMemcpyAsync(fr.fill, c->scratch.fill, (size_t)active * fb, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess && c->fp32) e = cudaMemcpyAsync(fr.comp, c->scratch.comp, (size_t)active * 4, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.vel, c->scratch.vel, (size_t)active * fb, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess && !c->fp32) e = cudaMemcpyAsync(fr.inc, c->scratch.inc, (size_t)active * 8, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.mob, c->scratch.mob, (size_t)active * 8, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.defg, c->scratch.defg, (size_t)active * 4, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.rxg, c->scratch.rxg, (size_t)active * 4, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.xyz, c->scratch.xyz, (size_t)active * 4, cudaMemcpyDeviceToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(fr.dir, c->scratch.dir, (size_t)active, cudaMemcpyDeviceToDevice, c->stream);
        if (e != cudaSuccess) return c->cuda_fail(e, "defragment copy");
        c->next_never[L] = active;
    }
    e = cudaMemcpyAsync((char*)c->d_state + offsetof(DevState, next_never), c->next_never, 8, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "defragment");
    return SCORE_OK;
}

// Return the domain to its loaded state on the device (grid from the pristine copy,
// empty fronts, empty P cache) and redo the start of solve_RXGROWTH
// (SCORE_Kernel.cpp:6513-6530): rho max, T, G/b, mobilities, dt0.
int reset_state(score_ctx* c) {
    DomainArgs& a = c->a;
    const uint64_t W = c->ncells;
    cudaStream_t st = c->stream;
    cudaError_t e = cudaMemcpyAsync(a.grid, c->d_grid_init, W * 4, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.claim, 0xFF, W * 4, st);
    for (int L = 0; L < 2 && e == cudaSuccess; ++L) {
        e = cudaMemsetAsync(a.f[L].dir, kInactive, std::max<size_t>(c->high_water[L], 1), st);
    }
    if (e == cudaSuccess && c->user_ptab.empty()) {
        // every entry unknown again: the whole table after allocation or a caller's table, else only the
        // entries the last runs wrote (a 512^3 run writes about 0.03 % of its 8 GB table)
        const size_t total = std::max<size_t>((size_t)c->nrxg * c->ndefg, 1);
        const size_t nt = c->ptab_touched.size();
        if (c->failed || c->ntouch > a.touchcap) c->ptab_dirty_all = true;  // a step that failed may have tagged entries it never reported
        if (c->ptab_dirty_all || nt + c->ntouch > total / 64 || !c->stage(nt * 8)) {
            e = cudaMemsetAsync(a.ptab, 0xFF, total * 8, st);
        } else {
            if (c->ntouch) {
                k_clear_ptab<<<blocks_for(c->ntouch, c->sms), kBlock, 0, st>>>(a.ptab, a.touched, c->ntouch);
                c->launches++;
                e = cudaGetLastError();
            }
            if (e == cudaSuccess && nt) e = cudaMemcpyAsync(c->d_stage, c->ptab_touched.data(), nt * 8, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess && nt) {
                k_clear_ptab<<<blocks_for(nt, c->sms), kBlock, 0, st>>>(a.ptab, (const unsigned long long*)c->d_stage, (uint32_t)nt);
                c->launches++;
                e = cudaGetLastError();
            }
        }
        c->ptab_touched.clear();
        c->ntouch = 0;
        c->ptab_dirty_all = false;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(a.defg_cnt, c->d_defg_cnt_init, (size_t)c->ndefg * 4, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.rxg_cnt, 0, std::max<size_t>(c->nrxg, 1) * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_state, 0, sizeof(DevState), st);
    // a group whose wait gave up leaves its arrivals and its last word: the next launch's barriers would open early
    if (e == cudaSuccess) e = cudaMemsetAsync(a.fuse, 0, sizeof(FuseDom), st);
    for (int L = 0; L < 2 && e == cudaSuccess; ++L) e = cudaMemsetAsync(a.f[L].scnt, 0, c->scnt_words[L] * 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.csct, 0, c->csct_words * 4, st);
    if (e != cudaSuccess) return c->cuda_fail(e, "reset domain");
    c->ans_idx.clear();
    c->ans_val.clear();
    c->log_info.clear();
    c->log_next = 0;
    c->log_cells.resize(std::min<uint32_t>(c->prm.n_logpoints, c->log_cap));
    for (size_t k = 0; k < c->log_cells.size(); ++k) c->log_cells[k] = c->prm.logpoint_x[k] * (double)c->N;  // log_initialization, :60-62
    memset(&c->h_box->snap, 0, sizeof(DevState));
    c->running = false;
    c->fuse_live = false;
    c->fuse_seq = fuse_next(c->fuse_seq);
    c->pre_done = false;
    c->fuse_replay = 0;
    c->pf_pending = false;
    c->trace.clear();
    c->rho = c->rho0;
    c->defg_cnt_host = c->defg_cnt_init_host;
    c->placed.assign(c->nrxg, 0);
    c->nuc_pos = 0;
    Physics& ph = c->ph;
    ph.init(&c->prm);
    ph.rhomax = rhomax_of(c->rho, c->defg_cnt_host);
    c->rho_version = 0; c->rhomax_version = 0; c->pf_rho_version = ~0ull;
    c->rho_cursor = 0;
    ph.update_temperature();
    ph.update_atomistic();
    ph.update_mobilities();
    ph.dt = ph.dt_minimum();
    c->pforce_host.clear();
    memset(c->mob_host, 0, sizeof c->mob_host);
    c->ahead = false;
    int s = upload_physics(c, c->rho.data(), c->rho_version);
    if (s != SCORE_OK) return s;
    // the staging buffer is rewritten while the first step runs: its copy must be done
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return c->cuda_fail(e, "reset domain");
    c->refresh = 0;  // the front is empty; new cells get their factors when they are created
    c->dt_cached = -1.0;
    c->Xcells = 0.0; c->step = 0; c->defrag_cnt = 0; c->n_nuclei = 0;
    c->next_never[0] = c->next_never[1] = 0;
    c->high_water[0] = c->high_water[1] = 0;
    c->eng->tm = score_timing{};
    c->eng->mark_run_start();
    c->last = score_step_stats{};
    c->last.dt = ph.dt;
    c->last.rhomax = ph.rhomax;
    c->failed = false;
    c->loaded = true;
    return SCORE_OK;
}

}  // namespace

// ------------------------------------------------------------------ step of one domain, host side
namespace {

// Before the launch: time-dependent nucleation, defragmentation at X logpoints and the
// argument block of this step.
int pre_step(score_ctx* c, uint32_t* newnuc) {
    Physics& ph = c->ph;
    c->t_step = ph.t;
    // on-the-fly defragmentation at user X logpoints (SCORE_Kernel.cpp:6625-6630, thresholds in cells)
    const bool defrag = c->prm.defragmentation && c->defrag_cnt < c->prm.n_defrag && c->Xcells >= c->prm.defrag_x[c->defrag_cnt] * (double)c->N;
    // time-dependent nucleation (no-op when site-saturated); on the device unless the host
    // defragments this step (it needs the slot counts on the host)
    int s = place_nuclei_upto(c, ph.t, newnuc, !defrag);
    if (s != SCORE_OK) return s;
    if (defrag) {
        for (int L = 0; L < 2; ++L) { s = defragment(c, L); if (s != SCORE_OK) return s; }
        c->defrag_cnt++;
    }
    set_step_args(c);
    DomainArgs& a = c->a;
    a.dt_changed = (ph.dt != c->dt_cached) ? 1 : 0;
    a.refresh = c->refresh;
    // load strategy of k_grow_fill from the INACTIVE share of the last step's scanned slots
    const uint64_t scanned = (uint64_t)c->last.next_never[0] + c->last.next_never[1];
    a.spec = 100 * (scanned - std::min<uint64_t>(c->last.Sv, scanned)) <= (uint64_t)c->eng->cfg.spec_pct * scanned ? 1 : 0;
    a.active = 1;
    c->dt_cached = ph.dt;
    c->refresh = 0;
    return SCORE_OK;
}

bool recovering(const score_ctx* c) {
    return c->prm.recovery_model != SCORE_RECOVERY_NONE && c->prm.recovery_model != SCORE_RECOVERY_NES_SOLUTEDRAG;
}

// The part of the master block of solve_RXGROWTH (SCORE_Kernel.cpp:6691-6740) that does not
// depend on the step's outcome, run while the step is on the GPU: t + dt, temperature, G and
// b, drag, mobilities, the recovered rho (into rho_next: the rho max of the step still needs
// the current values) and the next step's driving forces.  The rest (P max, X, rho max, dt)
// follows in post_step, in the reference's order; none of it feeds back into this part.
int physics_ahead(score_ctx* c) {
    Physics& ph = c->ph;
    ph.t += ph.dt;
    ph.update_temperature();
    ph.update_atomistic();
    ph.update_microchemistry();
    ph.update_mobilities();
    c->ahead = true;
    if (!recovering(c)) return upload_physics(c, c->rho.data(), c->rho_version);
    c->rho_next.resize(c->ndefg);
    for_grains(c, [&](size_t lo, size_t hi) { ph.update_substructure(c->rho_next.data(), c->rho.data(), c->rho0.data(), lo, hi); });
    return upload_physics(c, c->rho_next.data(), c->rho_version + 1);
}

// log_OUTPUT_Diehl's grain-evolution branch (SCORE_OnTheFlyCharacterization.cpp:646-650), stream-ordered
// before the next step: every grain's cell count (log_grainevo, :478-531) and the RX area profile of
// the clarified labels (log_rxareaprofile(threshold), :274-384), on the device; the host keeps the
// snapshot's time (before t += dt), X, step and 32-bit Sv.
int log_snapshot(score_ctx* c, uint64_t Sv) {
    const uint32_t k = (uint32_t)c->log_info.size();
    if (k >= c->log_cap) return c->fail(SCORE_ERR_CAPACITY, "grain-evolution log full");
    cudaStream_t st = c->stream;
    DomainArgs& a = c->a;
    const size_t G = (size_t)c->ndefg + c->nrxg;
    uint32_t* cnt = c->d_log_counts + (size_t)k * G;
    cudaError_t e = cudaMemcpyAsync(cnt, a.defg_cnt, (size_t)c->ndefg * 4, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess && c->nrxg) e = cudaMemcpyAsync(cnt + c->ndefg, a.rxg_cnt, (size_t)c->nrxg * 4, cudaMemcpyDeviceToDevice, st);
    // labels by the clarify rule into the attempt-mask array (free between steps)
    uint32_t* lab = a.amask;
    if (e == cudaSuccess) {
        k_unbrick<<<blocks_for(c->ncells, c->sms, 16), kBlock, 0, st>>>(a, a.grid, lab);
        c->launches++;
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return c->cuda_fail(e, "grain-evolution log");
    for (int L = 0; L < 2; ++L) {
        const uint32_t n = c->next_never[L];
        if (n == 0) continue;
        if (c->fp32) k_labels_front<true><<<blocks_for(n, c->sms), kBlock, 0, st>>>(a, L, n, lab);
        else k_labels_front<false><<<blocks_for(n, c->sms), kBlock, 0, st>>>(a, L, n, lab);
        c->launches++;
    }
    // per-slice sections of the rx grains, in chunks of slices whose histogram fits the win-mask array
    uint32_t* out = c->d_log_area + (size_t)k * 2 * c->nz;
    const uint32_t nxy = c->nx * c->ny, nr = std::max<uint32_t>(c->nrxg, 1);
    const uint32_t K = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(c->nz, c->N / nr));
    e = cudaMemsetAsync(a.tobm, 0, (size_t)K * nr * 4, st);
    if (e != cudaSuccess) return c->cuda_fail(e, "RX area profile");
    for (uint32_t z0 = 0; z0 < c->nz; z0 += K) {
        const uint32_t z1 = std::min(c->nz, z0 + K);
        k_area_hist<<<blocks_for((uint64_t)(z1 - z0) * nxy, c->sms, 16), kBlock, 0, st>>>(lab, nxy, z0, z1, c->ndefg, c->nrxg, a.tobm);
        k_area_sum<<<z1 - z0, kBlock, 0, st>>>(a.tobm, c->nrxg, nxy, c->prm.rxarea_threshold, out + 2 * (size_t)z0);
        c->launches += 2;
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return c->cuda_fail(e, "RX area profile");
    score_grainevo_info info{};
    info.t = c->t_step;
    info.X = c->Xcells / (double)c->N;
    info.step = c->step;
    info.Sv = (uint32_t)Sv;
    c->log_info.push_back(info);
    return SCORE_OK;
}

// After the step: the mailbox (scalars, weight requests, depleted grains), the host's
// weights for the requests (applied at the start of the next step), and the rest of the
// master block of solve_RXGROWTH (SCORE_Kernel.cpp:6691-6740).
int post_step(score_ctx* c, uint32_t newnuc, score_step_stats* out) {
    Physics& ph = c->ph;
    DomainArgs& a = c->a;
    cudaStream_t st = c->stream;
    const DevState hs = c->h_box->snap;
    if (hs.err) { c->failed = true; return check_device_errors(c, hs.err); }
    const uint64_t Sv = hs.sv[0] + hs.sv[1], nfull = (uint64_t)hs.nfull[0] + hs.nfull[1], nnew = (uint64_t)hs.nwin[0] + hs.nwin[1];
    newnuc += hs.nnuc;  // nuclei the device placed before the grow
    c->n_nuclei += hs.nnuc;

    // mobility weights requested this step: computed on the host (FP64, libm)
    double pmax_new = 0.0;
    if (hs.pmax_bits) memcpy(&pmax_new, &hs.pmax_bits, 8);
    uint32_t nreq = 0;  // distinct weights requested (void race slots excluded)
    c->ntouch = hs.ntouch;
    if (c->ans_ready) {  // computed by the engine over all domains' requests
        c->ans_ready = false;
        for (double v : c->ans_val) if (v > pmax_new) pmax_new = v;
        for (unsigned long long x : c->ans_idx) nreq += x != kMissVoid;
    } else if (hs.nmiss > 0) {
        c->ans_idx.clear();
        c->ans_val.clear();
        std::vector<unsigned long long> idx(hs.nmiss);
        std::vector<double> val;
        cudaError_t e = cudaSuccess;
        if (hs.nmiss <= kBoxMiss) {
            memcpy(idx.data(), c->h_box->miss, (size_t)hs.nmiss * 8);
        } else {
            e = cudaMemcpyAsync(idx.data(), a.miss, (size_t)hs.nmiss * 8, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return c->cuda_fail(e, "read misses");
        }
        const auto w_t0 = std::chrono::steady_clock::now();
        resolve_weights(c, idx, val);
        c->weights_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w_t0).count();
        for (double v : val) if (v > pmax_new) pmax_new = v;
        for (unsigned long long x : idx) nreq += x != kMissVoid;
        // staged by the engine into one host-to-device copy before the next step
        c->ans_idx.swap(idx);
        c->ans_val.swap(val);
    } else {
        c->ans_idx.clear();
        c->ans_val.clear();
    }
    for (unsigned long long x : c->ans_idx)
        if (x != kMissVoid) c->ptab_touched.push_back(x);
    // deformed grains that ran out of cells this step (synchronize_mydefpool_counts)
    if (hs.ndepleted > 0) {
        const uint32_t nd = std::min(hs.ndepleted, c->ndefg);
        if (nd <= kBoxDep) {
            for (uint32_t i = 0; i < nd; ++i) c->defg_cnt_host[c->h_box->depleted[i]] = 0;
        } else {
            std::vector<uint32_t> dep(nd);
            cudaError_t e = cudaMemcpyAsync(dep.data(), a.depleted, (size_t)nd * 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return c->cuda_fail(e, "read depleted grains");
            for (uint32_t g : dep) c->defg_cnt_host[g] = 0;
        }
        c->rhomax_version = ~0ull;  // the set of grains with cells left changed
    }
    for (int L = 0; L < 2; ++L) {
        c->next_never[L] = hs.next_never[L];
        c->high_water[L] = std::max(c->high_water[L], c->next_never[L]);
    }

    // master block, SCORE_Kernel.cpp:6691-6740
    const double dt_used = ph.dt;
    if (pmax_new >= ph.Pmax) ph.Pmax = pmax_new;  // running max over every P ever assigned, floored at 0
    c->Xcells = c->Xcells + (double)nfull;
    const double X = (c->Xcells / (double)c->N);
    if (c->rhomax_version != c->rho_version) {  // rho max only moves when rho or the grain set changes
        if (c->rho_version == 0 || c->prm.recovery_model == SCORE_RECOVERY_HYPERBOLIC) {
            // rho is rho0, or rho0 / (1 + k t) (same order): the first grain in descending-rho0
            // order that has cells
            while (c->rho_cursor < c->rho_order.size() && c->defg_cnt_host[c->rho_order[c->rho_cursor]] == 0) ++c->rho_cursor;
            const double best = c->rho_cursor < c->rho_order.size() ? c->rho[c->rho_order[c->rho_cursor]] : -1.0;
            ph.rhomax = (best >= kRhomaxWellAnnealed) ? best : kRhomaxWellAnnealed;
        } else {
            ph.rhomax = rhomax_of(c->rho, c->defg_cnt_host);
        }
        c->rhomax_version = c->rho_version;
    }
    const double rhomax_step = ph.rhomax;
    if (c->log_next < c->log_cells.size() && c->Xcells >= c->log_cells[c->log_next]) {
        const int ls = log_snapshot(c, Sv);
        if (ls != SCORE_OK) return ls;
        c->log_next++;
    }
    if (!c->ahead) {
        const int s = physics_ahead(c);
        if (s != SCORE_OK) return s;
    }
    c->ahead = false;
    if (recovering(c)) {
        c->rho.swap(c->rho_next);
        c->rho_version++;
    }
    ph.dt = ph.dt_minimum();
    c->step++;

    score_step_stats& o = c->last;
    o = score_step_stats{};
    o.step = c->step; o.n_nuclei = newnuc; o.t = ph.t; o.dt = ph.dt; o.dt_used = dt_used;
    o.Xcells = c->Xcells; o.X = X; o.Sv = Sv; o.n_full = nfull; o.n_new = nnew;
    o.Pmax = ph.Pmax; o.rhomax = rhomax_step; o.dXstep = 0.0;
    o.next_never[0] = c->next_never[0]; o.next_never[1] = c->next_never[1];
    o.n_recycled[0] = hs.nrec[0]; o.n_recycled[1] = hs.nrec[1];
    o.p_misses = nreq + hs.nknown;
    if (out) *out = o;
    return SCORE_OK;
}

// the stop rule at the top of the step loop, SCORE_Kernel.cpp:6619
bool domain_done(const score_ctx* c, double xt) {
    const double X = c->Xcells / (double)c->N;
    return (c->Xcells >= (double)c->N) || (X > xt) || (c->step > c->prm.nmax) || (c->ph.t > c->ph.t_end) || (c->ph.t > c->prm.tmax);
}

// phase boundary: a real event record node when the sequence is captured into a graph
inline void record(const Engine& E, int k) {
    if (!E.events) return;
    if (E.capturing) cudaEventRecordWithFlags(E.ev[k], E.stream, cudaEventRecordExternal);
    else cudaEventRecord(E.ev[k], E.stream);
}

template <bool FP32, int ITEMS>
void launch_grow(const Engine& E, int n) {
    const uint32_t g = (uint32_t)(E.sms * E.cfg.fill_bpsm);
    const int m = E.fill_mode;  // a single domain's is one of 0..4
    if (n == 1) {
        if (m == 4 || (FP32 && m == 3)) {
            // FP32 keeps no increment (its fill step is vel dt / cellsize), so grow mode 3 is mode 0 there
            k_grow_fill_sparse<FP32, ITEMS><<<g, kBlock, 0, E.stream>>>(E.base);
        } else if (m == 1) {
            k_grow_fill<FP32, ITEMS, true, 1><<<g, kBlock, 0, E.stream>>>(E.base, n);
        } else if (m == 2) {
            k_grow_fill<FP32, ITEMS, true, 2><<<g, kBlock, 0, E.stream>>>(E.base, n);
        } else if constexpr (FP32) {
            k_grow_fill<true, ITEMS, true, 0><<<g, kBlock, 0, E.stream>>>(E.base, n);
        } else if (m == 0) {
            k_grow_fill_pf0<ITEMS><<<g, kBlock, 0, E.stream>>>(E.base);
        } else if constexpr (ITEMS <= 8) {
            k_grow_fill_pf<ITEMS><<<g, kBlock, 0, E.stream>>>(E.base);
        } else {
            k_grow_fill<false, ITEMS, true, 3><<<g, kBlock, 0, E.stream>>>(E.base, n);  // 16 items spill in the pipelined kernel
        }
    } else if (m == 5) {  // a batch whose domains all step from cached increments
        k_grow_fill_sparse_batch<FP32, ITEMS><<<g, kBlock, 0, E.stream>>>(E.base, n);
    } else if (m == 2) {
        k_grow_fill<FP32, ITEMS, false, 2><<<g, kBlock, 0, E.stream>>>(E.base, n);
    } else {
        k_grow_fill<FP32, ITEMS, false, kFillAny><<<g, kBlock, 0, E.stream>>>(E.base, n);
    }
    record(E, 1);
    k_grow_lists<ITEMS><<<(uint32_t)E.sms * 8, kBlock, 0, E.stream>>>(E.base, n);
}

template <bool FP32>
void launch_sequence_t(const Engine& E, int n) {
    cudaStream_t st = E.stream;
    const int d = E.base;
    const uint32_t S = (uint32_t)E.sms;
    record(E, 0);
    if (E.cfg.items == 4) launch_grow<FP32, 4>(E, n);
    else if (E.cfg.items == 16) launch_grow<FP32, 16>(E, n);
    else launch_grow<FP32, 8>(E, n);
    record(E, 2);
    if (n == 1) k_claim<true><<<S * (uint32_t)E.cfg.claim_bpsm, kBlock, 0, st>>>(d, n);
    else k_claim<false><<<S * (uint32_t)E.cfg.claim_bpsm, kBlock, 0, st>>>(d, n);
    record(E, 3);
    const uint32_t gt = (uint32_t)(kBlock * E.cfg.items);
    if (n == 1) {
        k_resolve<true><<<S * (uint32_t)E.cfg.commit_bpsm, kBlock, 0, st>>>(d, n);
        k_commit<FP32, true><<<S * (uint32_t)E.cfg.commit_bpsm, kBlock, 0, st>>>(d, n, gt);  // ends the step too
    } else {
        k_resolve<false><<<S * (uint32_t)E.cfg.commit_bpsm, kBlock, 0, st>>>(d, n);
        k_commit<FP32, false><<<S * (uint32_t)E.cfg.commit_bpsm, kBlock, 0, st>>>(d, n, gt);
        k_step_end<<<(uint32_t)n, kBlock, 0, st>>>(d, n, gt);
    }
    record(E, 4);
}

// kernels per step: fill, lists, claim, resolve, commit, and for batches a separate step end
inline int step_kernels(int n) { return n == 1 ? 5 : 6; }

}  // namespace

void Engine::launch_sequence(int n) {
    if (fp32) launch_sequence_t<true>(*this, n);
    else launch_sequence_t<false>(*this, n);
}

// the argument copy and the kernels of one step, as a graph replay or direct launches
cudaError_t Engine::enqueue_step(int n, bool timed, int mode) {
    // the argument blocks only change when dt, the physics or a domain's state changes
    cudaError_t e = cudaSuccess;
    if (args_dirty || memcmp(h_args, h_args_dev.data(), (size_t)n * sizeof(DomainArgs)) != 0) {
        e = cudaMemcpyAsync(d_args, h_args, (size_t)n * sizeof(DomainArgs), cudaMemcpyHostToDevice, stream);
        memcpy(h_args_dev.data(), h_args, (size_t)n * sizeof(DomainArgs));
        args_dirty = false;
    }
    if (e != cudaSuccess) return e;
    events = timed;
    fill_mode = mode;
    if (!use_graph) {
        launch_sequence(n);
        launches += step_kernels(n);
        return cudaGetLastError();
    }
    const int k = (timed ? 1 : 0) + 2 * (mode == kFillAny ? 6 : mode);
    if (!gexec[k] || gndom[k] != n || !(gcfg[k] == cfg) || gfp32[k] != fp32) {
        if (gexec[k]) cudaGraphExecDestroy(gexec[k]);
        gexec[k] = nullptr;
        gndom[k] = -1;
        cudaGraph_t g = nullptr;
        e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return e;
        capturing = true;
        launch_sequence(n);
        capturing = false;
        e = cudaStreamEndCapture(stream, &g);
        if (e == cudaSuccess) e = cudaGraphInstantiate(&gexec[k], g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) { gexec[k] = nullptr; return e; }
        gndom[k] = n; gcfg[k] = cfg; gfp32[k] = fp32;
    }
    launches += step_kernels(n);
    return cudaGraphLaunch(gexec[k], stream);
}

// Pack every domain's answered weights into the pinned, device-mapped staging buffer
// and point the domains' argument blocks at their part of it.
int Engine::stage_answers() {
    size_t total = 0;
    for (score_ctx* c : dom) total += c->ans_idx.size();
    ans_total = 0;
    if (total == 0) return SCORE_OK;
    if (total > ans_cap) {
        const size_t cap = std::max<size_t>(total, 2 * ans_cap);
        if (h_ans_i) cudaFreeHost(h_ans_i);
        if (h_ans_v) cudaFreeHost(h_ans_v);
        h_ans_i = nullptr; h_ans_v = nullptr; d_ans_i = nullptr; d_ans_v = nullptr;
        ans_cap = 0;
        cudaError_t e = cudaHostAlloc((void**)&h_ans_i, cap * 8, cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostAlloc((void**)&h_ans_v, cap * 8, cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&d_ans_i, h_ans_i, 0);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&d_ans_v, h_ans_v, 0);
        if (e != cudaSuccess) return fail(SCORE_ERR_NOMEM, "weight staging buffers");
        ans_cap = cap;
    }
    size_t off = 0;
    for (score_ctx* c : dom) {
        const size_t k = c->ans_idx.size();
        if (!k) continue;
        memcpy(h_ans_i + off, c->ans_idx.data(), k * 8);
        memcpy(h_ans_v + off, c->ans_val.data(), k * 8);
        c->a.ans_idx = d_ans_i + off;
        c->a.ans_val = d_ans_v + off;
        off += k;
    }
    ans_total = total;
    return SCORE_OK;
}

// The requested weights of all running domains of a batch, spread evenly over the workers:
// after nucleation a few domains request thousands of weights and would hold up a step
// whose post-processing gives each domain to one worker.  Few requests stay with their
// domain's post step.
void Engine::balance_weights() {
    std::vector<score_ctx*> req;
    std::vector<size_t> off(1, 0);
    for (score_ctx* c : dom) {
        c->ans_ready = false;
        if (!c->running) continue;
        const DevState& hs = c->h_box->snap;
        if (hs.err || hs.nmiss == 0 || hs.nmiss > kBoxMiss) continue;
        req.push_back(c);
        off.push_back(off.back() + hs.nmiss);
    }
    const size_t total = off.back();
    if (total < 512) return;
    const auto t0 = std::chrono::steady_clock::now();
    for (size_t j = 0; j < req.size(); ++j) {
        score_ctx* c = req[j];
        c->ans_idx.assign(c->h_box->miss, c->h_box->miss + (off[j + 1] - off[j]));
        c->ans_val.assign(off[j + 1] - off[j], 0.0);
        c->ans_ready = true;
    }
    constexpr size_t kChunk = 64;
    const int nchunks = (int)((total + kChunk - 1) / kChunk);
    workers(15);
    pool->run(nchunks, [&](int k) {
        const size_t lo = (size_t)k * kChunk, hi = std::min(total, lo + kChunk);
        size_t j = (size_t)(std::upper_bound(off.begin(), off.end(), lo) - off.begin()) - 1;
        for (size_t i = lo; i < hi; ++i) {
            while (i >= off[j + 1]) ++j;
            score_ctx* c = req[j];
            const unsigned long long x = c->ans_idx[i - off[j]];
            // a void slot (lost race) keeps 0, which no cell reads
            if (x != kMissVoid) c->ans_val[i - off[j]] = weight_of(c, (uint32_t)(x / c->ndefg), (uint32_t)(x % c->ndefg));
        }
    });
    tm.weights_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// One step of every running domain.
int Engine::step(bool timed) {
    cudaSetDevice(device);
    const auto host_t0 = std::chrono::steady_clock::now();
    const int n = (int)dom.size();
    std::vector<uint32_t> newnuc(n, 0);
    int nrun = 0;
    for (int i = 0; i < n; ++i) {
        score_ctx* c = dom[i];
        if (c->running) {
            const int s = c->pre_done ? SCORE_OK : pre_step(c, &c->pre_newnuc);
            if (s != SCORE_OK) return fail(s, c->err);
            newnuc[i] = c->pre_newnuc;
            c->pre_done = false;
            if ((c->fuse_replay & kCmdForce) &&  // the forces of a command that no launch took
                cudaMemcpyAsync(c->d_pforce, c->h_box->fuse.pay.pf_src, (size_t)c->ndefg * 8, cudaMemcpyHostToDevice, c->stream) != cudaSuccess)
                return fail(SCORE_ERR_CUDA, "upload driving force");
            c->fuse_replay = 0;
            ++nrun;
        } else {
            c->a.active = 0;
        }
        h_args[i] = c->a;
    }
    if (nrun == 0) return SCORE_OK;
    const auto pre_t1 = std::chrono::steady_clock::now();
    tm.pre_ms += std::chrono::duration<double, std::milli>(pre_t1 - host_t0).count();
    // the grow mode every stepping domain shares (a kernel specialised to it), or per domain
    int mode = -2;
    for (int i = 0; i < n; ++i) {
        if (!dom[i]->running) continue;
        const DomainArgs& a = h_args[i];
        // 0 cached increments, 1 / 2 refresh, 3 as 0 with few holes and dt unchanged, 4 as 0 with many holes
        const int m = a.refresh == 2 ? 2 : a.refresh == 1 ? 1 : !a.spec ? 4 : !a.dt_changed ? 3 : 0;
        mode = (mode == -2 || mode == m) ? m : kFillAny;
    }
    // batches: the gathered-slot kernel when no domain refreshes, the refresh-only kernel when all
    // refresh from cached mobilities, else the per-domain one
    if (n > 1 && mode != 2) {
        bool cached = true;
        for (int i = 0; i < n; ++i)
            if (dom[i]->running && h_args[i].refresh != 0) cached = false;
        mode = cached ? 5 : kFillAny;
    }
    cudaError_t e = enqueue_step(n, timed, mode);
    ++run_steps;
    // while the GPU steps: each domain's outcome-independent physics for the next step
    std::vector<int> status(n, SCORE_OK);
    if (e == cudaSuccess) {
        auto ahead = [&](int i) {
            score_ctx* c = dom[i];
            if (!c->running) return;
            cudaSetDevice(device);  // the calling thread may be a worker
            status[i] = c->ahead ? flush_pforce(c) : physics_ahead(c);
        };
        if (n >= 4) {
            workers(15);
            pool->run(n, ahead);
        } else {
            for (int i = 0; i < n; ++i) ahead(i);
        }
    }
    const auto wait_t0 = std::chrono::steady_clock::now();
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);  // the one wait of the step: the mailboxes are filled
    const auto wait_t1 = std::chrono::steady_clock::now();
    tm.wait_ms += std::chrono::duration<double, std::milli>(wait_t1 - wait_t0).count();
    if (e != cudaSuccess) {
        for (score_ctx* c : dom) c->failed = true;
        return fail(SCORE_ERR_CUDA, std::string("growth step: ") + cudaGetErrorString(e));
    }
    if (timed) {
        float f = 0, g = 0, cl = 0, cm = 0;
        e = cudaEventElapsedTime(&f, ev[0], ev[1]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&g, ev[0], ev[2]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&cl, ev[2], ev[3]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&cm, ev[3], ev[4]);
        if (e != cudaSuccess) return fail(SCORE_ERR_CUDA, std::string("phase timing: ") + cudaGetErrorString(e));
        tm.fill_ms += f; tm.grow_ms += g; tm.claim_ms += cl; tm.commit_ms += cm;
        tm.total_ms += g + cl + cm;
        tm.timed_steps += 1;
    }
    tm.grow_launches += 1;
    const double bpu = fp32 ? 21.0 : 25.0;  // algorithmic bytes per front-cell update of k_grow_fill
    for (int i = 0; i < n; ++i)
        if (status[i] != SCORE_OK) return fail(status[i], dom[i]->err);
    if (n >= 4) balance_weights();
    // the master-block work of each domain (weights, P max, X, rho max, dt) is independent
    auto post = [&](int i) {
        score_ctx* c = dom[i];
        if (!c->running) return;
        cudaSetDevice(device);  // the calling thread may be a worker
        status[i] = post_step(c, newnuc[i], nullptr);
    };
    if (n >= 4) {
        workers(15);
        pool->run(n, post);
    } else {
        for (int i = 0; i < n; ++i) post(i);
    }
    for (int i = 0; i < n; ++i) {
        score_ctx* c = dom[i];
        if (!c->running) continue;
        if (status[i] != SCORE_OK) return fail(status[i], c->err);
        const score_step_stats& st = c->last;
        if (timed) {  // bytes of the timed steps, so that bytes / time is a rate
            tm.grow_bytes += bpu * (double)st.Sv;
            tm.step_bytes += bpu * (double)st.Sv + 120.0 * (double)st.n_full + 37.0 * (double)st.n_new;
        }
        tm.weights_ms += c->weights_ms;
        c->weights_ms = 0.0;
    }
    const int sa = stage_answers();
    if (sa != SCORE_OK) return sa;
    tm.post_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wait_t1).count();
    tm.host_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - host_t0).count();
    return SCORE_OK;
}

int Engine::mark_run_end() {
    cudaEventRecord(ev[6], stream);
    cudaError_t e = cudaEventSynchronize(ev[6]);
    float ms = 0.0f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ev[5], ev[6]);
    if (e != cudaSuccess) return fail(SCORE_ERR_CUDA, std::string("run timing: ") + cudaGetErrorString(e));
    tm.run_ms = ms;
    return SCORE_OK;
}

// ------------------------------------------------------------------ many steps in one launch
namespace {

uint32_t fuse_tiles(const score_ctx* c, int items) {
    const uint32_t tile = (uint32_t)(kFuse * items);
    return (c->next_never[0] + tile - 1) / tile + (c->next_never[1] + tile - 1) / tile;
}

FusePay fuse_pay(const score_ctx* c) {
    FusePay p{};
    const DomainArgs& a = c->a;
    p.mLAGB = a.mLAGB; p.mHAGB = a.mHAGB; p.mGS = a.mGS; p.mRH = a.mRH;
    p.dt = a.dt; p.cinv = a.cinv; p.dtc32 = a.dtc32;
    p.ans_idx = a.ans_idx; p.ans_val = a.ans_val;
    p.pf_src = c->h_pforce + (size_t)c->pf_buf * c->ndefg;
    return p;
}

uint32_t fuse_flags(const score_ctx* c) {
    const DomainArgs& a = c->a;
    return (a.dt_changed ? kCmdDtChanged : 0u) | (a.spec ? kCmdSpec : 0u) |
           (a.refresh == 1 ? kCmdRefresh1 : a.refresh == 2 ? kCmdRefresh2 : 0u);
}

inline void fuse_store(uint32_t* p, uint32_t v) { __atomic_store_n(p, v, __ATOMIC_RELEASE); }
inline uint32_t fuse_load(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }

// whether the next step needs the stream before it starts: nuclei due, a defragmentation
bool fuse_needs_stream(const score_ctx* c) {
    if (c->nuc_pos < c->nuc_order.size() && c->tincub[c->nuc_order[c->nuc_pos]] <= c->ph.t) return true;
    return c->prm.defragmentation && c->defrag_cnt < c->prm.n_defrag && c->Xcells >= c->prm.defrag_x[c->defrag_cnt] * (double)c->N;
}

// one domain of a session, as its host thread sees it
struct FuseServe {
    score_ctx* c = nullptr;
    size_t i = 0;
    uint32_t blocks = 0;
    bool open = false;      // its group steps, or was told to
    bool deferred = false;  // posted, but its post step needs the stream: after the launch
    int status = SCORE_OK;
    uint32_t steps = 0, timed = 0;
    uint32_t word = 0;      // its last command
    double bytes = 0.0, sbytes = 0.0, fill = 0.0, res = 0.0, com = 0.0, post = 0.0;
};

}  // namespace

// Steps run inside one launch while every running domain's front is small; the launch configuration's
// direct launches (use_graph 0, the autotuner) keep the separate kernels.
bool Engine::fused_ok() const {
    if (!fuse || !use_graph) return false;
    uint64_t nrun = 0, tiles = 0, slots = 0;
    for (const score_ctx* c : dom) {
        if (!c->running) continue;
        ++nrun;
        tiles += fuse_tiles(c, 4);
        const uint64_t s = (uint64_t)c->next_never[0] + c->next_never[1];
        if (s > lim.slots) return false;
        slots += s;
    }
    if (slots > (uint64_t)lim.block_slots * (uint64_t)fuse_sms) return false;
    // a domain's blocks follow its share of the tiles: kFuseMaxLocal tiles a block with room to grow
    return nrun > 0 && nrun < (uint64_t)fuse_sms && tiles + 4 * nrun <= (kFuseMaxLocal / 2) * ((uint64_t)fuse_sms - nrun);
}

// One launch that steps every running domain until it meets its stop rule, needs the stream (nuclei due, a
// logged step, a defragmentation, requests beyond the mailbox) or the launch has run for a while: other
// work of the device gets its turn then.  `one`: a single step.  done[i]: steps of domain i in this run.
int Engine::fused_session(double x_target, uint32_t max_steps, bool one, std::vector<uint32_t>& done) {
    cudaSetDevice(device);
    const auto t0 = std::chrono::steady_clock::now();
    const int n = (int)dom.size();
    uint64_t slots = 0;
    for (const score_ctx* c : dom)
        if (c->running) slots += (uint64_t)c->next_never[0] + c->next_never[1];
    // 4 slots a thread and tile once every block has several tiles of 2
    const int items = slots >= (uint64_t)lim.wide * (uint64_t)fuse_sms ? 4 : 2;
    std::vector<FuseServe> sv;
    FuseMap map{};
    uint64_t work = 0;
    for (int i = 0; i < n; ++i) {
        score_ctx* c = dom[i];
        if (!c->running) { c->a.active = 0; h_args[i] = c->a; continue; }
        const int s = c->pre_done ? SCORE_OK : pre_step(c, &c->pre_newnuc);
        if (s != SCORE_OK) return fail(s, c->err);
        c->pre_done = true;
        h_args[i] = c->a;
        FuseServe f;
        f.c = c; f.i = (size_t)i;
        sv.push_back(f);
        work += 2ull * fuse_tiles(c, items) + 8;
    }
    const auto t_pre = std::chrono::steady_clock::now();
    tm.pre_ms += std::chrono::duration<double, std::milli>(t_pre - t0).count();
    // blocks in proportion to the fronts, at least one a domain, no more than tiles a front may have soon
    uint32_t total = 0;
    {
        const uint32_t spare = (uint32_t)fuse_sms - (uint32_t)sv.size();
        size_t k = 0;
        for (int i = 0; i < n; ++i) {
            map.first[i] = (uint16_t)total;
            if (k < sv.size() && sv[k].i == (size_t)i) {
                const uint32_t want = 2 * fuse_tiles(sv[k].c, items) + 8;
                sv[k].blocks = std::min(want, 1u + (uint32_t)((uint64_t)spare * want / work));
                total += sv[k].blocks;
                map.seq[i] = sv[k].c->fuse_seq;
                ++k;
            }
        }
        map.first[n] = (uint16_t)total;
        map.ndom = (uint32_t)n;
        map.group_polls = lim.group_polls;
        map.host_polls = lim.host_polls;
    }
    cudaError_t e = cudaSuccess;
    if (args_dirty || memcmp(h_args, h_args_dev.data(), (size_t)n * sizeof(DomainArgs)) != 0) {
        e = cudaMemcpyAsync(d_args, h_args, (size_t)n * sizeof(DomainArgs), cudaMemcpyHostToDevice, stream);
        memcpy(h_args_dev.data(), h_args, (size_t)n * sizeof(DomainArgs));
        args_dirty = false;
    }
    for (FuseServe& f : sv) {
        score_ctx* c = f.c;
        if (c->fuse_replay) {
            f.word = c->fuse_replay & ((1u << kCmdShift) - 1u);
            c->fuse_sent = c->h_box->fuse.pay;
        } else {
            f.word = fuse_flags(c);
            c->fuse_sent = fuse_pay(c);
        }
        f.word |= (c->fuse_seq << kCmdShift) | (one ? kCmdLast : 0u);
        // numbers come back after 2^24 steps: the device's words of an earlier launch would be taken for this one's
        c->h_box->fuse.post = 0;
        c->h_box->fuse.left = 0;
        fuse_store(&c->h_box->fuse.cmd, f.word);
        c->fuse_live = true;
        f.open = true;
    }
    if (e == cudaSuccess) {
        void* args[] = {(void*)&map, (void*)&base};
        const void* k = items == 4 ? (fp32 ? (const void*)k_steps_fused<true, 4> : (const void*)k_steps_fused<false, 4>)
                                   : (fp32 ? (const void*)k_steps_fused<true, 2> : (const void*)k_steps_fused<false, 2>);
        if (lim.refuse_after == 0) e = cudaErrorCooperativeLaunchTooLarge;
        else e = cudaLaunchCooperativeKernel(k, dim3(total), dim3(kFuse), args, sizeof(FuseShared), stream);
        if (lim.refuse_after != ~0u) --lim.refuse_after;
    }
    if (e != cudaSuccess) {
        for (FuseServe& f : sv) f.c->fuse_live = false;
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources) {
            cudaGetLastError();
            fuse = false;  // the separate kernels from now on; they take a command to give again too
            return SCORE_OK;
        }
        for (score_ctx* c : dom) c->failed = true;
        return fail(SCORE_ERR_CUDA, std::string("growth steps: ") + cudaGetErrorString(e));
    }
    launches += 1;
    for (FuseServe& f : sv) f.c->fuse_replay = 0;
    std::atomic<bool> stop{false};
    // the launch's turn starts with its first step: one that has waited in the queue for other work has not used any
    std::atomic<int64_t> turn{0};
    auto now_us = [&] { return std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - t0).count() + 1; };
    const double bpu = fp32 ? 21.0 : 25.0;
    const uint64_t sample0 = run_steps;
    auto timed_step = [&](const FuseServe& f) {
        return cfg.timing_every > 0 && (sample0 + f.steps) % (uint64_t)cfg.timing_every == 0;
    };
    auto leave = [&](FuseServe& f) {  // the posted step's group leaves the launch
        score_ctx* c = f.c;
        f.open = false;
        if (one) return;  // it has left
        fuse_store(&c->h_box->fuse.cmd, (c->fuse_seq << kCmdShift) | kCmdLeave);
        c->fuse_seq = fuse_next(c->fuse_seq);
    };
    // after the post of a step: the host's part of it, and the next command
    auto finish_step = [&](FuseServe& f) -> int {
        score_ctx* c = f.c;
        const FuseHost& h = c->h_box->fuse;
        const auto p0 = std::chrono::steady_clock::now();
        const bool is_timed = timed_step(f);
        if (is_timed) {
            f.timed++;
            f.fill += 1e-6 * h.phase_ns[0]; f.res += 1e-6 * h.phase_ns[1]; f.com += 1e-6 * h.phase_ns[2];
        }
        c->pre_done = false;
        const int s = post_step(c, c->pre_newnuc, nullptr);
        if (s != SCORE_OK) return s;
        if (is_timed || sv.size() > 1) {
            f.bytes += bpu * (double)c->last.Sv;
            f.sbytes += 120.0 * (double)c->last.n_full + 37.0 * (double)c->last.n_new;
        }
        if (!c->ans_idx.empty() && c->ans_idx.size() <= kBoxMiss) {
            memcpy(c->h_box->ans_idx, c->ans_idx.data(), c->ans_idx.size() * 8);
            memcpy(c->h_box->ans_val, c->ans_val.data(), c->ans_val.size() * 8);
            c->a.ans_idx = c->d_box->ans_idx;
            c->a.ans_val = c->d_box->ans_val;
        }
        f.steps++;
        done[f.i]++;
        if (!one) c->trace.push_back(c->last);
        f.post += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - p0).count();
        return SCORE_OK;
    };
    // one look at a domain's mailbox; false when there was nothing new
    auto poll = [&](FuseServe& f) -> bool {
        score_ctx* c = f.c;
        FuseHost& h = c->h_box->fuse;
        const uint32_t seq = c->fuse_seq;
        if (fuse_load(&h.post) != seq) {
            if (fuse_load(&h.left) != seq) return false;
            f.open = false;  // the group left before it saw the command: the next launch takes the step
            c->fuse_seq = fuse_next(seq);
            c->fuse_replay = (f.word & ((1u << kCmdShift) - 1u) & ~kCmdLast) | kCmdReplay;
            return true;
        }
        c->fuse_seq = fuse_next(seq);
        if (turn.load(std::memory_order_relaxed) == 0) {
            int64_t none = 0;
            turn.compare_exchange_strong(none, now_us());
        }
        const DevState& hs = c->h_box->snap;
        if (hs.err || hs.nmiss > kBoxMiss || hs.ndepleted > kBoxDep) {
            f.deferred = true;
            stop.store(true, std::memory_order_relaxed);
            leave(f);
            return true;
        }
        const size_t logged = c->log_info.size();
        f.status = finish_step(f);
        const double xt = x_target < 0 ? c->prm.xmax : x_target;
        const bool needs = f.status == SCORE_OK && (c->log_info.size() != logged || fuse_needs_stream(c) ||
                           (uint64_t)c->next_never[0] + c->next_never[1] > lim.slots || fuse_tiles(c, items) > std::min(kFuseMaxLocal * f.blocks, kFuseMaxTiles - 512));
        if (f.status != SCORE_OK || needs) stop.store(true, std::memory_order_relaxed);
        if (f.status != SCORE_OK || needs || one || domain_done(c, xt) || (max_steps && done[f.i] >= max_steps) ||
            stop.load(std::memory_order_relaxed)) {
            leave(f);
            return true;
        }
        f.status = pre_step(c, &c->pre_newnuc);  // no nuclei, no defragmentation: arguments only
        if (f.status != SCORE_OK) { stop.store(true, std::memory_order_relaxed); leave(f); return true; }
        c->pre_done = true;
        uint32_t w = (c->fuse_seq << kCmdShift) | fuse_flags(c);
        const FusePay pay = fuse_pay(c);
        if (c->pf_pending) { w |= kCmdForce | kCmdPayload; c->pf_pending = false; }
        if (memcmp(&pay, &c->fuse_sent, sizeof pay) != 0) w |= kCmdPayload;
        if (w & kCmdPayload) { h.pay = pay; c->fuse_sent = pay; }
        f.word = w;
        fuse_store(&h.cmd, w);
        f.status = physics_ahead(c);  // while the group steps
        if (f.status != SCORE_OK) stop.store(true, std::memory_order_relaxed);
        return true;
    };
    // serve domains first, first + every, ... until all their groups have left
    auto serve = [&](size_t first, size_t every) {
        cudaSetDevice(device);  // the calling thread may be a worker
        for (size_t k = first; k < sv.size(); k += every) {
            if (!sv[k].c->ahead) sv[k].status = physics_ahead(sv[k].c);
            if (sv[k].status != SCORE_OK) stop.store(true, std::memory_order_relaxed);
        }
        uint32_t idle = 0;
        for (;;) {
            bool open = false, any = false;
            for (size_t k = first; k < sv.size(); k += every) {
                if (!sv[k].open) continue;
                any |= poll(sv[k]);
                open |= sv[k].open;
            }
            if (!open) return;
            if (any) idle = 0;
            if (any || (++idle & 0xFFFu) == 0) {
                const int64_t since = turn.load(std::memory_order_relaxed);
                if (since != 0 && now_us() - since > kFuseTurnUs) stop.store(true, std::memory_order_relaxed);
            }
            if (any || (idle & 0xFFFFu) != 0) continue;
            // long silence: has the launch ended (an error, or a wait on the device that gave up)?
            const cudaError_t q = cudaStreamQuery(stream);
            if (q == cudaErrorNotReady) continue;
            for (size_t k = first; k < sv.size(); k += every) {
                if (!sv[k].open || poll(sv[k])) continue;  // its posts came before its end
                sv[k].open = false;
                sv[k].c->failed = true;
                sv[k].status = q != cudaSuccess ? sv[k].c->cuda_fail(q, "growth steps")
                                                : sv[k].c->fail(SCORE_ERR_TIMEOUT, "a bounded device wait gave up");
            }
        }
    };
    const size_t threads = std::min<size_t>(sv.size(), sv.size() > 1 ? 16 : 1);
    if (threads > 1) {
        WorkerPool& p = workers(15);
        const size_t every = std::min<size_t>(threads, p.size() + 1);
        p.run((int)every, [&](int w) { serve((size_t)w, every); });
    } else {
        serve(0, 1);
    }
    if (!one) {
        e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) {
            for (score_ctx* c : dom) c->failed = true;
            return fail(SCORE_ERR_CUDA, std::string("growth steps: ") + cudaGetErrorString(e));
        }
    }
    bool staged = false;
    int status = SCORE_OK;
    for (FuseServe& f : sv) {
        score_ctx* c = f.c;
        c->fuse_live = false;
        if (f.deferred && f.status == SCORE_OK) {
            f.status = finish_step(f);
            staged |= c->ans_idx.size() > kBoxMiss;
        }
        if (f.status == SCORE_OK && !c->fuse_replay) f.status = flush_pforce(c);
        if (f.status != SCORE_OK && status == SCORE_OK) { status = f.status; fail(status, c->err); }
        tm.weights_ms += c->weights_ms;
        c->weights_ms = 0.0;
    }
    if (status == SCORE_OK && staged) status = stage_answers();
    // the first domain's steps and phases stand for the launch's; bytes are every domain's in the timed share
    const FuseServe& f0 = sv[0];
    double bytes = 0.0, sbytes = 0.0;
    for (const FuseServe& f : sv) { bytes += f.bytes; sbytes += f.sbytes; }
    const double share = sv.size() == 1 ? 1.0 : f0.steps ? (double)f0.timed / f0.steps : 0.0;
    tm.fill_ms += f0.fill; tm.grow_ms += f0.fill + f0.res; tm.commit_ms += f0.com; tm.total_ms += f0.fill + f0.res + f0.com;
    tm.timed_steps += f0.timed;
    tm.grow_launches += f0.steps;
    tm.grow_bytes += bytes * share;
    tm.step_bytes += (bytes + sbytes) * share;
    run_steps += f0.steps;
    const double wall = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    double post = 0.0;
    for (const FuseServe& f : sv) post = std::max(post, f.post);
    tm.host_ms += wall;
    tm.post_ms += post;
    tm.wait_ms += std::max(0.0, wall - post - std::chrono::duration<double, std::milli>(t_pre - t0).count());
    return status;
}

// Step every domain until each meets its stop rule (X > x_target, time or step limits);
// a domain that stops leaves the launches, the others go on.  Each domain's per-step
// stats are kept in its trace.
int Engine::run_until(double x_target, uint32_t max_steps, uint32_t* steps_done) {
    uint32_t k = 0;
    std::vector<uint32_t> done(dom.size(), 0);  // steps of each domain
    for (;;) {
        int nrun = 0;
        for (size_t i = 0; i < dom.size(); ++i) {
            score_ctx* c = dom[i];
            const double xt = x_target < 0 ? c->prm.xmax : x_target;
            // a step that is prepared and waits for its next launch belongs to the run: its time has moved on already
            c->running = c->loaded && !c->failed && (c->pre_done || (!domain_done(c, xt) && !(max_steps && done[i] >= max_steps)));
            nrun += c->running;
        }
        if (nrun == 0) break;
        const bool fused = fused_ok();
        const int s = fused ? fused_session(x_target, max_steps, false, done) : step(sample_step());
        if (!fused && s == SCORE_OK)
            for (size_t i = 0; i < dom.size(); ++i)
                if (dom[i]->running) { dom[i]->trace.push_back(dom[i]->last); ++done[i]; }
        k = done.empty() ? 0 : *std::max_element(done.begin(), done.end());
        if (s != SCORE_OK) { if (steps_done) *steps_done = k; return s; }
    }
    for (score_ctx* c : dom) c->running = false;
    if (steps_done) *steps_done = k;
    return mark_run_end();
}

// ------------------------------------------------------------------ contexts
namespace {

int check_params(const score_params* p, int device) {
    if (p->nx < 3 || p->ny < 3 || p->nz < 3) return SCORE_ERR_ARG;
    const uint64_t N = (uint64_t)p->nx * p->ny * p->nz;
    if (N >= 0x7FFFFFFFull) return SCORE_ERR_ARG;  // slot counters and ranks are 32-bit with headroom
    if (8ull * ((p->nx + 1) / 2) * ((p->ny + 1) / 2) * ((p->nz + 1) / 2) >= 0x7FFFFFFFull) return SCORE_ERR_ARG;  // grid words
    if (p->n_schedule < 1) return SCORE_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return SCORE_ERR_NOT_BUILT; }
    if (device < 0 || device >= ndev) return SCORE_ERR_ARG;
    return SCORE_OK;
}

// a domain context stepped by `eng` (owned: a single-domain context; else a batch member)
int make_ctx(const score_params* p, Engine* eng, bool own, score_ctx** out) {
    score_ctx* c = new score_ctx();
    c->prm = *p;
    c->device = eng->device;
    c->nx = p->nx; c->ny = p->ny; c->nz = p->nz; c->N = (uint64_t)p->nx * p->ny * p->nz;
    c->ncells = 8ull * ((p->nx + 1) / 2) * ((p->ny + 1) / 2) * ((p->nz + 1) / 2);
    c->fp32 = p->precision == SCORE_PRECISION_FP32_KAHAN;
    c->eng = eng;
    c->own_eng = own;
    eng->dom.push_back(c);
    c->stream = eng->stream;
    c->sms = eng->sms;
    cudaError_t e = cudaMallocHost((void**)&c->h_state, sizeof(DevState));
    if (e == cudaSuccess) e = cudaHostAlloc((void**)&c->h_box, sizeof(HostBox), cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&c->d_box, c->h_box, 0);
    if (e != cudaSuccess) {
        eng->dom.pop_back();
        if (!own) c->eng = nullptr;
        delete c;
        return SCORE_ERR_CUDA;
    }
    // pinned memory comes back from an earlier context as that one left it: a post or a notice of leaving
    // with the number of a step of this context would be taken for its own
    memset(&c->h_box->fuse, 0, sizeof(FuseHost));
    memset(&c->h_box->snap, 0, sizeof(DevState));
    *out = c;
    return SCORE_OK;
}

}  // namespace

// ------------------------------------------------------------------ autotuner
// Runs real steps (results do not depend on the tile configuration: every compaction
// keeps slot order and claims are decided by ordinal) while cycling candidate
// configurations step by step, and keeps per kernel group the candidate with the least
// time per unit of work: k_grow_fill + k_grow_lists per front slot, k_claim per full
// cell, k_resolve + k_commit per full cell.  Direct launches while tuning.
int Engine::autotune(double x_target, uint32_t max_steps, score_tune* out) {
    static const int kItems[3] = {4, 8, 16};
    static const int kFill[4] = {4, 8, 16, 32};
    static const int kOther[4] = {2, 4, 8, 16};
    double ft[12] = {0}, fu[12] = {0}, ct[4] = {0}, cu[4] = {0}, mt[4] = {0}, mu[4] = {0};
    const bool graph = use_graph;
    use_graph = false;
    uint32_t k = 0;
    int status = SCORE_OK;
    for (;; ++k) {
        int nrun = 0;
        double slots = 0.0;
        for (score_ctx* c : dom) {
            const double xt = x_target < 0 ? c->prm.xmax : x_target;
            c->running = c->loaded && !c->failed && !domain_done(c, xt);
            if (c->running) { ++nrun; slots += (double)c->next_never[0] + (double)c->next_never[1]; }
        }
        if (nrun == 0 || (max_steps && k >= max_steps)) break;
        const int fi = (int)(k % 12), ci = (int)(k % 4), mi = (int)((k / 4) % 4);
        cfg.items = kItems[fi / 4];
        cfg.fill_bpsm = kFill[fi % 4];
        cfg.claim_bpsm = kOther[ci];
        cfg.commit_bpsm = kOther[mi];
        const score_timing before = tm;
        status = step(true);
        if (status != SCORE_OK) break;
        double full = 0.0;
        for (score_ctx* c : dom) if (c->running) full += (double)c->last.n_full;
        ft[fi] += tm.grow_ms - before.grow_ms; fu[fi] += slots;
        ct[ci] += tm.claim_ms - before.claim_ms; cu[ci] += full;
        mt[mi] += tm.commit_ms - before.commit_ms; mu[mi] += full;
    }
    for (score_ctx* c : dom) c->running = false;
    use_graph = graph;
    if (status != SCORE_OK) return status;
    auto best = [](const double* t, const double* u, int n) {
        int b = -1;
        for (int i = 0; i < n; ++i)
            if (u[i] > 0 && (b < 0 || t[i] / u[i] < t[b] / u[b])) b = i;
        return b;
    };
    const int bf = best(ft, fu, 12), bc = best(ct, cu, 4), bm = best(mt, mu, 4);
    TuneCfg t = cfg;  // the load strategy and the timing sample stay as they were set
    if (bf >= 0) { t.items = kItems[bf / 4]; t.fill_bpsm = kFill[bf % 4]; }
    if (bc >= 0) t.claim_bpsm = kOther[bc];
    if (bm >= 0) t.commit_bpsm = kOther[bm];
    cfg = t;
    if (out) {
        get_tune(out);
        out->fill_ns_per_slot = bf >= 0 ? 1e6 * ft[bf] / fu[bf] : 0.0;
        out->claim_ns_per_cell = bc >= 0 ? 1e6 * ct[bc] / cu[bc] : 0.0;
        out->commit_ns_per_cell = bm >= 0 ? 1e6 * mt[bm] / mu[bm] : 0.0;
        out->steps = k;
    }
    return SCORE_OK;
}

void Engine::get_tune(score_tune* out) const {
    *out = score_tune{};
    out->items = cfg.items;
    out->fill_blocks_per_sm = cfg.fill_bpsm;
    out->claim_blocks_per_sm = cfg.claim_bpsm;
    out->commit_blocks_per_sm = cfg.commit_bpsm;
    out->use_graph = use_graph ? 1 : 0;
    out->spec_holes_pct = cfg.spec_pct;
    out->timing_every = cfg.timing_every;
}

int Engine::set_tune(const score_tune* t) {
    if (t->items != 4 && t->items != 8 && t->items != 16) return fail(SCORE_ERR_ARG, "items must be 4, 8 or 16");
    for (int v : {t->fill_blocks_per_sm, t->claim_blocks_per_sm, t->commit_blocks_per_sm})
        if (v < 1 || v > 64) return fail(SCORE_ERR_ARG, "blocks per SM must be in 1..64");
    if (t->spec_holes_pct < 0 || t->spec_holes_pct > 100) return fail(SCORE_ERR_ARG, "spec_holes_pct must be in 0..100");
    if (t->timing_every < 0) return fail(SCORE_ERR_ARG, "timing_every must be >= 0");
    cfg.timing_every = t->timing_every;
    cfg.items = t->items;
    cfg.spec_pct = t->spec_holes_pct;
    cfg.fill_bpsm = t->fill_blocks_per_sm;
    cfg.claim_bpsm = t->claim_blocks_per_sm;
    cfg.commit_bpsm = t->commit_blocks_per_sm;
    use_graph = t->use_graph != 0;
    return SCORE_OK;
}

// ------------------------------------------------------------------ grain-evolution logs
namespace {

int grainevo_get(score_ctx* c, uint32_t i, score_grainevo_info* info, uint32_t* counts, uint32_t* rxarea) {
    if (i >= c->log_info.size()) return c->fail(SCORE_ERR_ARG, "no such grain-evolution snapshot");
    cudaSetDevice(c->device);
    if (info) *info = c->log_info[i];
    const size_t G = (size_t)c->ndefg + c->nrxg;
    cudaError_t e = cudaSuccess;
    if (counts) e = cudaMemcpyAsync(counts, c->d_log_counts + i * G, G * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && rxarea)
        e = cudaMemcpyAsync(rxarea, c->d_log_area + (size_t)i * 2 * c->nz, (size_t)2 * c->nz * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "read grain-evolution log");
    return SCORE_OK;
}

// Rows of k_rediscr_rows held at a time: the domains go in groups of up to kRowBytes (one at least), and a staging buffer larger
// than kRowKeep goes back after the call.
constexpr size_t kRowBytes = 256u << 20, kRowKeep = 64u << 20;

// Ensemble post-processing of the domains' grain-evolution logs on the device: kinetics (cls null)
// or macrotexture by orientation class.  Writes the time slots and [slot] or [slot][class] sums.
int rediscr(const std::vector<score_ctx*>& doms, uint32_t nslots, const uint32_t* cls, uint32_t nclass, double* t_out,
            double* out, double* boxvol_out, std::string& err) {
    if (doms.empty() || nslots < 2 || !t_out || !out) { err = "bad argument"; return SCORE_ERR_ARG; }
    if (cls && (nclass == 0 || nclass > kMaxClasses)) { err = "1 to 32 orientation classes"; return SCORE_ERR_ARG; }
    const int dev = doms[0]->device;
    double tmax = 0.0, box = 0.0;
    size_t ntimes = 0, ncls = 0;
    for (score_ctx* c : doms) {
        if (!c->loaded || c->device != dev) { err = "every domain must be loaded, on one device"; return SCORE_ERR_STATE; }
        // get_interpCellCount reads the first snapshot before the first log time: a domain needs one
        if (c->log_info.empty()) { err = "a domain has no grain-evolution snapshot (no logpoint reached)"; return SCORE_ERR_STATE; }
        if (c->ph.t >= tmax) tmax = c->ph.t;  // postprocess_init: the latest tsimend
        box = box + (double)c->N;
        ntimes += c->log_info.size();
        ncls += (size_t)c->ndefg + c->nrxg;
    }
    // postprocess_initrediscrtimes (REDISCR_TIME_EQUIDISTANT, tensmin 0)
    const double ttmin = 0.0, dt = (tmax - ttmin) / ((double)(nslots - 1));
    for (uint32_t n = 0; n < nslots; ++n) t_out[n] = ttmin + ((double)(n + 1) * dt);
    if (boxvol_out) *boxvol_out = box;
    cudaSetDevice(dev);
    for (score_ctx* c : doms) {  // every domain's last run is complete
        const cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) { err = cudaGetErrorString(e); return SCORE_ERR_CUDA; }
    }
    const uint32_t ndom = (uint32_t)doms.size(), m = cls ? nslots * nclass : nslots, nc = cls ? nclass : 1u;
    // one block of the first domain's staging buffer: what the host sends (descriptors, snapshot times, slot times,
    // grains by class), then rows and sums
    auto ngr_of = [&](const score_ctx* c) { return cls ? (size_t)c->ndefg + c->nrxg : (size_t)c->ndefg; };
    auto rows_of = [&](const score_ctx* c) { return (c->log_info.size() + 2) * ngr_of(c); };
    std::vector<uint32_t> group(1, 0);  // first domain of each group, and the end
    size_t nrows = 0, in_group = 0, maxgr = 0;
    for (uint32_t d = 0; d < ndom; ++d) {
        const size_t r = rows_of(doms[d]);
        if (d > group.back() && (in_group + r) * 16 > kRowBytes) { group.push_back(d); in_group = 0; }
        in_group += r;
        nrows = std::max(nrows, in_group);
        maxgr = std::max(maxgr, ngr_of(doms[d]));
    }
    group.push_back(ndom);
    const size_t b_evo = ndom * sizeof(EvoDev), b_t = ntimes * 8, b_w = (size_t)nslots * 8, b_o = cls ? ncls * 4 : 0, b_f = cls ? (size_t)ndom * (nc + 1) * 4 : 0;
    const size_t b_pd = (size_t)ndom * m * 8, b_out = (size_t)m * 8;
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t o_t = up(b_evo), o_w = o_t + up(b_t), o_o = o_w + up(b_w), o_f = o_o + up(b_o), sent = o_f + up(b_f);
    const size_t o_pd = sent + up(nrows * 16), o_out = o_pd + up(b_pd);
    if (!doms[0]->stage(o_out + up(b_out))) { err = "post-processing buffers"; return SCORE_ERR_NOMEM; }
    char* const blk = (char*)doms[0]->d_stage;
    std::vector<char> host(sent);
    EvoDev* evo = (EvoDev*)host.data();
    double* times = (double*)(host.data() + o_t);
    uint32_t* order = (uint32_t*)(host.data() + o_o);
    uint32_t* first = (uint32_t*)(host.data() + o_f);
    memcpy(host.data() + o_w, t_out, b_w);
    size_t toff = 0, coff = 0, roff = 0;
    for (uint32_t d = 0; d < ndom; ++d) {
        score_ctx* c = doms[d];
        EvoDev v{};
        const uint32_t G = c->ndefg + c->nrxg;
        v.t = (const double*)(blk + o_t) + toff;
        v.counts = c->d_log_counts;
        v.fin_defg = c->a.defg_cnt;
        v.fin_rxg = c->a.rxg_cnt;
        v.ndefg = c->ndefg; v.nrxg = c->nrxg; v.nsnap = (uint32_t)c->log_info.size();
        v.ngr = (uint32_t)ngr_of(c);
        v.tsimend = c->ph.t; v.nboxvol = (double)c->N;
        if (cls) {  // grains by class, in grain order within a class
            v.order = (const uint32_t*)(blk + o_o) + coff;
            v.first = (const uint32_t*)(blk + o_f) + (size_t)d * (nc + 1);
            uint32_t* f = first + (size_t)d * (nc + 1);
            for (uint32_t k = 0; k <= nc; ++k) f[k] = 0;
            for (uint32_t g = 0; g < G; ++g) f[cls[coff + g] + 1]++;
            for (uint32_t k = 0; k < nc; ++k) f[k + 1] += f[k];
            uint32_t at[kMaxClasses];
            for (uint32_t k = 0; k < nc; ++k) at[k] = f[k];
            for (uint32_t g = 0; g < G; ++g) order[coff + at[cls[coff + g]]++] = g;
        }
        if (std::find(group.begin(), group.end(), d) != group.end()) roff = 0;
        v.rows = (double2*)(blk + sent) + roff;
        for (const auto& info : c->log_info) times[toff++] = info.t;
        coff += G;
        roff += rows_of(c);
        evo[d] = v;
    }
    cudaStream_t st = doms[0]->stream;
    cudaError_t e = cudaMemcpyAsync(blk, host.data(), sent, cudaMemcpyHostToDevice, st);
    double* const d_pd = (double*)(blk + o_pd);
    double* const d_out = (double*)(blk + o_out);
    for (size_t k = 0; k + 1 < group.size() && e == cudaSuccess; ++k) {
        const uint32_t d0 = group[k], nd = group[k + 1] - d0;
        const EvoDev* d_evo = (const EvoDev*)blk + d0;
        k_rediscr_rows<<<dim3((unsigned)((maxgr + 255) / 256), nd), 256, 0, st>>>(d_evo);
        k_rediscr_sum<<<dim3((nslots + 31) / 32, nc, nd), 32, 0, st>>>(d_evo, (const double*)(blk + o_w), nslots, nc, cls ? 0 : 1,
                                                                       d_pd + (size_t)d0 * m);
        doms[0]->launches += 2;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        k_rediscr_ensemble<<<(m + 127) / 128, 128, 0, st>>>(d_pd, ndom, m, d_out);
        doms[0]->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_out, b_out, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (doms[0]->stage_cap > kRowKeep) doms[0]->unstage();
    if (e != cudaSuccess) { err = std::string("post-processing: ") + cudaGetErrorString(e); return SCORE_ERR_CUDA; }
    return SCORE_OK;
}

}  // namespace

// ------------------------------------------------------------------ C ABI
extern "C" {

int score_abi_version(void) { return SCORE_ABI_VERSION; }

const char* score_status_string(int s) {
    switch (s) {
        case SCORE_OK: return "ok";
        case SCORE_ERR_ARG: return "bad argument";
        case SCORE_ERR_CUDA: return "CUDA error";
        case SCORE_ERR_NOMEM: return "out of memory";
        case SCORE_ERR_CAPACITY: return "front list capacity exceeded";
        case SCORE_ERR_BORDER_CAPACITY: return "Border list exceeded the reference's 2(xy+xz+yz) slots";
        case SCORE_ERR_TIMEOUT: return "bounded device wait gave up";
        case SCORE_ERR_STATE: return "call out of sequence";
        case SCORE_ERR_IO: return "input file error";
        case SCORE_ERR_KEYLIMIT: return "too many infection attempts in one step";
        case SCORE_ERR_NOT_BUILT: return "CUDA device unavailable";
        case SCORE_ERR_SCRATCH_LIMIT: return "input larger than the static scratch of a no-allocation entry point (nrxg > 65536)";
        default: return "unknown status";
    }
}

const char* score_last_error(const score_ctx* c) { return c ? c->err.c_str() : "null context"; }

int score_create(score_ctx** out, const score_params* p, int device) {
    if (!out || !p) return SCORE_ERR_ARG;
    *out = nullptr;
    int s = check_params(p, device);
    if (s != SCORE_OK) return s;
    Engine* eng = new Engine();
    s = eng->init(device, 1);
    if (s != SCORE_OK) { delete eng; return s; }
    eng->fp32 = p->precision == SCORE_PRECISION_FP32_KAHAN;
    score_ctx* c = nullptr;
    s = make_ctx(p, eng, true, &c);
    if (s != SCORE_OK) return s;
    *out = c;
    return SCORE_OK;
}

void score_destroy(score_ctx* c) { delete c; }

int score_load_domain(score_ctx* c, const uint32_t* grid, const double* defg_quat, const double* defg_rho0, uint32_t ndefg,
                      const double* rxg_quat, const uint32_t* rxg_site, const double* rxg_tincub, uint32_t nrxg,
                      const double* ptable) {
    if (!c || !grid || !defg_quat || !defg_rho0 || !rxg_quat || !rxg_site || ndefg == 0) return SCORE_ERR_ARG;
    if ((uint64_t)ndefg + nrxg >= 4096000000ull) return c->fail(SCORE_ERR_ARG, "too many grains");
    const uint64_t N = c->N;
    for (uint32_t r = 0; r < nrxg; ++r) if (rxg_site[r] >= N) return c->fail(SCORE_ERR_ARG, "nucleation site outside the domain");
    cudaSetDevice(c->device);
    // a context reloads in place when the pool sizes match; otherwise it reallocates
    const bool reuse = c->a.grid && c->ndefg == ndefg && c->nrxg == nrxg;
    if (!reuse && c->a.grid) c->release_domain();
    c->loaded = false;
    c->ndefg = ndefg; c->nrxg = nrxg;
    c->defg_q.assign(defg_quat, defg_quat + 4 * (size_t)ndefg);
    c->rxg_q.assign(rxg_quat, rxg_quat + 4 * (size_t)nrxg);
    c->rho0.assign(defg_rho0, defg_rho0 + ndefg);
    c->site.assign(rxg_site, rxg_site + nrxg);
    {
        const uint32_t gbx = (c->nx + 1) / 2, gby = (c->ny + 1) / 2, nxy = c->nx * c->ny;
        c->gsite.resize(nrxg);
        for (uint32_t r = 0; r < nrxg; ++r) {
            const uint32_t s = rxg_site[r], z = s / nxy, y = (s - z * nxy) / c->nx, x = s - z * nxy - y * c->nx;
            c->gsite[r] = gindex(gbx, gby, x, y, z);
        }
    }
    c->site_defg.resize(nrxg);
    for (uint32_t r = 0; r < nrxg; ++r) c->site_defg[r] = grid[rxg_site[r]];
    c->tincub.assign(nrxg, 0.0);
    if (rxg_tincub) c->tincub.assign(rxg_tincub, rxg_tincub + nrxg);
    c->rho_order.resize(ndefg);
    for (uint32_t g = 0; g < ndefg; ++g) c->rho_order[g] = g;
    std::stable_sort(c->rho_order.begin(), c->rho_order.end(), [&](uint32_t x, uint32_t y) { return c->rho0[x] > c->rho0[y]; });
    c->nuc_order.resize(nrxg);
    for (uint32_t r = 0; r < nrxg; ++r) c->nuc_order[r] = r;
    std::stable_sort(c->nuc_order.begin(), c->nuc_order.end(), [&](uint32_t x, uint32_t y) { return c->tincub[x] < c->tincub[y]; });
    c->user_ptab.clear();
    if (ptable) c->user_ptab.assign(ptable, ptable + (size_t)nrxg * ndefg);
    if (ptable || !reuse) c->ptab_dirty_all = true;  // a later reset without a caller's table clears it all

    const score_params& p = c->prm;
    DomainArgs& a = c->a;
    const size_t ptab_words = (size_t)nrxg * ndefg;
    cudaError_t e = cudaSuccess;
    if (!reuse) {
        a.nx = c->nx; a.ny = c->ny; a.nz = c->nz;
        a.gbx = (c->nx + 1) / 2; a.gby = (c->ny + 1) / 2; a.gbxy = a.gbx * a.gby;
        a.dgbx = make_fastdiv(a.gbx); a.dgbxy = make_fastdiv(a.gbxy);
        a.ncells = (uint32_t)c->ncells;
        a.ndefg = ndefg; a.nrxg = nrxg;
        a.border_ref_cap = 2 * ((c->nx * c->ny) + (c->nx * c->nz) + (c->ny * c->nz));
        a.border_policy = p.border_policy; a.boundary = p.boundary; a.mobility_model = p.mobility_model;
        // capacities: at most N infections ever happen, so N slots per list never overflow
        const uint32_t capI = (uint32_t)N;
        const uint32_t capB = (p.border_policy == SCORE_BORDER_REFERENCE_LIMIT) ? std::min<uint32_t>((uint32_t)N, a.border_ref_cap + 1) : (uint32_t)N;
        // recycle-list caps (ompshar_init_myRXFront{Inside,Border}, SCORE_Kernel.cpp:3615, 3670)
        const uint32_t recI = (uint32_t)(p.initial_cache * (double)N * p.maxfillperstep * kFullRecyclingFactor);
        const uint32_t recB = (uint32_t)((double)a.border_ref_cap * p.maxfillperstep * kFullRecyclingFactor);
        const uint32_t caps[2] = {capI, capB}, recs[2] = {recI, recB};
        const size_t fb = c->fp32 ? 4 : 8;
        for (int L = 0; L < 2; ++L) {
            DFront& f = a.f[L];
            f.cap = caps[L]; f.reccap = recs[L];
            if (e == cudaSuccess) e = cudaMalloc(&f.fill, (size_t)caps[L] * fb);
            if (e == cudaSuccess && c->fp32) e = cudaMalloc((void**)&f.comp, (size_t)caps[L] * 4);
            if (e == cudaSuccess) e = cudaMalloc(&f.vel, (size_t)caps[L] * fb);
            if (e == cudaSuccess && !c->fp32) e = dalloc(&f.inc, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.mob, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.defg, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.rxg, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.xyz, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.dir, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.full, caps[L]);
            if (e == cudaSuccess) e = dalloc(&f.recyc, recs[L]);
            // sized for the smallest grow tile (kBlock * 4 slots) and the largest (kBlock * 16)
            const size_t tiles = (size_t)caps[L] / (kBlock * 4) + 2;
            const size_t words = (size_t)caps[L] / 32 + 2 * GrowShape<16>::kWords;
            c->scnt_words[L] = 2 * (tiles / kSuper + 2);
            if (e == cudaSuccess) e = dalloc(&f.fmask, words);
            if (e == cudaSuccess) e = dalloc(&f.imask, words);
            if (e == cudaSuccess) e = dalloc(&f.tcnt, 2 * tiles * kWarps);
            if (e == cudaSuccess) e = dalloc(&f.scnt, c->scnt_words[L]);
        }
        c->csct_words = 2 * ((N / kBlock + 2) / kSuper + 2);
        a.misscap = (uint32_t)std::min<uint64_t>(N, 1ull << 25);
        if (e == cudaSuccess) e = dalloc(&a.grid, c->ncells);
        if (e == cudaSuccess) e = dalloc(&c->d_grid_init, c->ncells);
        if (e == cudaSuccess) e = dalloc(&a.claim, c->ncells);
        if (e == cudaSuccess) e = dalloc(&a.amask, N);
        if (e == cudaSuccess) e = dalloc(&a.tobm, N);
        if (e == cudaSuccess) e = dalloc(&a.fcell, N);
        if (e == cudaSuccess) e = dalloc(&a.ctcnt, 2 * (N / kBlock + 2));
        if (e == cudaSuccess) e = dalloc(&a.csct, c->csct_words);
        if (e == cudaSuccess) e = dalloc(&a.ptab, ptab_words);
        if (e == cudaSuccess) e = dalloc(&a.defg_cnt, ndefg);
        if (e == cudaSuccess) e = dalloc(&c->d_defg_cnt_init, ndefg);
        if (e == cudaSuccess) e = dalloc(&a.rxg_cnt, nrxg);
        if (e == cudaSuccess) e = dalloc(&a.depleted, ndefg);
        if (e == cudaSuccess) e = dalloc(&a.miss, a.misscap);
        // a restart clears the listed entries up to 1/64 of the table, else all of it: no more than that is listed, and no more
        // than 8 MB (a 512^3 run lists 0.3 M entries)
        a.touchcap = (uint32_t)std::min<uint64_t>({a.misscap, ptab_words / 64 + 1, 1ull << 20});
        if (e == cudaSuccess) e = dalloc(&a.touched, a.touchcap);
        if (e == cudaSuccess) e = dalloc((float4**)&a.rxq, nrxg);
        if (e == cudaSuccess) e = dalloc((float4**)&a.dfq, ndefg);
        if (e == cudaSuccess) e = dalloc(&c->d_state, 1);
        if (e == cudaSuccess) e = dalloc(&a.fuse, 1);
        if (e == cudaSuccess) e = dalloc(&c->d_pforce, ndefg);
        if (e == cudaSuccess) e = cudaMallocHost((void**)&c->h_pforce, std::max<size_t>(ndefg, 1) * 16);
        if (e == cudaSuccess) e = cudaMallocHost((void**)&c->h_due, kDueMax * sizeof(NucDue));
        if (e == cudaSuccess) e = dalloc(&c->d_due, kDueMax);
        if (e == cudaSuccess) e = dalloc(&c->d_u32tmp, 64);
        // at most one grain-evolution snapshot per logpoint
        c->log_cap = std::min<uint32_t>(p.n_logpoints, SCORE_MAX_TABLE);
        if (e == cudaSuccess && c->log_cap) e = dalloc(&c->d_log_counts, (size_t)c->log_cap * (ndefg + nrxg));
        if (e == cudaSuccess && c->log_cap) e = dalloc(&c->d_log_area, (size_t)c->log_cap * 2 * c->nz);
        if (e != cudaSuccess) { c->release_domain(); return c->fail(SCORE_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e)); }
        a.pforce = c->d_pforce;
        a.st = c->d_state;
        a.box = c->d_box;
        c->high_water[0] = a.f[0].cap; c->high_water[1] = a.f[1].cap;  // the reset clears every slot once
    } else {
        c->high_water[0] = std::max(c->high_water[0], c->next_never[0]);
        c->high_water[1] = std::max(c->high_water[1], c->next_never[1]);
    }
    {   // orientations in FP32 for the classification of new pairs (none where the caller gave every weight)
        std::vector<float> q(4 * ((size_t)nrxg + ndefg));
        for (size_t i = 0; i < 4 * (size_t)nrxg; ++i) q[i] = (float)rxg_quat[i];
        for (size_t i = 0; i < 4 * (size_t)ndefg; ++i) q[4 * (size_t)nrxg + i] = (float)defg_quat[i];
        if (nrxg) e = cudaMemcpyAsync((void*)a.rxq, q.data(), (size_t)nrxg * 16, cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync((void*)a.dfq, q.data() + 4 * (size_t)nrxg, (size_t)ndefg * 16, cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return c->cuda_fail(e, "load domain");
        a.cls = make_weight_class(p);
    }
    // the linear grid goes through the claim array (reset before the first step) into bricks
    e = cudaMemcpyAsync(a.claim, grid, N * 4, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess && ptable) e = cudaMemcpyAsync(a.ptab, ptable, ptab_words * 8, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_defg_cnt_init, 0, (size_t)ndefg * 4, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_state, 0, sizeof(DevState), c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "load domain");
    // per-grain cell counts (solve_REPLACE_CA_STRUCTURE, SCORE_Kernel.cpp:6394-6400)
    k_brick<<<blocks_for(c->ncells, c->sms, 16), kBlock, 0, c->stream>>>(a, a.claim, c->d_grid_init, c->d_defg_cnt_init);
    c->launches++;
    c->defg_cnt_init_host.assign(ndefg, 0);
    e = cudaMemcpyAsync(c->defg_cnt_init_host.data(), c->d_defg_cnt_init, (size_t)ndefg * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->h_state, c->d_state, sizeof(DevState), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "count grains");
    if (c->h_state->err) return c->fail(SCORE_ERR_ARG, "grid holds ids >= ndefg");
    return reset_state(c);
}

int score_restart(score_ctx* c) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->a.grid || c->ndefg == 0) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    cudaSetDevice(c->device);
    c->high_water[0] = std::max(c->high_water[0], c->next_never[0]);
    c->high_water[1] = std::max(c->high_water[1], c->next_never[1]);
    return reset_state(c);
}

int score_place_nuclei(score_ctx* c, uint32_t* n_placed) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    if (c->failed) return SCORE_ERR_STATE;
    cudaSetDevice(c->device);
    return place_nuclei_upto(c, c->ph.t, n_placed, false);
}

int score_step(score_ctx* c, score_step_stats* out) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    if (c->failed) return SCORE_ERR_STATE;  // a device error left the front lists undefined
    c->running = true;
    std::vector<uint32_t> done(1, 0);
    int s = SCORE_OK;
    while (s == SCORE_OK && done[0] == 0) {  // a launch that is refused, or that its group leaves early, makes no step
        if (c->eng->fused_ok()) {
            s = c->eng->fused_session(2.0, 1, true, done);
        } else {
            s = c->eng->step(c->eng->sample_step());
            done[0] = 1;
        }
    }
    c->running = false;
    if (s != SCORE_OK) { if (c->err.empty()) c->err = c->eng->err; return s; }
    if (out) *out = c->last;
    return SCORE_OK;
}

int score_run_until(score_ctx* c, double x_target, score_step_stats* trace, uint32_t trace_cap, uint32_t* n_steps) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    if (c->failed) return SCORE_ERR_STATE;
    c->trace.clear();
    uint32_t k = 0;
    const int s = c->eng->run_until(x_target, 0, &k);
    if (trace) for (uint32_t i = 0; i < k && i < trace_cap && i < c->trace.size(); ++i) trace[i] = c->trace[i];
    if (n_steps) *n_steps = k;
    if (s != SCORE_OK && c->err.empty()) c->err = c->eng->err;
    return s;
}

int score_get_stats(score_ctx* c, score_step_stats* out) {
    if (!c || !out) return SCORE_ERR_ARG;
    *out = c->last;
    out->step = c->step; out->t = c->ph.t; out->dt = c->ph.dt; out->Xcells = c->Xcells;
    out->X = c->N ? c->Xcells / (double)c->N : 0.0; out->Pmax = c->ph.Pmax;
    return SCORE_OK;
}

int score_export_labels(score_ctx* c, uint32_t* labels) {
    if (!c || !labels) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    cudaSetDevice(c->device);
    uint32_t* d_lab = c->a.amask;  // N words, free between steps
    k_unbrick<<<blocks_for(c->ncells, c->sms, 16), kBlock, 0, c->stream>>>(c->a, c->a.grid, d_lab);
    c->launches++;
    cudaError_t e = cudaGetLastError();
    for (int L = 0; L < 2 && e == cudaSuccess; ++L) {
        const uint32_t n = c->next_never[L];
        if (n == 0) continue;
        if (c->fp32) k_labels_front<true><<<blocks_for(n, c->sms), kBlock, 0, c->stream>>>(c->a, L, n, d_lab);
        else k_labels_front<false><<<blocks_for(n, c->sms), kBlock, 0, c->stream>>>(c->a, L, n, d_lab);
        c->launches++;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(labels, d_lab, c->N * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "export labels");
    return SCORE_OK;
}

int score_grain_counts(score_ctx* c, uint32_t* rxg_counts, uint32_t* defg_counts) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    cudaSetDevice(c->device);
    cudaError_t e = cudaSuccess;
    if (rxg_counts && c->nrxg) e = cudaMemcpyAsync(rxg_counts, c->a.rxg_cnt, (size_t)c->nrxg * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && defg_counts) e = cudaMemcpyAsync(defg_counts, c->a.defg_cnt, (size_t)c->ndefg * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return c->cuda_fail(e, "grain counts");
    return SCORE_OK;
}

int score_grainevo_count(score_ctx* c, uint32_t* n) {
    if (!c || !n) return SCORE_ERR_ARG;
    *n = (uint32_t)c->log_info.size();
    return SCORE_OK;
}

int score_grainevo(score_ctx* c, uint32_t i, score_grainevo_info* info, uint32_t* counts, uint32_t* rxarea) {
    if (!c) return SCORE_ERR_ARG;
    return grainevo_get(c, i, info, counts, rxarea);
}

int score_rediscr_kinetics(score_ctx* c, uint32_t nslots, double* t_out, double* rxvol_out, double* boxvol_out) {
    if (!c) return SCORE_ERR_ARG;
    const int s = rediscr({c}, nslots, nullptr, 0, t_out, rxvol_out, boxvol_out, c->err);
    return s;
}

int score_percolation_analyze(score_ctx* c, int mode, score_perc_result* out, uint32_t* sizes, uint32_t sizes_cap, uint32_t* labels) {
    if (!c) return SCORE_ERR_ARG;
    if (!c->loaded) return c->fail(SCORE_ERR_STATE, "no domain loaded");
    cudaSetDevice(c->device);
    // the full-cell arrays (N words each) are free between steps
    if (!c->stage(percolation_scratch(c->nx, c->ny, c->nz))) return c->fail(SCORE_ERR_NOMEM, "percolation buffers");
    PercBuffers b{};
    b.grid = c->a.grid;
    b.parent = c->a.tobm;
    b.size = c->a.f[0].full;
    b.label = c->a.amask;
    b.compact = c->a.fcell;
    b.scratch = c->d_stage;
    c->launches += 7 + (labels ? 1 : 0);
    return percolation_analyze(b, c->a.gbx, c->a.gby, c->nx, c->ny, c->nz, c->ndefg, mode, c->stream, c->sms, out, sizes, sizes_cap, labels, c->err);
}

int score_get_timing(score_ctx* c, score_timing* out) {
    if (!c || !out) return SCORE_ERR_ARG;
    *out = c->eng->tm;
    out->kernel_launches = c->launches + c->eng->launches;
    return SCORE_OK;
}

int score_get_tune(score_ctx* c, score_tune* out) {
    if (!c || !out) return SCORE_ERR_ARG;
    c->eng->get_tune(out);
    return SCORE_OK;
}

int score_set_tune(score_ctx* c, const score_tune* t) {
    if (!c || !t) return SCORE_ERR_ARG;
    const int s = c->eng->set_tune(t);
    if (s != SCORE_OK) c->err = c->eng->err;
    return s;
}

int score_autotune(score_ctx* c, double x_target, uint32_t max_steps, score_tune* out) {
    if (!c) return SCORE_ERR_ARG;
    int s = score_restart(c);
    if (s == SCORE_OK) s = score_place_nuclei(c, nullptr);
    if (s == SCORE_OK) s = c->eng->autotune(x_target, max_steps, out);
    if (s != SCORE_OK) { if (c->err.empty()) c->err = c->eng->err; return s; }
    s = score_restart(c);
    if (s == SCORE_OK) s = score_place_nuclei(c, nullptr);
    return s;
}

}  // extern "C"

// ------------------------------------------------------------------ batched ensemble
// A batch splits its domains into groups of about equal cell count, each stepped by its own
// engine (stream, argument slots, graphs, workers) from its own host thread: the groups'
// latency-bound kernels overlap on the GPU and their host work overlaps on the CPU.  Within a
// group small fronts step inside one launch, each domain at its own pace (k_steps_fused); larger ones step
// together, one sequence of launches per step.
struct score_batch {
    std::vector<std::unique_ptr<Engine>> engs;
    std::vector<score_ctx*> dom;
    std::string err;
    ~score_batch() {
        for (score_ctx* c : dom) delete c;
        dom.clear();
    }
    int fail(int code, const std::string& m) { err = m; return code; }
    int dom_fail(score_ctx* c, int code) { err = c->err; return code; }
    // f(g) for every group on its own thread (the calling thread takes group 0); first error wins
    template <class F>
    int each_group(F f) {
        const size_t G = engs.size();
        std::vector<int> st(G, SCORE_OK);
        std::vector<std::thread> th;
        for (size_t g = 1; g < G; ++g) th.emplace_back([&, g] { st[g] = f(g); });
        st[0] = f(0);
        for (auto& t : th) t.join();
        for (size_t g = 0; g < G; ++g)
            if (st[g] != SCORE_OK) return fail(st[g], engs[g]->err);
        return SCORE_OK;
    }
};

namespace {
constexpr uint32_t kGroupDomains = 32;  // domains per group (per engine and stream) of a batch
}

extern "C" {

int score_batch_create(score_batch** out, const score_params* params, uint32_t n, int device) {
    if (!out || !params || n == 0 || n > (uint32_t)kMaxDomains) return SCORE_ERR_ARG;
    *out = nullptr;
    for (uint32_t i = 0; i < n; ++i) {
        const int s = check_params(&params[i], device);
        if (s != SCORE_OK) return s;
        if (params[i].precision != params[0].precision) return SCORE_ERR_ARG;  // one precision per batch
    }
    score_batch* b = new score_batch();
    // groups of about equal cell count: largest domain first, to the lightest group
    const uint32_t G = std::max(1u, std::min(n / kGroupDomains, 4u));
    std::vector<uint32_t> order(n), group(n), count(G, 0);
    std::vector<uint64_t> load(G, 0);
    for (uint32_t i = 0; i < n; ++i) order[i] = i;
    auto cells = [&](uint32_t i) { return (uint64_t)params[i].nx * params[i].ny * params[i].nz; };
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return cells(x) > cells(y); });
    for (uint32_t i : order) {
        const uint32_t g = (uint32_t)(std::min_element(load.begin(), load.end()) - load.begin());
        group[i] = g; load[g] += cells(i); ++count[g];
    }
    const unsigned hw = std::max(2u, std::thread::hardware_concurrency());
    for (uint32_t g = 0; g < G; ++g) {
        b->engs.emplace_back(new Engine());
        Engine& E = *b->engs.back();
        const int si = E.init(device, (int)count[g]);
        if (si != SCORE_OK) { delete b; return si; }
        E.fp32 = params[0].precision == SCORE_PRECISION_FP32_KAHAN;
        E.fuse_sms = std::max(1, E.sms / (int)G);  // the groups' launches run side by side
        E.pool_threads = std::max(1u, (hw - 1) / G);
    }
    for (uint32_t i = 0; i < n; ++i) {
        score_ctx* c = nullptr;
        const int s = make_ctx(&params[i], b->engs[group[i]].get(), false, &c);
        if (s != SCORE_OK) { delete b; return s; }
        b->dom.push_back(c);
    }
    *out = b;
    return SCORE_OK;
}

void score_batch_destroy(score_batch* b) { delete b; }

const char* score_batch_last_error(const score_batch* b) { return b ? b->err.c_str() : "null batch"; }

int score_batch_load_domain(score_batch* b, uint32_t d, const uint32_t* grid, const double* defg_quat,
                            const double* defg_rho0, uint32_t ndefg, const double* rxg_quat, const uint32_t* rxg_site,
                            const double* rxg_tincub, uint32_t nrxg, const double* ptable) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const int s = score_load_domain(b->dom[d], grid, defg_quat, defg_rho0, ndefg, rxg_quat, rxg_site, rxg_tincub, nrxg, ptable);
    return s == SCORE_OK ? s : b->dom_fail(b->dom[d], s);
}

int score_batch_restart(score_batch* b) {
    if (!b) return SCORE_ERR_ARG;
    for (score_ctx* c : b->dom) {
        if (!c->a.grid) continue;
        const int s = score_restart(c);
        if (s != SCORE_OK) return b->dom_fail(c, s);
    }
    for (auto& E : b->engs) E->mark_run_start();
    return SCORE_OK;
}

int score_batch_place_nuclei(score_batch* b) {
    if (!b) return SCORE_ERR_ARG;
    for (score_ctx* c : b->dom) {
        if (!c->loaded) continue;
        const int s = score_place_nuclei(c, nullptr);
        if (s != SCORE_OK) return b->dom_fail(c, s);
    }
    return SCORE_OK;
}

int score_batch_run_until(score_batch* b, double x_target, uint32_t max_steps, uint32_t* steps_done) {
    if (!b) return SCORE_ERR_ARG;
    for (score_ctx* c : b->dom) c->trace.clear();
    std::vector<uint32_t> steps(b->engs.size(), 0);
    const int s = b->each_group([&](size_t g) { return b->engs[g]->run_until(x_target, max_steps, &steps[g]); });
    if (steps_done) *steps_done = *std::max_element(steps.begin(), steps.end());
    return s;
}

int score_batch_get_stats(score_batch* b, uint32_t d, score_step_stats* out) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    return score_get_stats(b->dom[d], out);
}

int score_batch_trace(score_batch* b, uint32_t d, score_step_stats* trace, uint32_t cap, uint32_t* n_steps) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const std::vector<score_step_stats>& t = b->dom[d]->trace;
    if (trace) for (uint32_t i = 0; i < cap && i < t.size(); ++i) trace[i] = t[i];
    if (n_steps) *n_steps = (uint32_t)t.size();
    return SCORE_OK;
}

int score_batch_export_labels(score_batch* b, uint32_t d, uint32_t* labels) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const int s = score_export_labels(b->dom[d], labels);
    return s == SCORE_OK ? s : b->dom_fail(b->dom[d], s);
}

int score_batch_grain_counts(score_batch* b, uint32_t d, uint32_t* rxg_counts, uint32_t* defg_counts) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const int s = score_grain_counts(b->dom[d], rxg_counts, defg_counts);
    return s == SCORE_OK ? s : b->dom_fail(b->dom[d], s);
}

int score_batch_grainevo_count(score_batch* b, uint32_t d, uint32_t* n) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    return score_grainevo_count(b->dom[d], n);
}

int score_batch_grainevo(score_batch* b, uint32_t d, uint32_t i, score_grainevo_info* info, uint32_t* counts, uint32_t* rxarea) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const int s = grainevo_get(b->dom[d], i, info, counts, rxarea);
    return s == SCORE_OK ? s : b->dom_fail(b->dom[d], s);
}

int score_batch_rediscr_kinetics(score_batch* b, uint32_t nslots, double* t_out, double* rxvol_out, double* boxvol_out) {
    if (!b) return SCORE_ERR_ARG;
    return rediscr(b->dom, nslots, nullptr, 0, t_out, rxvol_out, boxvol_out, b->err);
}

int score_batch_rediscr_texture(score_batch* b, uint32_t nslots, const uint32_t* grain_class, uint32_t nclass, double* t_out,
                                double* vol_out) {
    if (!b || !grain_class) return SCORE_ERR_ARG;
    size_t n = 0;
    for (score_ctx* c : b->dom) n += (size_t)c->ndefg + c->nrxg;
    for (size_t i = 0; i < n; ++i)
        if (grain_class[i] >= nclass) return b->fail(SCORE_ERR_ARG, "orientation class out of range");
    return rediscr(b->dom, nslots, grain_class, nclass, t_out, vol_out, nullptr, b->err);
}

int score_batch_final_grain_sizes(score_batch* b, uint32_t* rx_cells) {
    if (!b || !rx_cells) return SCORE_ERR_ARG;
    size_t off = 0;
    for (score_ctx* c : b->dom) {
        if (!c->loaded) return b->fail(SCORE_ERR_STATE, "every domain must be loaded");
        cudaSetDevice(c->device);
        cudaError_t e = c->nrxg ? cudaMemcpyAsync(rx_cells + off, c->a.rxg_cnt, (size_t)c->nrxg * 4, cudaMemcpyDeviceToHost, c->stream)
                                : cudaSuccess;
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) return b->fail(SCORE_ERR_CUDA, std::string("final grain sizes: ") + cudaGetErrorString(e));
        off += c->nrxg;
    }
    return SCORE_OK;
}

int score_batch_percolation_analyze(score_batch* b, uint32_t d, int mode, score_perc_result* out, uint32_t* sizes, uint32_t sizes_cap,
                            uint32_t* labels) {
    if (!b || d >= b->dom.size()) return SCORE_ERR_ARG;
    const int s = score_percolation_analyze(b->dom[d], mode, out, sizes, sizes_cap, labels);
    return s == SCORE_OK ? s : b->dom_fail(b->dom[d], s);
}

int score_batch_get_timing(score_batch* b, score_timing* out) {
    if (!b || !out) return SCORE_ERR_ARG;
    // device and host times summed over the groups (they run concurrently), the run span the longest
    *out = score_timing{};
    uint64_t launches = 0;
    for (auto& E : b->engs) {
        const score_timing& t = E->tm;
        out->total_ms += t.total_ms; out->grow_ms += t.grow_ms; out->claim_ms += t.claim_ms; out->commit_ms += t.commit_ms;
        out->host_ms += t.host_ms; out->grow_launches += t.grow_launches; out->grow_bytes += t.grow_bytes;
        out->step_bytes += t.step_bytes; out->fill_ms += t.fill_ms; out->wait_ms += t.wait_ms; out->weights_ms += t.weights_ms;
        out->pre_ms += t.pre_ms; out->post_ms += t.post_ms; out->timed_steps += t.timed_steps;
        out->run_ms = std::max(out->run_ms, t.run_ms);
        launches += E->launches;
    }
    for (score_ctx* c : b->dom) launches += c->launches;
    out->kernel_launches = launches;
    return SCORE_OK;
}

int score_batch_get_tune(score_batch* b, score_tune* out) {
    if (!b || !out) return SCORE_ERR_ARG;
    b->engs[0]->get_tune(out);
    return SCORE_OK;
}

int score_batch_set_tune(score_batch* b, const score_tune* t) {
    if (!b || !t) return SCORE_ERR_ARG;
    for (auto& E : b->engs) {
        const int s = E->set_tune(t);
        if (s != SCORE_OK) return b->fail(s, E->err);
    }
    return SCORE_OK;
}

int score_batch_autotune(score_batch* b, double x_target, uint32_t max_steps, score_tune* out) {
    if (!b) return SCORE_ERR_ARG;
    int s = score_batch_restart(b);
    if (s == SCORE_OK) s = score_batch_place_nuclei(b);
    if (s != SCORE_OK) return s;
    std::vector<score_tune> tunes(b->engs.size());
    s = b->each_group([&](size_t g) { return b->engs[g]->autotune(x_target, max_steps, &tunes[g]); });
    if (s != SCORE_OK) return s;
    if (out) *out = tunes[0];
    s = score_batch_restart(b);
    if (s == SCORE_OK) s = score_batch_place_nuclei(b);
    return s;
}

}  // extern "C"

// Lower limits of a context's or a batch's fused steps, for the tests; not part of the C interface (the header does not
// declare it).  null: the defaults.
namespace {
StepLimits lowered(const StepLimits* l) {
    const StepLimits d;
    if (!l) return d;
    StepLimits r;
    r.host_polls = std::max(1u, std::min(l->host_polls, d.host_polls));
    r.group_polls = std::max(1u, std::min(l->group_polls, d.group_polls));
    r.wide = std::min(l->wide, d.wide);
    r.block_slots = std::min(l->block_slots, d.block_slots);
    r.slots = std::min(l->slots, d.slots);
    r.refuse_after = l->refuse_after;
    r.stage = l->stage;
    return r;
}
}  // namespace

extern "C" int score_internal_step_limits(score_ctx* c, score_batch* b, const StepLimits* l) {
    auto set = [l](Engine& E) {
        E.lim = lowered(l);
        if (l && l->number)
            for (score_ctx* d : E.dom) d->fuse_seq = std::min(l->number, kCmdSeqMask);
    };
    if (c) set(*c->eng);
    if (b) for (auto& E : b->engs) set(*E);
    return c || b ? SCORE_OK : SCORE_ERR_ARG;
}

// ------------------------------------------------------------------ no-allocation table
// Device FP64 mobility-weight table P(rxg, defg) for all pairs, with the grid-wide
// maximum, in a form that allocates no memory: the only scratch is the file-scope
// static device array below, whose address is resolved once per device.
//
// The table is the reference's formula (SCORE_Kernel.cpp:2460-2527: Sebald-Gottstein
// -1 / 0 / cos^2 near 40deg<111>, or the Rollett-Holm sigmoid) evaluated with CUDA's
// FP64 math functions (acos, cos, exp, pow) instead of the host libm, so entries agree
// with score_mobility_weight to a few ulp; pairs whose disorientation lies within a
// few ulp of a class threshold (15 deg, 10 deg from 40deg<111>) can land in the other
// class.  The growth step itself does not use this table: it keeps the host's values.
namespace {

// Static scratch of the entry point: 256 B of header + one word per table row.
//   word 0          blocks of the current launch that have finished.  Cleared on the
//                   stream before every launch (a launch that was cut short could leave
//                   it non-zero), and set back to 0 by the last block of each launch.
//   words 32 .. 32 + blocks - 1   maximum P of each block (FP64 bits), written before read.
constexpr uint32_t kTableMaxRows = 65536;
constexpr uint32_t kTableHeaderWords = 32;
static __device__ __align__(256) unsigned long long g_table_scratch[kTableHeaderWords + kTableMaxRows];  // 512 KiB + 256 B

struct TableArgs {
    int32_t model;                  // SCORE_MOBILITY_*
    double fac, lagb, maxdev, m40[4];
    double rh_cut, rh_trans, rh_expo;
    WeightClass cls;
};

__device__ double d_weight(const DomainArgs& A, const TableArgs& t, const double pr[4], const double qd[4]) {
    // the 24 Grimmer candidates once: their largest |component| gives the disorientation
    // angle and, for the Sebald-Gottstein weight, the candidate whose axis is compared
    // with 40deg<111>
    double c[6][4];
    d_grimmer(A, pr, qd, c);
    int mi = 0;
    double om = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (abs_above(c[i][j], om)) { om = fabs(c[i][j]); mi = i; }
    const double theta = om < (1.0 - 5.0e-16) ? 2.0 * acos(om) : 0.0;
    if (t.model == SCORE_MOBILITY_ROLLETT_HOLM)
        return 1.0 - (t.rh_cut * exp(-1.0 * t.rh_trans * pow(theta / t.lagb, t.rh_expo)));
    if (theta <= t.lagb) return -1.0;
    // disorientation quaternion of the best symmetry candidate, components sorted descending
    double s[4] = {fabs(c[mi][0]), fabs(c[mi][1]), fabs(c[mi][2]), fabs(c[mi][3])};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3 - i; ++k)
            if (s[k] > s[k + 1]) { const double x = s[k]; s[k] = s[k + 1]; s[k + 1] = x; }
    const double qdis[4] = {s[3], s[2], s[1], s[0]};
    const double dev = d_disori(A, qdis, t.m40, nullptr);
    if (dev < t.maxdev) {
        const double cs = cos(0.5 * kPi * dev / t.maxdev);
        return cs * cs;
    }
    return 0.0;
}

// Bound by the FP64 pipe where every pair takes both disorientations in FP64 (3 M pairs: 2,157 us at 1/64
// rate), so FP32 classifies the pairs first (weight_class) and only those it cannot settle, a few per cent,
// go through FP64, gathered into a list so that whole warps of them run together.  A block takes
// kTableRows rows and 256 columns at a time: a column is loaded and rounded to FP32 once for its rows.
// The last block to finish reduces the block maxima.
constexpr uint32_t kTableRows = 8, kTableCols = 256, kTableGridY = 8;

__global__ void __launch_bounds__(kTableCols) k_mobility_table(TableArgs t, const double* __restrict__ rxq, uint32_t nrxg,
                                                               const double* __restrict__ dfq, uint32_t ndefg,
                                                               double* __restrict__ table, double* __restrict__ pmax,
                                                               unsigned long long* scratch, uint32_t per) {
    DomainArgs A{};
    A.pc_fac = t.fac;
    __shared__ double s_max[8];
    __shared__ bool s_last;
    __shared__ float4 s_rx[kTableRows];
    __shared__ uint16_t s_q[kTableRows * kTableCols];  // pairs for FP64: row << 8 | column
    __shared__ uint32_t s_n;
    const uint32_t row0 = blockIdx.x * per, rows = min(per, nrxg - row0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < rows) {
        const double* q = rxq + 4 * (size_t)(row0 + threadIdx.x);
        s_rx[threadIdx.x] = make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    }
    double m = -HUGE_VAL;
    uint32_t seen = 0;  // constants met: bit 0: -1, bit 1: 0, bit 2: 1
    for (uint32_t col0 = blockIdx.y * kTableCols; col0 < ndefg; col0 += gridDim.y * kTableCols) {
        __syncthreads();
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        const uint32_t j = col0 + threadIdx.x;
        if (j < ndefg) {
            const double* q = dfq + 4 * (size_t)j;
            const float4 df = make_float4((float)q[0], (float)q[1], (float)q[2], (float)q[3]);
            for (uint32_t r = 0; r < rows; ++r) {
                const int c = weight_class<true>(t.cls, s_rx[r], df);
                if (c == kWeightUnknown) {
                    s_q[atomicAdd(&s_n, 1u)] = (uint16_t)((r << 8) | threadIdx.x);
                } else {
                    // the double's bits without a conversion on the FP64 pipe
                    const uint32_t hi = c == 0 ? 0u : c < 0 ? 0xBFF00000u : 0x3FF00000u;
                    table[(size_t)(row0 + r) * ndefg + j] = __hiloint2double((int)hi, 0);
                    seen |= 1u << (c + 1);
                }
            }
        }
        __syncthreads();
        const uint32_t n = s_n;
        for (uint32_t k = threadIdx.x; k < n; k += kTableCols) {
            const uint32_t r = s_q[k] >> 8, col = col0 + (s_q[k] & 255u);
            const double* a = rxq + 4 * (size_t)(row0 + r);
            const double* b = dfq + 4 * (size_t)col;
            const double pr[4] = {a[0], a[1], a[2], a[3]}, qd[4] = {b[0], b[1], b[2], b[3]};
            const double P = d_weight(A, t, pr, qd);
            table[(size_t)(row0 + r) * ndefg + col] = P;
            m = fmax(m, P);
        }
    }
    if (seen & 1u) m = fmax(m, -1.0);
    if (seen & 2u) m = fmax(m, 0.0);
    if (seen & 4u) m = fmax(m, 1.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (lane == 0) s_max[warp] = m;
    __syncthreads();
    const uint32_t blocks = gridDim.x * gridDim.y;
    if (threadIdx.x == 0) {
        double bm = s_max[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) bm = fmax(bm, s_max[w]);
        scratch[kTableHeaderWords + blockIdx.y * gridDim.x + blockIdx.x] = (unsigned long long)__double_as_longlong(bm);
        __threadfence();
        const unsigned long long done = atomicAdd(&scratch[0], 1ull);
        s_last = (done == (unsigned long long)blocks - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double g = -HUGE_VAL;
    for (uint32_t r = threadIdx.x; r < blocks; r += blockDim.x)
        g = fmax(g, __longlong_as_double((long long)__ldcg(&scratch[kTableHeaderWords + r])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g = fmax(g, __shfl_xor_sync(0xFFFFFFFFu, g, o));
    if (lane == 0) s_max[warp] = g;
    __syncthreads();
    if (threadIdx.x == 0) {
        double bm = s_max[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) bm = fmax(bm, s_max[w]);
        *pmax = bm;
        scratch[0] = 0ull;  // ready for the next launch
    }
}
static_assert(((kTableMaxRows + kTableRows - 1) / kTableRows) * kTableGridY <= kTableMaxRows, "a scratch word a block");

// scratch address per device ordinal, resolved once with that device current
constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
unsigned long long* g_scratch_of[kMaxDevices] = {};

int table_scratch(int device, unsigned long long** out) {
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_scratch_of[device]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_table_scratch);
        if (e != cudaSuccess || !p) return SCORE_ERR_CUDA;
        g_scratch_of[device] = (unsigned long long*)p;
    }
    *out = g_scratch_of[device];
    return SCORE_OK;
}

}  // namespace

extern "C" int score_mobility_table_noalloc(const score_params* p, const double* d_rxg_quat, uint32_t nrxg,
                                            const double* d_defg_quat, uint32_t ndefg, double* d_table,
                                            double* d_pmax, void* stream) {
    if (!p || !d_rxg_quat || !d_defg_quat || !d_table || !d_pmax || nrxg == 0 || ndefg == 0) return SCORE_ERR_ARG;
    if (nrxg > kTableMaxRows) return SCORE_ERR_SCRATCH_LIMIT;
    if (p->mobility_model != SCORE_MOBILITY_SEBALD_GOTTSTEIN && p->mobility_model != SCORE_MOBILITY_ROLLETT_HOLM)
        return SCORE_ERR_ARG;
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0) return SCORE_ERR_NOT_BUILT;
    if (device >= kMaxDevices) return SCORE_ERR_ARG;
    unsigned long long* scratch = nullptr;
    const int s = table_scratch(device, &scratch);
    if (s != SCORE_OK) return s;
    TableArgs t{};
    t.model = p->mobility_model;
    double theta_sat = 0.0;
    weight_constants(*p, &t.fac, &t.lagb, &t.maxdev, t.m40, &theta_sat);
    t.rh_cut = p->RH_cut;
    t.rh_trans = p->RH_trans;
    t.rh_expo = p->RH_exponent;
    t.cls = make_weight_class(*p);
    cudaStream_t st = (cudaStream_t)stream;
    // the completion counter starts at 0 whatever an earlier launch left behind
    if (cudaMemsetAsync(scratch, 0, sizeof(unsigned long long), st) != cudaSuccess) return SCORE_ERR_CUDA;
    // rows a block: as many as leave the SMs two blocks each, so that a small table's chains run side by side
    // (75 x 128 pairs: 22 us with one row a block, 28 with eight; 2000 x 1500: 154 us with eight)
    const uint32_t gy = std::min((ndefg + kTableCols - 1) / kTableCols, kTableGridY);
    const uint32_t per = (uint32_t)std::min<uint64_t>(kTableRows, std::max<uint64_t>({1, (uint64_t)nrxg * gy / 304, (nrxg * gy + kTableMaxRows - 1) / kTableMaxRows}));
    // the launch's own status (not cudaGetLastError, which would also report, and clear,
    // an error left behind by the caller's earlier work)
    void* args[] = {(void*)&t, (void*)&d_rxg_quat, (void*)&nrxg, (void*)&d_defg_quat, (void*)&ndefg, (void*)&d_table,
                    (void*)&d_pmax, (void*)&scratch, (void*)&per};
    const dim3 grid((nrxg + per - 1) / per, gy);
    const cudaError_t e = cudaLaunchKernel((const void*)k_mobility_table, grid, dim3(kTableCols), args, 0, st);
    return e == cudaSuccess ? SCORE_OK : SCORE_ERR_CUDA;
}
