// One launch for many growth steps of domains whose fronts are too small to fill the GPU.
//
// What bounds such a domain is neither bytes nor operations but the chain of a step: five or six
// launches, each with its own start, constant-cache misses and dependent loads, then a stream
// synchronization and the host's master block (64^3 domain, front of 30 k slots: 51 us a step, of which the
// bytes take 0.1; 128^3: 59 us; here 24 and 28).  A group of blocks steps one domain inside one
// cooperative launch:
//   A  fill of the group's tiles, 2 or 4 consecutive slots a thread; full cells into records; the 26 infection
//      attempts of every full cell, four lanes a cell.  The attempt ordinal is 26 s + d with s the
//      full cell's slot (Border slots after the Inside ones) instead of its rank among the full cells:
//      the same order, and no list has to exist before the claims;
//   -- group barrier --
//   B  recycle list (only as far as this step can use it); attempts whose claim holds their ordinal won;
//   -- group barrier --
//   C  new cells ranked over the group's tiles in slot order take recycled, then new slots;
//   -- group barrier --
//   D  the group's first block posts the step to the domain's mailbox; the host runs its master block
//      (time, mobilities, weights it was asked for, dt) and answers with one word, so that a step costs a
//      round trip over the host link and not a launch and a synchronization.
// Every wait is bounded: a block that waits too long for its group sets an error and returns; a first
// block that hears nothing from the host for a while leaves with its group, and the host launches again
// from the posted state.  The groups of a batch share nothing but the launch.
#pragma once
#include "growth_kernels.cuh"

namespace score {

constexpr int kFuse = 1024;                               // threads per block, one block per SM
// 1,024 threads of 64 registers: 512 of 110 took 10 % more on the 64^3 domain and 24 % on a recovering 384^3 one
constexpr int kFuseWarps = kFuse / 32;
// slots per tile: ITEMS per thread
template <int ITEMS>
struct FuseShape {
    static constexpr uint32_t kTile = kFuse * ITEMS;
    static constexpr uint32_t kWords = kTile / 32;
    static_assert(kWords == 32 * ITEMS && kFuseWarps == 32, "a word of a tile per warp and item");
};
constexpr uint32_t kFuseMaxTiles = 4096;                  // tiles of a domain (both lists)
constexpr uint32_t kFuseMaxLocal = 512;                   // tiles of one block
constexpr uint32_t kFuseRec = 2048;                       // full cells of a block and step kept in shared memory
constexpr uint32_t kFuseMask = 2048;                      // mask words of a block kept in shared memory
constexpr uint32_t kFuseWins = 4096;                      // new cells listed at a time
constexpr uint32_t kFuseSpin = 1u << 22;                  // polls of a group wait before it gives up (seconds), at most
constexpr uint32_t kFuseHostSpin = 1u << 12;              // polls of the host's answer before the group leaves (milliseconds), at most

// the host's word: step number (equality is all that counts) and flags
constexpr uint32_t kCmdLeave = 1u;        // no further step in this launch
constexpr uint32_t kCmdLast = 2u;         // leave after this step without asking again
constexpr uint32_t kCmdDtChanged = 4u;
constexpr uint32_t kCmdSpec = 8u;
constexpr uint32_t kCmdRefresh1 = 16u;
constexpr uint32_t kCmdRefresh2 = 32u;
constexpr uint32_t kCmdPayload = 64u;     // the payload changed
constexpr uint32_t kCmdForce = 128u;      // new driving forces in payload.pf_src
constexpr uint32_t kCmdReplay = 1u << 31; // host only, in place of the step number: a command to give again
constexpr uint32_t kCmdShift = 8u;
constexpr uint32_t kCmdSeqMask = 0xFFFFFFu;
// Step numbers run from 1 to kCmdSeqMask and start again: 0, which `post`, `left` and `go` hold when nothing was written, is
// none.
__host__ __device__ __forceinline__ uint32_t fuse_next(uint32_t seq) { return seq == kCmdSeqMask ? 1u : seq + 1u; }

// device memory: one per domain
struct FuseDom {
    uint32_t bar;              // arrivals at the group's barriers of this launch (0 between launches)
    uint32_t pad0[31];
    uint32_t go;               // the host's word, passed on by the group's first block
    uint32_t pad1[31];
    FusePay pay;
};

struct FuseMap {
    uint16_t first[kMaxDomains + 1];   // blocks [first[i], first[i + 1]) step domain i
    uint32_t ndom;
    uint32_t group_polls, host_polls;  // limits of the waits
    uint32_t seq[kMaxDomains];         // step number of domain i's first command in this launch
};

// polls are relaxed loads; one fence after the last of them orders what follows (an acquire per poll would
// drop the SM's L1 each time)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void fence_sys() { asm volatile("fence.acq_rel.sys;" ::: "memory"); }
__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_sys(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_sys(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t now_ns() {
    uint32_t v;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(v));
    return v;
}

struct FuseShared {
    DomainArgs a;
    uint32_t rec_key[kFuseRec];        // slot | list << 31
    uint32_t rec_cell[kFuseRec];
    uint32_t rec_win[kFuseRec];        // attempts made, then attempts won
    uint32_t rec_tob[kFuseRec];        // won attempts that go to the Border list
    uint16_t rec_lt[kFuseRec];         // the record's tile among the block's
    uint32_t fm[kFuseMask], im[kFuseMask];         // full and INACTIVE masks of the block's tiles while they fit
    uint16_t wl[kFuseWins];            // new cells of a chunk of records: record in the chunk << 5 | direction
    uint32_t c_win[kFuse], c_tob[kFuse], c_rA[kFuse], c_rB[kFuse], c_cell[kFuse], c_rs[kFuse];
    double c_over[kFuse];
    uint32_t tw[2][kFuseMaxLocal];     // wins of the block's tiles per destination list
    uint32_t pre[2][kFuseMaxLocal];    // prefix of the domain's counts at the block's tiles
    uint32_t off[kFuseMaxLocal + 1];   // first record of each of the block's tiles
    uint32_t w1[kFuseWarps], w2[kFuseWarps];
    uint32_t t0[2], tot[2];            // counts before the Border list's tiles, and in all
    uint32_t dir[26];                  // dir_word of the directions
    uint32_t word, ok;
};

// Arrival of the block at its group's barrier and, with `wait`, the wait for the whole group.  target: arrivals
// of the launch so far when everyone is there.  False (for the whole block) when the wait gave up.
__device__ __forceinline__ bool group_barrier(FuseShared& sh, uint32_t* bar, uint32_t G, uint32_t target, uint32_t polls, bool wait) {
    __syncthreads();
    if (G == 1) return true;
    if (threadIdx.x == 0) {
        fence_gpu();   // cumulative: the block's stores, ordered before thread 0 by the block barrier
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        bool ok = !wait;
        for (uint32_t k = 0; !ok && k < polls; ++k) ok = (int32_t)(ld_relaxed_gpu(bar) - target) >= 0;
        fence_gpu();
        sh.ok = ok ? 1u : 0u;
    }
    __syncthreads();
    return sh.ok != 0u;
}

// a wait that gave up: where (1 to 4 the step's barriers, 5 the host's word), the block, and how far it was
__device__ __forceinline__ void fuse_gave_up(DevState* st, uint32_t where, uint32_t rank, uint32_t at) {
    if (atomicCAS(&st->err_info, 0u, (where << 28) | ((rank & 0xFFFu) << 16) | (at & 0xFFFFu)) == 0u) atomicOr(&st->err, kErrTimeout);
}

// Block-wide inclusive scan of (x, y); the block's totals in tx, ty.  The caller's values come back exclusive.
__device__ __forceinline__ void block_scan2(FuseShared& sh, uint32_t& x, uint32_t& y, uint32_t& tx, uint32_t& ty) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t ix = x, iy = y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t p = __shfl_up_sync(0xFFFFFFFFu, ix, o), q = __shfl_up_sync(0xFFFFFFFFu, iy, o);
        if (lane >= o) { ix += p; iy += q; }
    }
    __syncthreads();
    if (lane == 31) { sh.w1[warp] = ix; sh.w2[warp] = iy; }
    __syncthreads();
    uint32_t vx = lane < kFuseWarps ? sh.w1[lane] : 0u, vy = lane < kFuseWarps ? sh.w2[lane] : 0u;
#pragma unroll
    for (int o = 1; o < kFuseWarps; o <<= 1) {
        const uint32_t p = __shfl_up_sync(0xFFFFFFFFu, vx, o), q = __shfl_up_sync(0xFFFFFFFFu, vy, o);
        if (lane >= o) { vx += p; vy += q; }
    }
    tx = __shfl_sync(0xFFFFFFFFu, vx, kFuseWarps - 1);
    ty = __shfl_sync(0xFFFFFFFFu, vy, kFuseWarps - 1);
    const uint32_t bx = __shfl_sync(0xFFFFFFFFu, vx, warp ? warp - 1 : 0), by = __shfl_sync(0xFFFFFFFFu, vy, warp ? warp - 1 : 0);
    x = ix - x + (warp ? bx : 0u);
    y = iy - y + (warp ? by : 0u);
}

// Exclusive prefix of the domain's T count pairs at the block's tiles (sh.pre), the prefix at tile T0 (sh.t0)
// and the totals (sh.tot).
__device__ __forceinline__ void tile_scan(FuseShared& sh, const uint2* cnt, uint32_t T, uint32_t T0, uint32_t rank, uint32_t G) {
    const uint32_t per = (T + kFuse - 1) / kFuse;   // at most kFuseMaxTiles / kFuse
    const uint32_t lo = threadIdx.x * per;
    uint2 v[kFuseMaxTiles / kFuse];
    uint32_t x = 0, y = 0;
#pragma unroll
    for (uint32_t j = 0; j < kFuseMaxTiles / kFuse; ++j) {
        v[j] = make_uint2(0u, 0u);
        if (j < per && lo + j < T) v[j] = __ldcg(&cnt[lo + j]);
        x += v[j].x; y += v[j].y;
    }
    uint32_t tx, ty;
    block_scan2(sh, x, y, tx, ty);
#pragma unroll
    for (uint32_t j = 0; j < kFuseMaxTiles / kFuse; ++j) {
        const uint32_t u = lo + j;
        if (j < per && u < T) {
            if (u >= rank && (u - rank) % G == 0) { sh.pre[0][(u - rank) / G] = x; sh.pre[1][(u - rank) / G] = y; }
            if (u == T0) { sh.t0[0] = x; sh.t0[1] = y; }
        }
        x += v[j].x; y += v[j].y;
    }
    if (threadIdx.x == 0) {
        sh.tot[0] = tx; sh.tot[1] = ty;
        if (T0 >= T) { sh.t0[0] = tx; sh.t0[1] = ty; }
    }
    __syncthreads();
}

// overshoot of a full cell, for the cells it infects
template <bool FP32>
__device__ __forceinline__ double full_over(const DFront& fr, uint32_t slot) {
    if (!FP32) return __dsub_rn(((const double*)fr.fill)[slot], 1.0);
    return (double)((((const float*)fr.fill)[slot] - 1.0f) - fr.comp[slot]);
}

// The records of a block's full cells: the first kFuseRec in shared memory, the rest in the domain's per-full-cell
// arrays at the full cell's own slot position (a position no other full cell has; n0 + n1 slots never exceed the
// arrays' N words, as every slot stands for a cell infected once).  `pos` is looked up from the tile offsets.
template <int ITEMS>
struct FuseRecs {
    static constexpr uint32_t kTile = FuseShape<ITEMS>::kTile;
    FuseShared& sh;
    uint32_t rank, G, T0, n0, nlt;
    __device__ __forceinline__ uint32_t pos(uint32_t i) const {
        uint32_t lt = nlt - 1;
        while (sh.off[lt] > i) --lt;
        const uint32_t u = rank + lt * G;
        return (u >= T0 ? n0 + (u - T0) * kTile : u * kTile) + (i - sh.off[lt]);
    }
    __device__ __forceinline__ uint32_t key(uint32_t i) const { return i < kFuseRec ? sh.rec_key[i] : sh.a.f[0].full[pos(i)]; }
    __device__ __forceinline__ uint32_t cell(uint32_t i) const { return i < kFuseRec ? sh.rec_cell[i] : sh.a.fcell[pos(i)]; }
    __device__ __forceinline__ uint32_t win(uint32_t i) const { return i < kFuseRec ? sh.rec_win[i] : sh.a.amask[pos(i)]; }
    __device__ __forceinline__ uint32_t tob(uint32_t i) const { return i < kFuseRec ? sh.rec_tob[i] : sh.a.tobm[pos(i)]; }
    __device__ __forceinline__ void set_key(uint32_t i, uint32_t v) const { if (i < kFuseRec) sh.rec_key[i] = v; else sh.a.f[0].full[pos(i)] = v; }
    __device__ __forceinline__ void set_cell(uint32_t i, uint32_t v) const { if (i < kFuseRec) sh.rec_cell[i] = v; else sh.a.fcell[pos(i)] = v; }
    __device__ __forceinline__ void set_win(uint32_t i, uint32_t v) const { if (i < kFuseRec) sh.rec_win[i] = v; else sh.a.amask[pos(i)] = v; }
    __device__ __forceinline__ void set_tob(uint32_t i, uint32_t v) const { if (i < kFuseRec) sh.rec_tob[i] = v; else sh.a.tobm[pos(i)] = v; }
    // local tile of record i with key k
    __device__ __forceinline__ uint32_t tile(uint32_t i, uint32_t k) const {
        if (i < kFuseRec) return sh.rec_lt[i];
        const uint32_t tl = (k & 0x7FFFFFFFu) / kTile;
        return ((k >> 31 ? T0 + tl : tl) - rank) / G;
    }
};

// V consecutive values as one access (4 or 2 of 1, 4 or 8 bytes; 32 bytes as two)
template <int V> struct Vec;
template <> struct Vec<2> {
    static __device__ __forceinline__ uint32_t bytes(const uint8_t* p) { return *(const uint16_t*)p | 0xFFFF0000u; }
    static __device__ __forceinline__ void load(const double* p, double (&v)[2]) { const double2 x = *(const double2*)p; v[0] = x.x; v[1] = x.y; }
    static __device__ __forceinline__ void load(const float* p, float (&v)[2]) { const float2 x = *(const float2*)p; v[0] = x.x; v[1] = x.y; }
    static __device__ __forceinline__ void load(const uint32_t* p, uint32_t (&v)[2]) { const uint2 x = *(const uint2*)p; v[0] = x.x; v[1] = x.y; }
    static __device__ __forceinline__ void store(double* p, const double (&v)[2]) { *(double2*)p = make_double2(v[0], v[1]); }
    static __device__ __forceinline__ void store(float* p, const float (&v)[2]) { *(float2*)p = make_float2(v[0], v[1]); }
};
template <> struct Vec<4> {
    static __device__ __forceinline__ uint32_t bytes(const uint8_t* p) { return *(const uint32_t*)p; }
    static __device__ __forceinline__ void load(const double* p, double (&v)[4]) {
        const double2 x = *(const double2*)p, y = *(const double2*)(p + 2);
        v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
    }
    static __device__ __forceinline__ void load(const float* p, float (&v)[4]) { const float4 x = *(const float4*)p; v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
    static __device__ __forceinline__ void load(const uint32_t* p, uint32_t (&v)[4]) { const uint4 x = *(const uint4*)p; v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
    static __device__ __forceinline__ void store(double* p, const double (&v)[4]) { *(double2*)p = make_double2(v[0], v[1]); *(double2*)(p + 2) = make_double2(v[2], v[3]); }
    static __device__ __forceinline__ void store(float* p, const float (&v)[4]) { *(float4*)p = make_float4(v[0], v[1], v[2], v[3]); }
};

// infector bytes of slots s .. s + V - 1 of a list of n slots (INACTIVE past the list)
template <int V>
__device__ __forceinline__ uint32_t fuse_dirs(const DFront& fr, uint32_t s, uint32_t n) {
    if (s + V <= n) return Vec<V>::bytes(fr.dir + s);
    uint32_t w = 0xFFFFFFFFu;
    for (uint32_t k = 0; s + k < n; ++k) w = (w & ~(0xFFu << (8 * k))) | ((uint32_t)fr.dir[s + k] << (8 * k));
    return w;
}

// The fill update of V consecutive slots with infector bytes dw, the arithmetic of grow_items.  V slots are one
// access a field (slot V-aligned, arrays 256-byte aligned): whole sectors move in FP64 whether one of four
// slots is ACTIVE or all, so a hole costs nothing but its byte unless the four are mixed, and the fields of
// INACTIVE slots among them are written back as they were read (increments, velocities and mobilities of an
// INACTIVE slot mean nothing).  act / full: bit k for slot s + k.
template <bool FP32, int V>
__device__ __forceinline__ void fuse_grow(const DomainArgs& a, const DFront& fr, uint32_t s, uint32_t dw, uint32_t& act, uint32_t& full) {
    act = 0; full = 0;
#pragma unroll
    for (int k = 0; k < V; ++k)
        if (((dw >> (8 * k)) & 0xFFu) != kInactive) act |= 1u << k;
    if (!act) return;
    const bool whole = s + V <= fr.cap;  // else the last slots of the list's arrays, one by one
    using X = Vec<V>;
    if (!FP32) {
        double w[V], fill[V];
        double* const pf = (double*)fr.fill + s;
        double* const pv = (double*)fr.vel + s;
        double* const pi = fr.inc + s;
        if (whole) X::load((const double*)pf, fill);
        else
#pragma unroll
            for (int k = 0; k < V; ++k) fill[k] = (act >> k) & 1u ? pf[k] : 0.0;
        const bool dtc = a.dt_changed != 0;
        if (a.refresh == 0) {
            const double* src = dtc ? pv : pi;
            if (whole) X::load(src, w);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) w[k] = (act >> k) & 1u ? src[k] : -1.0;
#pragma unroll
            for (int k = 0; k < V; ++k) {  // nuclei, cells answered by the host: no increment yet
                const uint8_t d = (uint8_t)(dw >> (8 * k));
                if (!((act >> k) & 1u) || !(d & kStale)) continue;
                if (d & kPend) {
                    w[k] = answered_velocity(a, fr, s + k, d, ((const unsigned long long*)fr.vel)[s + k]);
                    pv[k] = w[k];
                } else if (!dtc) {
                    w[k] = pv[k];
                }
            }
        } else {
            double mo[V];
            uint32_t g[V];
            if (whole) X::load((const uint32_t*)fr.defg + s, g);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) g[k] = (act >> k) & 1u ? fr.defg[s + k] : 0u;
            if (a.refresh == 2) {
                if (whole) X::load((const double*)fr.mob + s, mo);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) mo[k] = (act >> k) & 1u ? fr.mob[s + k] : 0.0;
            } else {
                uint32_t r[V];
                if (whole) X::load((const uint32_t*)fr.rxg + s, r);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) r[k] = (act >> k) & 1u ? fr.rxg[s + k] : 0u;
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    mo[k] = 0.0;
                    if (((act >> k) & 1u) && !((dw >> (8 * k)) & kPend))
                        mo[k] = mobility(a, __longlong_as_double((long long)a.ptab[(unsigned long long)r[k] * a.ndefg + g[k]]));
                }
                if (whole) X::store(fr.mob + s, mo);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) if ((act >> k) & 1u) fr.mob[s + k] = mo[k];
            }
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const uint8_t d = (uint8_t)(dw >> (8 * k));
                w[k] = -1.0;
                if (!((act >> k) & 1u)) continue;
                if (d & kPend) w[k] = answered_velocity(a, fr, s + k, d, ((const unsigned long long*)fr.vel)[s + k]);
                else w[k] = velocity_from_mobility(a, mo[k], g[k], d & kCodeMask);
            }
            if (whole) X::store(pv, w);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) if ((act >> k) & 1u) pv[k] = w[k];
        }
        const bool fresh = dtc || a.refresh != 0;  // every increment is new
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const uint8_t d = (uint8_t)(dw >> (8 * k));
            if (!((act >> k) & 1u)) { w[k] = -1.0; continue; }
            if (fresh || (d & kStale)) {
                if (__double_as_longlong(w[k]) >= 0) w[k] = __dmul_rn(__dmul_rn(w[k], a.dt), a.cinv);
                if (!fresh) pi[k] = w[k];
                if (d & kStale) fr.dir[s + k] = d & kCodeMask;
            }
        }
        if (fresh) {
            if (whole) X::store(pi, w);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) if ((act >> k) & 1u) pi[k] = w[k];
        }
        uint32_t moved = 0;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            if (__double_as_longlong(w[k]) < 0) continue;  // INACTIVE, or no driving force
            fill[k] = __dadd_rn(fill[k], w[k]);
            moved |= 1u << k;
            if (__double_as_longlong(fill[k]) >= 0x3FF0000000000000ll) full |= 1u << k;  // f >= 1.0, never negative
        }
        if (whole) { if (moved) X::store(pf, fill); }
        else
#pragma unroll
            for (int k = 0; k < V; ++k) if ((moved >> k) & 1u) pf[k] = fill[k];
    } else {
        float vel[V], fill[V], comp[V];
        float* const pf = (float*)fr.fill + s;
        float* const pv = (float*)fr.vel + s;
        float* const pc = fr.comp + s;
        if (whole) { X::load((const float*)pf, fill); X::load((const float*)pc, comp); }
        else
#pragma unroll
            for (int k = 0; k < V; ++k) { fill[k] = (act >> k) & 1u ? pf[k] : 0.0f; comp[k] = (act >> k) & 1u ? pc[k] : 0.0f; }
        if (a.refresh == 0) {
            if (whole) X::load((const float*)pv, vel);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) vel[k] = (act >> k) & 1u ? pv[k] : -1.0f;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const uint8_t d = (uint8_t)(dw >> (8 * k));
                if (!((act >> k) & 1u) || !(d & kPend)) continue;
                vel[k] = (float)answered_velocity(a, fr, s + k, d, ((const uint32_t*)fr.vel)[s + k]);
                pv[k] = vel[k];
            }
        } else {
            double mo[V];
            uint32_t g[V];
            if (whole) X::load((const uint32_t*)fr.defg + s, g);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) g[k] = (act >> k) & 1u ? fr.defg[s + k] : 0u;
            if (a.refresh == 2) {
                if (whole) X::load((const double*)fr.mob + s, mo);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) mo[k] = (act >> k) & 1u ? fr.mob[s + k] : 0.0;
            } else {
                uint32_t r[V];
                if (whole) X::load((const uint32_t*)fr.rxg + s, r);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) r[k] = (act >> k) & 1u ? fr.rxg[s + k] : 0u;
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    mo[k] = 0.0;
                    if (((act >> k) & 1u) && !((dw >> (8 * k)) & kPend))
                        mo[k] = mobility(a, __longlong_as_double((long long)a.ptab[(unsigned long long)r[k] * a.ndefg + g[k]]));
                }
                if (whole) X::store(fr.mob + s, mo);
                else
#pragma unroll
                    for (int k = 0; k < V; ++k) if ((act >> k) & 1u) fr.mob[s + k] = mo[k];
            }
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const uint8_t d = (uint8_t)(dw >> (8 * k));
                vel[k] = -1.0f;
                if (!((act >> k) & 1u)) continue;
                if (d & kPend) vel[k] = (float)answered_velocity(a, fr, s + k, d, ((const uint32_t*)fr.vel)[s + k]);
                else vel[k] = velocity32_from_mobility(a, mo[k], g[k], d & kCodeMask);
            }
            if (whole) X::store(pv, vel);
            else
#pragma unroll
                for (int k = 0; k < V; ++k) if ((act >> k) & 1u) pv[k] = vel[k];
        }
        uint32_t moved = 0;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const uint8_t d = (uint8_t)(dw >> (8 * k));
            if (!((act >> k) & 1u)) continue;
            if (d & kStale) fr.dir[s + k] = d & kCodeMask;
            if (vel[k] >= 0.0f) {
                // Kahan-compensated accumulation of the fill
                const float inc = vel[k] * a.dtc32;
                const float y = inc - comp[k];
                const float t = fill[k] + y;
                const float c = (t - fill[k]) - y;
                fill[k] = t; comp[k] = c;
                moved |= 1u << k;
                if ((t - c) >= 1.0f) full |= 1u << k;
            }
        }
        if (whole) { if (moved) { X::store(pf, fill); X::store(pc, comp); } }
        else
#pragma unroll
            for (int k = 0; k < V; ++k) if ((moved >> k) & 1u) { pf[k] = fill[k]; pc[k] = comp[k]; }
    }
}

// What a full cell leaves behind: its grains, its overshoot, and the cells of its deformed grain before (gold) this warp's
// gk of them went, for the lane that counted them.  Makes the cell recrystallized: grid, slot, cell counts.
struct FullCell {
    uint32_t rs, gs, gk, gold;
    double over;
};
template <bool FP32, class Recs>
__device__ __forceinline__ void take_full(const DomainArgs& cst, const DomainArgs& a, const Recs& rec, uint32_t i, uint32_t F, FullCell& c) {
    c.rs = 0; c.gs = 0; c.gk = 0; c.gold = 0; c.over = 0.0;
    if (i < F) {
        const uint32_t key = rec.key(i), slot = key & 0x7FFFFFFFu;
        const DFront& fr = a.f[key >> 31];
        c.rs = fr.rxg[slot];
        c.gs = fr.defg[slot];
        c.over = full_over<FP32>(fr, slot);
        cst.grid[rec.cell(i)] = cst.ndefg + c.rs;
        fr.dir[slot] = kInactive;
        if (!FP32) ((double*)fr.fill)[slot] = 0.0;
        else { ((float*)fr.fill)[slot] = 0.0f; fr.comp[slot] = 0.0f; }
    }
    count_full(cst, i < F, c.rs, c.gs, c.gk, c.gold);
}

template <bool FP32, int ITEMS>
__global__ void __launch_bounds__(kFuse, 1) k_steps_fused(const __grid_constant__ FuseMap map, int base) {
    extern __shared__ __align__(16) char s_raw[];
    FuseShared& sh = *reinterpret_cast<FuseShared*>(s_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int dom = 0;
    while ((uint32_t)dom + 1 < map.ndom && blockIdx.x >= map.first[dom + 1]) ++dom;
    const uint32_t rank = blockIdx.x - map.first[dom], G = map.first[dom + 1] - map.first[dom];
    for (uint32_t i = threadIdx.x; i < sizeof(DomainArgs) / 4; i += kFuse)
        ((uint32_t*)&sh.a)[i] = ((const uint32_t*)&c_args[base + dom])[i];
    __syncthreads();
    const DomainArgs& a = sh.a;                  // with what changes between steps
    const DomainArgs& cst = c_args[base + dom];   // the rest, by the constant cache: uniform registers, no shared loads
    if (!cst.active) return;
    constexpr uint32_t kTile = FuseShape<ITEMS>::kTile, kWords = FuseShape<ITEMS>::kWords;
    DevState* const st = a.st;
    FuseDom* const fd = a.fuse;
    FuseHost* const fh = &a.box->fuse;
    const bool first = rank == 0;
    uint32_t n0 = st->next_never[0], n1 = st->next_never[1];
    uint32_t seq = map.seq[dom], arrived = 0;
    if (threadIdx.x < 26)
        sh.dir[threadIdx.x] = c_dir.v[threadIdx.x];
    for (;;) {
        // ---- the host's word for step `seq`
        if (first) {
            if (threadIdx.x == 0) {
                uint32_t w = 0;
                bool ok = false;
                for (uint32_t k = 0; !ok && k < map.host_polls; ++k) {
                    w = ld_relaxed_sys(&fh->cmd);
                    ok = (w >> kCmdShift) == seq;
                }
                fence_sys();
                sh.word = ok ? w : (seq << kCmdShift) | kCmdLeave;
                sh.ok = ok ? 1u : 0u;
            }
            __syncthreads();
            const uint32_t w = sh.word;
            if (w & kCmdPayload) {
                const volatile uint32_t* src = (const volatile uint32_t*)&fh->pay;
                if (threadIdx.x < sizeof(FusePay) / 4) ((uint32_t*)&fd->pay)[threadIdx.x] = src[threadIdx.x];
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                if (w & kCmdLeave) fd->bar = 0u;  // everyone has arrived at the last barrier
                fence_gpu();
                st_relaxed_gpu(&fd->go, w);
                if (!sh.ok) st_relaxed_sys(&fh->left, seq);
            }
        } else {
            if (threadIdx.x == 0) {
                uint32_t w = 0;
                bool ok = false;
                for (uint32_t k = 0; !ok && k < map.group_polls; ++k) {
                    w = ld_relaxed_gpu(&fd->go);
                    ok = (w >> kCmdShift) == seq;
                }
                if (!ok) { fuse_gave_up(st, 5u, rank, seq); w = kCmdLeave; }
                fence_gpu();
                sh.word = w;
            }
            __syncthreads();
        }
        const uint32_t w = sh.word;
        if (w & kCmdLeave) return;
        uint32_t t_start = now_ns();
        if (threadIdx.x == 0) {
            DomainArgs& m = sh.a;
            m.dt_changed = (w & kCmdDtChanged) ? 1 : 0;
            m.spec = (w & kCmdSpec) ? 1 : 0;
            m.refresh = (w & kCmdRefresh1) ? 1 : (w & kCmdRefresh2) ? 2 : 0;
            if (w & kCmdPayload) {
                const FusePay& p = fd->pay;
                m.mLAGB = p.mLAGB; m.mHAGB = p.mHAGB; m.mGS = p.mGS; m.mRH = p.mRH;
                m.dt = p.dt; m.cinv = p.cinv; m.dtc32 = p.dtc32;
                m.ans_idx = p.ans_idx; m.ans_val = p.ans_val;
            }
        }
        if (w & kCmdForce) {
            const double* src = fd->pay.pf_src;
            for (uint32_t g = rank * kFuse + threadIdx.x; g < a.ndefg; g += G * kFuse) ((double*)a.pforce)[g] = src[g];
            arrived += G;
            if (!group_barrier(sh, &fd->bar, G, arrived, map.group_polls, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 1u, rank, arrived); return; }
        }
        __syncthreads();

        // ---- A: fill
        const uint32_t T0 = (n0 + kTile - 1) / kTile, T = T0 + (n1 + kTile - 1) / kTile;
        const uint32_t nlt = T > rank ? (T - rank + G - 1) / G : 0u;
        uint2* const cntA = (uint2*)cst.f[0].tcnt;   // per tile (full, INACTIVE)
        uint2* const cntB = cntA + T;              // per tile wins (Inside, Border)
        const FuseRecs<ITEMS> rec{sh, rank, G, T0, n0, nlt};
        // the masks of a few tiles stay in shared memory
        const bool own = nlt * kWords <= kFuseMask;
        // the next tile's infector bytes are in flight while this tile's fields are
        const uint32_t in_tile = (uint32_t)threadIdx.x * ITEMS;
        uint32_t dirs = 0xFFFFFFFFu;
        if (nlt) dirs = rank >= T0 ? fuse_dirs<ITEMS>(cst.f[1], (rank - T0) * kTile + in_tile, n1) : fuse_dirs<ITEMS>(cst.f[0], rank * kTile + in_tile, n0);
        for (uint32_t lt = 0; lt < nlt; ++lt) {
            const uint32_t u = rank + lt * G, un = u + G;
            uint32_t next = 0xFFFFFFFFu;
            if (lt + 1 < nlt) next = un >= T0 ? fuse_dirs<ITEMS>(cst.f[1], (un - T0) * kTile + in_tile, n1) : fuse_dirs<ITEMS>(cst.f[0], un * kTile + in_tile, n0);
            const int L = u >= T0 ? 1 : 0;
            const uint32_t tl = L ? u - T0 : u, n = L ? n1 : n0;
            const DFront& fr = cst.f[L];
            const uint32_t slot = tl * kTile + in_tile;
            uint32_t act, full;
            fuse_grow<FP32, ITEMS>(a, fr, slot, dirs, act, full);
            dirs = next;
            // 32 / ITEMS lanes share a mask word
            const uint32_t left = n > slot ? min(n - slot, (uint32_t)ITEMS) : 0u;
            const uint32_t sh0 = ((uint32_t)lane * ITEMS) & 31u;
            uint32_t mf = full << sh0, mi = (~act & ((1u << left) - 1u)) << sh0;
#pragma unroll
            for (int o = 1; o < 32 / ITEMS; o <<= 1) {
                mf |= __shfl_xor_sync(0xFFFFFFFFu, mf, o);
                mi |= __shfl_xor_sync(0xFFFFFFFFu, mi, o);
            }
            if (sh0 == 0u) {
                const uint32_t wt = in_tile >> 5;
                if (own) {
                    sh.fm[lt * kWords + wt] = mf;
                    sh.im[lt * kWords + wt] = mi;
                } else {
                    fr.fmask[tl * kWords + wt] = mf;
                    fr.imask[tl * kWords + wt] = mi;
                }
            }
        }
        for (uint32_t lt = threadIdx.x; lt < nlt; lt += kFuse) { sh.off[lt] = 0xFFFFFFFFu; sh.tw[0][lt] = 0u; sh.tw[1][lt] = 0u; }
        __syncthreads();
        // full cells into records in slot order, tile by tile; the tiles' counts
        uint32_t F = 0;
        for (uint32_t w0 = 0; w0 < nlt * kWords; w0 += kFuse) {
            const uint32_t wi = w0 + threadIdx.x, lt = wi / kWords;
            uint32_t fw = 0, iw = 0, key0 = 0;
            if (lt < nlt) {
                const uint32_t u = rank + lt * G;
                const int L = u >= T0 ? 1 : 0;
                const uint32_t word = (L ? u - T0 : u) * kWords + (wi - lt * kWords);
                fw = own ? sh.fm[wi] : cst.f[L].fmask[word];
                iw = own ? sh.im[wi] : cst.f[L].imask[word];
                key0 = (word * 32u) | ((uint32_t)L << 31);
            }
            const uint32_t c = __popc(fw), ci = __popc(iw);
            uint32_t x = c, y = ci, tx, ty;
            block_scan2(sh, x, y, tx, ty);
            if (lt < nlt && (wi & (kWords - 1)) == 0) sh.off[lt] = F + x;
            // the tile's counts: the last of its words knows the sum from the first's prefix
            __syncthreads();
            if (lt < nlt && (wi & (kWords - 1)) == 0) sh.pre[1][lt] = y;
            __syncthreads();
            if (lt < nlt && (wi & (kWords - 1)) == kWords - 1)
                cntA[rank + lt * G] = make_uint2(F + x + c - sh.off[lt], y + ci - sh.pre[1][lt]);
            uint32_t i = F + x;
            for (uint32_t m = fw; m; m &= m - 1u, ++i) {
                rec.set_key(i, key0 + (uint32_t)(__ffs(m) - 1));
                if (i < kFuseRec) sh.rec_lt[i] = (uint16_t)lt;
            }
            F += tx;
        }
        __syncthreads();
        // the infection attempts: four lanes a full cell; an interior cell's 8 bricks two a lane, a face cell's directions
        // 6 or 7 a lane (a warp a cell and a lane a direction spent its time on addresses: 33 us a step of a
        // 16-domain batch).  The next cells' positions are in flight meanwhile.
        {
            auto position = [&](uint32_t i, uint32_t& key) -> uint32_t {
                if (i >= F) return 0u;
                key = rec.key(i);
                return (key >> 31 ? cst.f[1].xyz : cst.f[0].xyz)[key & 0x7FFFFFFFu];
            };
            uint32_t i = (uint32_t)warp * 8u + (uint32_t)(lane >> 2), key = 0, key_next = 0;
            uint32_t cell = position(i, key);
            for (uint32_t i0 = (uint32_t)warp * 8u; i0 < F; i0 += kFuseWarps * 8u) {
                const uint32_t in = i + kFuseWarps * 8u, cell_next = position(in, key_next);
                uint32_t mask = 0;
                if (i < F) {
                    const uint32_t ord = ((key & 0x7FFFFFFFu) + (key >> 31 ? n0 : 0u)) * 26u;
                    mask = attempt_quarter(cst, (int)(key >> 31), cell, ord, lane & 3, sh.dir);
                }
                mask |= __shfl_xor_sync(0xFFFFFFFFu, mask, 1);
                mask |= __shfl_xor_sync(0xFFFFFFFFu, mask, 2);
                if (i < F && (lane & 3) == 0) {
                    rec.set_win(i, mask);
                    rec.set_cell(i, cell);
                }
                i = in; key = key_next; cell = cell_next;
            }
        }
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, map.group_polls, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 2u, rank, arrived); return; }
        const uint32_t t_a = now_ns();

        // ---- B: recycle list, wins
        tile_scan(sh, cntA, T, T0, rank, G);
        const uint32_t Ftot = sh.tot[0], F0 = sh.t0[0], I0 = sh.t0[1], I1 = sh.tot[1] - I0;
        const uint32_t nrec0 = min(I0, cst.f[0].reccap), nrec1 = min(I1, cst.f[1].reccap);
        {
            // slots that this step cannot hand out are not listed: at most 26 new cells a full cell (a count of the
            // attempts would bound it closer, but took 1 us a step of a small domain)
            const uint32_t most = (uint32_t)min(26ull * Ftot, 0xFFFFFFFFull);
            for (uint32_t lt = 0; lt < nlt; ++lt) {
                const uint32_t u = rank + lt * G;
                const int L = u >= T0 ? 1 : 0;
                const uint32_t cap = min(L ? nrec1 : nrec0, most), r0 = sh.pre[1][lt] - (L ? I0 : 0u);
                if (r0 >= cap) continue;  // uniform over the block
                // warp w lists the slots of words w and w + kFuseWarps: their ranks from all words' counts
                const DFront& fr = cst.f[L];
                const uint32_t word0 = (L ? u - T0 : u) * kWords;
                uint32_t iw[ITEMS], ci[ITEMS], before = 0;
#pragma unroll
                for (int h = 0; h < ITEMS; ++h) {
                    const uint32_t k = 32u * (uint32_t)h + (uint32_t)lane;
                    iw[h] = own ? sh.im[lt * kWords + k] : fr.imask[word0 + k];
                    ci[h] = __popc(iw[h]);
                }
#pragma unroll
                for (int h = 0; h < ITEMS; ++h) {  // word 32 h + warp
                    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, ci[h]);
                    const uint32_t part = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? ci[h] : 0u);
                    const uint32_t wj = __shfl_sync(0xFFFFFFFFu, iw[h], warp);
                    const uint32_t rr = r0 + before + part + __popc(wj & lanemask_lt());
                    if (((wj >> lane) & 1u) && rr < cap) fr.recyc[rr] = (word0 + 32u * (uint32_t)h + (uint32_t)warp) * 32u + (uint32_t)lane;
                    before += all;
                }
            }
        }
        for (uint32_t i0 = (uint32_t)warp * 8u; i0 < F; i0 += kFuseWarps * 8u) {
            const uint32_t i = i0 + (uint32_t)(lane >> 2);
            uint32_t win = 0, tob = 0, key = 0;
            if (i < F) {
                key = rec.key(i);
                const uint32_t s = (key & 0x7FFFFFFFu) + (key >> 31 ? n0 : 0u);
                win_quarter(cst, (int)(key >> 31), rec.cell(i), rec.win(i), s * 26u, lane & 3, sh.dir, win, tob);
            }
            win |= __shfl_xor_sync(0xFFFFFFFFu, win, 1);
            tob |= __shfl_xor_sync(0xFFFFFFFFu, tob, 1);
            win |= __shfl_xor_sync(0xFFFFFFFFu, win, 2);
            tob |= __shfl_xor_sync(0xFFFFFFFFu, tob, 2);
            if (i < F && (lane & 3) == 0) {
                rec.set_win(i, win);
                rec.set_tob(i, tob);
                const uint32_t lt = rec.tile(i, key), cB = __popc(tob), cA = __popc(win) - cB;
                if (cA) atomicAdd(&sh.tw[0][lt], cA);
                if (cB) atomicAdd(&sh.tw[1][lt], cB);
            }
        }
        // a thread takes one full cell a chunk: its grains and overshoot, and what needs no rank, the first chunk's before
        // the barrier, whose wait hides the loads and the atomics' answers (a run of a recovering 384^3 domain 135.3 ms with
        // them after it, 132.4 before; sheets 170.7 and 168.4; 64^3 10.2 and 10.3)
        FullCell fc;
        take_full<FP32>(cst, a, rec, threadIdx.x, F, fc);
        __syncthreads();
        for (uint32_t lt = threadIdx.x; lt < nlt; lt += kFuse) cntB[rank + lt * G] = make_uint2(sh.tw[0][lt], sh.tw[1][lt]);
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, map.group_polls, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 3u, rank, arrived); return; }
        const uint32_t t_b = now_ns();

        // ---- C: commit
        tile_scan(sh, cntB, T, T0, rank, G);
        const uint32_t W0 = sh.tot[0], W1 = sh.tot[1];
        if (warp == 0) {  // the block's own wins before each of its tiles
            uint32_t ca = 0, cb = 0;
            for (uint32_t l0 = 0; l0 < nlt; l0 += 32) {
                const uint32_t lt = l0 + (uint32_t)lane;
                const uint32_t va = lt < nlt ? sh.tw[0][lt] : 0u, vb = lt < nlt ? sh.tw[1][lt] : 0u;
                uint32_t xa = va, xb = vb;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t p = __shfl_up_sync(0xFFFFFFFFu, xa, o), q = __shfl_up_sync(0xFFFFFFFFu, xb, o);
                    if (lane >= o) { xa += p; xb += q; }
                }
                if (lt < nlt) { sh.pre[0][lt] -= ca + xa - va; sh.pre[1][lt] -= cb + xb - vb; }  // may wrap: differences only
                ca += __shfl_sync(0xFFFFFFFFu, xa, 31);
                cb += __shfl_sync(0xFFFFFFFFu, xb, 31);
            }
        }
        __syncthreads();
        double pmax = 0.0;
        uint32_t ntag = 0, ca = 0, cb = 0;   // the block's wins in the chunks before
        for (uint32_t i0 = 0; i0 < F; i0 += kFuse) {
            const uint32_t i = i0 + threadIdx.x;
            if (i0) take_full<FP32>(cst, a, rec, i, F, fc);
            uint32_t win = 0, tob = 0;
            if (i < F) { win = rec.win(i); tob = rec.tob(i); }
            const uint32_t cB = __popc(tob), cA = __popc(win) - cB;
            uint32_t xa = cA, xb = cB, ta, tb;
            block_scan2(sh, xa, xb, ta, tb);
            if (i < F) {
                const uint32_t key = rec.key(i), lt = rec.tile(i, key);
                sh.c_win[threadIdx.x] = win;
                sh.c_tob[threadIdx.x] = tob;
                sh.c_rA[threadIdx.x] = sh.pre[0][lt] + ca + xa;
                sh.c_rB[threadIdx.x] = sh.pre[1][lt] + cb + xb;
                sh.c_cell[threadIdx.x] = rec.cell(i) | (key & 0x80000000u);
                sh.c_rs[threadIdx.x] = fc.rs;
                sh.c_over[threadIdx.x] = fc.over;
            }
            // the chunk's new cells in record and direction order, kFuseWins at a time
            const uint32_t W = ta + tb;
            for (uint32_t w0 = 0; w0 < W; w0 += kFuseWins) {
                if (w0) __syncthreads();
                uint32_t q = xa + xb;
                for (uint32_t m = win; m; m &= m - 1u, ++q)
                    if (q - w0 < kFuseWins) sh.wl[q - w0] = (uint16_t)((threadIdx.x << 5) | (uint32_t)(__ffs(m) - 1));
                __syncthreads();
                for (uint32_t k = threadIdx.x; k < min(W - w0, kFuseWins); k += kFuse) {
                    const uint32_t e = sh.wl[k], t = e >> 5;
                    const int d = (int)(e & 31u);
                    const uint32_t m = sh.c_win[t], tbm = sh.c_tob[t], below = m & ((1u << d) - 1u);
                    const int D = (tbm >> d) & 1u;
                    const uint32_t r = D ? sh.c_rB[t] + __popc(below & tbm) : sh.c_rA[t] + __popc(below & ~tbm);
                    const uint32_t sc = sh.c_cell[t];
                    int x, y, z;
                    decode(cst, sc & 0x7FFFFFFFu, x, y, z);
                    uint32_t tgt;
                    bool inter;
                    target_of(cst, (int)(sc >> 31), x, y, z, sh.dir[d], tgt, inter);
                    const uint32_t gt = cst.grid[tgt];
                    const DFront& dst = a.f[D];
                    const uint32_t nrec = D ? nrec1 : nrec0;
                    const uint32_t ns = r < nrec ? dst.recyc[r] : (D ? n1 : n0) + (r - nrec);
                    if (ns >= dst.cap) { atomicOr(&st->err, kErrCapacity); continue; }
                    if (D == 1 && cst.border_policy == 0 && r >= nrec && ns >= cst.border_ref_cap) atomicOr(&st->err, kErrBorderRef);
                    new_cell<FP32>(a, dst, ns, tgt, gt, sh.c_rs[t], sh.c_over[t], sh.dir[d], pmax, ntag);
                }
            }
            if (fc.gk && fc.gold == fc.gk) {  // the deformed grain's last cells
                const uint32_t q = atomicAdd(&st->ndepleted, 1u);
                if (q < cst.ndefg) cst.depleted[q] = fc.gs;
            }
            ca += ta; cb += tb;
            __syncthreads();
        }
        if (__any_sync(0xFFFFFFFFu, pmax > 0.0 || ntag)) flush_new(a, pmax, ntag);
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, map.group_polls, first)) { if (threadIdx.x == 0) fuse_gave_up(st, 4u, rank, arrived); return; }
        // the lists' ends after this step, the same in every block
        const uint32_t p0 = n0, p1 = n1;
        if (W0 > nrec0) n0 += W0 - nrec0;
        if (W1 > nrec1) n1 += W1 - nrec1;
        bool over_cap = false;
        if (n0 > cst.f[0].cap) { n0 = cst.f[0].cap; over_cap = true; }
        if (n1 > cst.f[1].cap) { n1 = cst.f[1].cap; over_cap = true; }

        // ---- D: the step to the host
        if (first) {
            HostBox* const box = cst.box;
            const uint32_t nm = min(min(__ldcg(&st->nmiss), cst.misscap), kBoxMiss), nd = min(min(__ldcg(&st->ndepleted), cst.ndefg), kBoxDep);
            for (uint32_t i = threadIdx.x; i < nm; i += kFuse) box->miss[i] = __ldcg(&cst.miss[i]);
            for (uint32_t i = threadIdx.x; i < nd; i += kFuse) box->depleted[i] = __ldcg(&cst.depleted[i]);
            if (threadIdx.x == 0) {
                DevState v;
                v.next_never[0] = n0; v.next_never[1] = n1;
                v.err = __ldcg(&st->err) | (over_cap ? kErrCapacity : 0u);
                v.err_info = __ldcg(&st->err_info);
                v.ntouch = __ldcg(&st->ntouch);
                for (int j = 0; j < 3; ++j) v.reserved[j] = 0;
                v.nfull[0] = F0; v.nfull[1] = Ftot - F0;
                v.ninactive[0] = I0; v.ninactive[1] = I1;
                v.nrec[0] = nrec0; v.nrec[1] = nrec1;
                v.nwin[0] = W0; v.nwin[1] = W1;
                v.nmiss = __ldcg(&st->nmiss); v.ntagged = __ldcg(&st->ntagged);
                v.ndepleted = __ldcg(&st->ndepleted); v.nnuc = __ldcg(&st->nnuc);
                v.nknown = __ldcg(&st->nknown);
                v.commit_done = 0;
                v.sv[0] = p0 - I0; v.sv[1] = p1 - I1;
                v.pmax_bits = __ldcg(&st->pmax_bits);
                v.dv[0] = v.dv[1] = 0.0;
                box->snap = v;
                st->next_never[0] = n0; st->next_never[1] = n1;
                st->err = v.err;
                st->nmiss = 0; st->ntagged = 0; st->nknown = 0; st->ndepleted = 0; st->nnuc = 0; st->pmax_bits = 0;
                const uint32_t t_c = now_ns();
                fh->phase_ns[0] = t_a - t_start; fh->phase_ns[1] = t_b - t_a; fh->phase_ns[2] = t_c - t_b; fh->phase_ns[3] = t_c - t_start;
                if (w & kCmdLast) fd->bar = 0u;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                fence_sys();
                st_relaxed_sys(&fh->post, seq);
            }
        }
        if (w & kCmdLast) return;
        seq = fuse_next(seq);
    }
}

}  // namespace score
