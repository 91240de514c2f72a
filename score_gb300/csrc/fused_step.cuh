// One launch for many growth steps of domains whose fronts are too small to fill the GPU.
//
// What bounds such a domain is neither bytes nor operations but the chain of a step: five or six
// launches, each with its own start, constant-cache misses and dependent loads, then a stream
// synchronization and the host's master block (64^3 domain, front of 30 k slots: 51 us a step, of which the
// bytes take 0.1; 128^3: 59 us; here 26 and 33).  A group of blocks steps one domain inside one
// cooperative launch:
//   A  fill of the group's tiles; full cells into records; the 26 infection attempts of every full
//      cell, a warp per full cell and a lane per direction.  The attempt ordinal is 26 s + d with s the
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
constexpr int kFuseItems = 2;
constexpr uint32_t kFuseTile = kFuse * kFuseItems;        // slots per tile
constexpr uint32_t kFuseTileWords = kFuseTile / 32;
static_assert(kFuseTileWords == 32 * kFuseItems && kFuseWarps == 32, "a word of a tile per warp and item");
constexpr uint32_t kFuseMaxTiles = 4096;                  // tiles of a domain (both lists)
constexpr uint32_t kFuseMaxLocal = 512;                   // tiles of one block
constexpr uint32_t kFuseRec = 3072;                       // full cells of a block and step kept in shared memory
constexpr uint32_t kFuseSpin = 1u << 22;                  // polls of a group wait before it gives up (seconds)
constexpr uint32_t kFuseHostSpin = 1u << 12;              // polls of the host's answer before the group leaves (milliseconds)

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
    uint32_t fm[kFuse], im[kFuse];     // full and INACTIVE masks of the block's tiles while they fit
    uint16_t wl[kFuse * 26];           // wins of a chunk of records: record in the chunk << 5 | direction
    uint32_t c_win[kFuse], c_tob[kFuse], c_rA[kFuse], c_rB[kFuse], c_cell[kFuse], c_rs[kFuse];
    double c_over[kFuse];
    uint32_t tw[2][kFuseMaxLocal];     // wins of the block's tiles per destination list
    uint32_t pre[2][kFuseMaxLocal];    // prefix of the domain's counts at the block's tiles
    uint32_t off[kFuseMaxLocal + 1];   // first record of each of the block's tiles
    uint32_t w1[kFuseWarps], w2[kFuseWarps], w3[kFuseWarps];
    uint32_t t0[2], tot[2];            // counts before the Border list's tiles, and in all
    uint32_t word, ok;
};

// Arrival of the block at its group's barrier and, with `wait`, the wait for the whole group.  target: arrivals
// of the launch so far when everyone is there.  False (for the whole block) when the wait gave up.
__device__ __forceinline__ bool group_barrier(FuseShared& sh, uint32_t* bar, uint32_t G, uint32_t target, bool wait) {
    __syncthreads();
    if (G == 1) return true;
    if (threadIdx.x == 0) {
        fence_gpu();   // cumulative: the block's stores, ordered before thread 0 by the block barrier
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        bool ok = !wait;
        for (uint32_t k = 0; !ok && k < kFuseSpin; ++k) ok = (int32_t)(ld_relaxed_gpu(bar) - target) >= 0;
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

// target_of for a lane's own direction
__device__ __forceinline__ bool target_lane(const DomainArgs& a, int L, int x, int y, int z, int dx, int dy, int dz, uint32_t& t,
                                            bool& interior) {
    int tx = x + dx, ty = y + dy, tz = z + dz;
    if (L == 1) {
        if (tx < 0) tx += (int)a.nx;
        if (tx >= (int)a.nx) tx -= (int)a.nx;
        if (ty < 0) ty += (int)a.ny;
        if (ty >= (int)a.ny) ty -= (int)a.ny;
        if (a.boundary == 0) {
            if (tz < 0 || tz >= (int)a.nz) return false;
        } else {
            if (tz < 0) tz += (int)a.nz;
            if (tz >= (int)a.nz) tz -= (int)a.nz;
        }
    } else if (tx < 0 || ty < 0 || tz < 0 || tx >= (int)a.nx || ty >= (int)a.ny || tz >= (int)a.nz) {
        atomicOr(&a.st->err, kErrBounds);
        return false;
    }
    interior = tx > 0 && tx < (int)a.nx - 1 && ty > 0 && ty < (int)a.ny - 1 && tz > 0 && tz < (int)a.nz - 1;
    t = gindex(a, (uint32_t)tx, (uint32_t)ty, (uint32_t)tz);
    return true;
}

// The records of a block's full cells: the first kFuseRec in shared memory, the rest in the domain's per-full-cell
// arrays at the full cell's own slot position (a position no other full cell has; n0 + n1 slots never exceed the
// arrays' N words, as every slot stands for a cell infected once).  `pos` is looked up from the tile offsets.
struct FuseRecs {
    FuseShared& sh;
    uint32_t rank, G, T0, n0, nlt;
    __device__ __forceinline__ uint32_t pos(uint32_t i) const {
        uint32_t lt = nlt - 1;
        while (sh.off[lt] > i) --lt;
        const uint32_t u = rank + lt * G;
        return (u >= T0 ? n0 + (u - T0) * kFuseTile : u * kFuseTile) + (i - sh.off[lt]);
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
        const uint32_t tl = (k & 0x7FFFFFFFu) / kFuseTile;
        return ((k >> 31 ? T0 + tl : tl) - rank) / G;
    }
};

template <bool FP32>
__device__ __forceinline__ void fuse_grow(const DomainArgs& a, const DFront& fr, uint32_t base, uint32_t n, uint32_t& act, uint32_t& full) {
    if (a.refresh == 2) grow_items<FP32, 2, kFuseItems>(a, fr, base, n, act, full);
    else if (a.refresh == 1) grow_items<FP32, 1, kFuseItems>(a, fr, base, n, act, full);
    else if (a.spec && !a.dt_changed) grow_items<FP32, 3, kFuseItems>(a, fr, base, n, act, full);
    else grow_items<FP32, 0, kFuseItems>(a, fr, base, n, act, full);
}

template <bool FP32>
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
    const DomainArgs& a = sh.a;
    if (!a.active) return;
    DevState* const st = a.st;
    FuseDom* const fd = a.fuse;
    FuseHost* const fh = &a.box->fuse;
    const bool first = rank == 0;
    uint32_t n0 = st->next_never[0], n1 = st->next_never[1];
    uint32_t seq = map.seq[dom] & kCmdSeqMask, arrived = 0;
    // this lane's direction
    const int dl = lane < 26 ? lane : 25;
    const int dx = c_dx[dl], dy = c_dy[dl], dz = c_dz[dl];
    for (;;) {
        // ---- the host's word for step `seq`
        if (first) {
            if (threadIdx.x == 0) {
                uint32_t w = 0;
                bool ok = false;
                for (uint32_t k = 0; !ok && k < kFuseHostSpin; ++k) {
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
                for (uint32_t k = 0; !ok && k < kFuseSpin; ++k) {
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
            if (!group_barrier(sh, &fd->bar, G, arrived, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 1u, rank, arrived); return; }
        }
        __syncthreads();

        // ---- A: fill
        const uint32_t T0 = (n0 + kFuseTile - 1) / kFuseTile, T = T0 + (n1 + kFuseTile - 1) / kFuseTile;
        const uint32_t nlt = T > rank ? (T - rank + G - 1) / G : 0u;
        uint2* const cntA = (uint2*)a.f[0].tcnt;   // per tile (full, INACTIVE)
        uint2* const cntB = cntA + T;              // per tile wins (Inside, Border)
        const FuseRecs rec{sh, rank, G, T0, n0, nlt};
        // the masks of a few tiles stay in shared memory
        const bool own = nlt * kFuseTileWords <= (uint32_t)kFuse;
        for (uint32_t lt = 0; lt < nlt; ++lt) {
            const uint32_t u = rank + lt * G;
            const int L = u >= T0 ? 1 : 0;
            const uint32_t tl = L ? u - T0 : u, n = L ? n1 : n0;
            const DFront& fr = a.f[L];
            const uint32_t slot = tl * kFuseTile + (uint32_t)warp * 32u * kFuseItems + (uint32_t)lane;
            uint32_t act, full;
            fuse_grow<FP32>(a, fr, slot, n, act, full);
            uint32_t mf = 0, mi = 0;
#pragma unroll
            for (int k = 0; k < kFuseItems; ++k) {
                const uint32_t f = __ballot_sync(0xFFFFFFFFu, (full >> k) & 1u);
                const uint32_t i = __ballot_sync(0xFFFFFFFFu, !((act >> k) & 1u) && slot + 32u * (uint32_t)k < n);
                if (lane == k) { mf = f; mi = i; }
            }
            if (lane < kFuseItems) {
                const uint32_t wt = (uint32_t)(warp * kFuseItems + lane);
                if (own) {
                    sh.fm[lt * kFuseTileWords + wt] = mf;
                    sh.im[lt * kFuseTileWords + wt] = mi;
                } else {
                    fr.fmask[tl * kFuseTileWords + wt] = mf;
                    fr.imask[tl * kFuseTileWords + wt] = mi;
                }
            }
        }
        for (uint32_t lt = threadIdx.x; lt < nlt; lt += kFuse) { sh.off[lt] = 0xFFFFFFFFu; sh.tw[0][lt] = 0u; sh.tw[1][lt] = 0u; }
        __syncthreads();
        // full cells into records in slot order, tile by tile; the tiles' counts
        uint32_t F = 0;
        for (uint32_t w0 = 0; w0 < nlt * kFuseTileWords; w0 += kFuse) {
            const uint32_t wi = w0 + threadIdx.x, lt = wi / kFuseTileWords;
            uint32_t fw = 0, iw = 0, key0 = 0;
            if (lt < nlt) {
                const uint32_t u = rank + lt * G;
                const int L = u >= T0 ? 1 : 0;
                const uint32_t word = (L ? u - T0 : u) * kFuseTileWords + (wi - lt * kFuseTileWords);
                fw = own ? sh.fm[wi] : a.f[L].fmask[word];
                iw = own ? sh.im[wi] : a.f[L].imask[word];
                key0 = (word * 32u) | ((uint32_t)L << 31);
            }
            const uint32_t c = __popc(fw), ci = __popc(iw);
            uint32_t x = c, y = ci, tx, ty;
            block_scan2(sh, x, y, tx, ty);
            if (lt < nlt && (wi & (kFuseTileWords - 1)) == 0) sh.off[lt] = F + x;
            // the tile's counts: the last of its words knows the sum from the first's prefix
            __syncthreads();
            if (lt < nlt && (wi & (kFuseTileWords - 1)) == 0) sh.pre[1][lt] = y;
            __syncthreads();
            if (lt < nlt && (wi & (kFuseTileWords - 1)) == kFuseTileWords - 1)
                cntA[rank + lt * G] = make_uint2(F + x + c - sh.off[lt], y + ci - sh.pre[1][lt]);
            uint32_t i = F + x;
            for (uint32_t m = fw; m; m &= m - 1u, ++i) {
                rec.set_key(i, key0 + (uint32_t)(__ffs(m) - 1));
                if (i < kFuseRec) sh.rec_lt[i] = (uint16_t)lt;
            }
            F += tx;
        }
        __syncthreads();
        // the infection attempts: a warp takes 4 full cells at a time, a lane one direction of each
        for (uint32_t i0 = (uint32_t)warp; i0 < F; i0 += kFuseWarps * 4u) {
            uint32_t key[4], cell[4], tg[4], gv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) key[j] = i0 + kFuseWarps * j < F ? rec.key(i0 + kFuseWarps * j) : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) cell[j] = i0 + kFuseWarps * j < F ? a.f[key[j] >> 31].xyz[key[j] & 0x7FFFFFFFu] : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                gv[j] = 0xFFFFFFFFu;
                if (i0 + kFuseWarps * j < F && lane < 26) {
                    int x, y, z;
                    bool inter;
                    decode(a, cell[j], x, y, z);
                    if (target_lane(a, (int)(key[j] >> 31), x, y, z, dx, dy, dz, tg[j], inter)) gv[j] = a.grid[tg[j]];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool at = gv[j] < a.ndefg;
                if (at) {
                    const uint32_t s = (key[j] & 0x7FFFFFFFu) + (key[j] >> 31 ? n0 : 0u);
                    atomicMin(&a.claim[tg[j]], s * 26u + (uint32_t)lane);
                }
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, at);
                if (lane == 0 && i0 + kFuseWarps * j < F) { rec.set_win(i0 + kFuseWarps * j, m); rec.set_cell(i0 + kFuseWarps * j, cell[j]); }
            }
        }
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 2u, rank, arrived); return; }
        const uint32_t t_a = now_ns();

        // ---- B: recycle list, wins
        tile_scan(sh, cntA, T, T0, rank, G);
        const uint32_t Ftot = sh.tot[0], F0 = sh.t0[0], I0 = sh.t0[1], I1 = sh.tot[1] - I0;
        const uint32_t nrec0 = min(I0, a.f[0].reccap), nrec1 = min(I1, a.f[1].reccap);
        {
            // slots that this step cannot hand out are not listed: at most 26 new cells a full cell
            const uint32_t most = (uint32_t)min(26ull * Ftot, 0xFFFFFFFFull);
            for (uint32_t lt = 0; lt < nlt; ++lt) {
                const uint32_t u = rank + lt * G;
                const int L = u >= T0 ? 1 : 0;
                const uint32_t cap = min(L ? nrec1 : nrec0, most), r0 = sh.pre[1][lt] - (L ? I0 : 0u);
                if (r0 >= cap) continue;  // uniform over the block
                // warp w lists the slots of words w and w + kFuseWarps: their ranks from all words' counts
                const DFront& fr = a.f[L];
                const uint32_t word0 = (L ? u - T0 : u) * kFuseTileWords;
                uint32_t iw[kFuseItems], ci[kFuseItems], before = 0;
#pragma unroll
                for (int h = 0; h < kFuseItems; ++h) {
                    const uint32_t k = 32u * (uint32_t)h + (uint32_t)lane;
                    iw[h] = own ? sh.im[lt * kFuseTileWords + k] : fr.imask[word0 + k];
                    ci[h] = __popc(iw[h]);
                }
#pragma unroll
                for (int h = 0; h < kFuseItems; ++h) {  // word 32 h + warp
                    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, ci[h]);
                    const uint32_t part = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? ci[h] : 0u);
                    const uint32_t wj = __shfl_sync(0xFFFFFFFFu, iw[h], warp);
                    const uint32_t rr = r0 + before + part + __popc(wj & lanemask_lt());
                    if (((wj >> lane) & 1u) && rr < cap) fr.recyc[rr] = (word0 + 32u * (uint32_t)h + (uint32_t)warp) * 32u + (uint32_t)lane;
                    before += all;
                }
            }
        }
        for (uint32_t i0 = (uint32_t)warp; i0 < F; i0 += kFuseWarps * 4u) {
            uint32_t key[4], cl[4];
            bool at[4], tb[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                at[j] = false; tb[j] = false; cl[j] = kClaimFree; key[j] = 0u;
                if (i0 + kFuseWarps * j < F) {
                    key[j] = rec.key(i0 + kFuseWarps * j);
                    at[j] = (rec.win(i0 + kFuseWarps * j) >> lane) & 1u;
                    if (at[j]) {
                        const int L = (int)(key[j] >> 31);
                        int x, y, z;
                        decode(a, rec.cell(i0 + kFuseWarps * j), x, y, z);
                        uint32_t t;
                        bool inter;
                        target_lane(a, L, x, y, z, dx, dy, dz, t, inter);
                        cl[j] = a.claim[t];
                        // Inside full cells near a face infect into the Border list (SCORE_Kernel.cpp:4606-4609);
                        // Border full cells send strictly interior targets to the Inside list (:4387)
                        const bool allB = !(x > 1 && x < (int)a.nx - 2 && y > 1 && y < (int)a.ny - 2 && z > 1 && z < (int)a.nz - 2);
                        tb[j] = L == 0 ? allB : !inter;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t s = (key[j] & 0x7FFFFFFFu) + (key[j] >> 31 ? n0 : 0u);
                const bool won = at[j] && cl[j] == s * 26u + (uint32_t)lane;
                const uint32_t win = __ballot_sync(0xFFFFFFFFu, won), tob = __ballot_sync(0xFFFFFFFFu, won && tb[j]);
                if (lane == 0 && i0 + kFuseWarps * j < F) {
                    rec.set_win(i0 + kFuseWarps * j, win);
                    rec.set_tob(i0 + kFuseWarps * j, tob);
                    const uint32_t lt = rec.tile(i0 + kFuseWarps * j, key[j]), cB = __popc(tob), cA = __popc(win) - cB;
                    if (cA) atomicAdd(&sh.tw[0][lt], cA);
                    if (cB) atomicAdd(&sh.tw[1][lt], cB);
                }
            }
        }
        __syncthreads();
        for (uint32_t lt = threadIdx.x; lt < nlt; lt += kFuse) cntB[rank + lt * G] = make_uint2(sh.tw[0][lt], sh.tw[1][lt]);
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, true)) { if (threadIdx.x == 0) fuse_gave_up(st, 3u, rank, arrived); return; }
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
            uint32_t win = 0, tob = 0, key = 0, cell = 0, rs = 0, gs = 0;
            double over = 0.0;
            if (i < F) {
                key = rec.key(i); cell = rec.cell(i); win = rec.win(i); tob = rec.tob(i);
                const DFront& fr = a.f[key >> 31];
                const uint32_t slot = key & 0x7FFFFFFFu;
                rs = fr.rxg[slot];
                gs = fr.defg[slot];
                if (win) {
                    if (!FP32) over = __dsub_rn(((const double*)fr.fill)[slot], 1.0);
                    else over = (double)((((const float*)fr.fill)[slot] - 1.0f) - fr.comp[slot]);
                }
            }
            // the grains' counts: the atomic's answer is looked at after the new cells
            const uint32_t has = __ballot_sync(0xFFFFFFFFu, i < F);
            uint32_t gk = 0, gold = 0;
            if (has) {
                const uint32_t mr = __match_any_sync(0xFFFFFFFFu, i < F ? rs : 0xFFFFFFFFu) & has;
                const uint32_t mg = __match_any_sync(0xFFFFFFFFu, i < F ? gs : 0xFFFFFFFFu) & has;
                if (i < F && (__ffs(mr) - 1) == lane) atomicAdd(&a.rxg_cnt[rs], (uint32_t)__popc(mr));
                if (i < F && (__ffs(mg) - 1) == lane) {
                    gk = (uint32_t)__popc(mg);
                    gold = atomicSub(&a.defg_cnt[gs], gk);
                }
            }
            const uint32_t cB = __popc(tob), cA = __popc(win) - cB;
            uint32_t xa = cA, xb = cB, ta, tb;
            block_scan2(sh, xa, xb, ta, tb);
            if (i < F) {
                const uint32_t lt = rec.tile(i, key);
                sh.c_win[threadIdx.x] = win;
                sh.c_tob[threadIdx.x] = tob;
                sh.c_rA[threadIdx.x] = sh.pre[0][lt] + ca + xa;
                sh.c_rB[threadIdx.x] = sh.pre[1][lt] + cb + xb;
                sh.c_cell[threadIdx.x] = cell | (key & 0x80000000u);
                sh.c_rs[threadIdx.x] = rs;
                sh.c_over[threadIdx.x] = over;
                uint32_t q = xa + xb;
                for (uint32_t m = win; m; m &= m - 1u) sh.wl[q++] = (uint16_t)((threadIdx.x << 5) | (uint32_t)(__ffs(m) - 1));
            }
            __syncthreads();
            const uint32_t W = ta + tb;
            for (uint32_t k = threadIdx.x; k < W; k += kFuse) {
                const uint32_t e = sh.wl[k], t = e >> 5;
                const int d = (int)(e & 31u);
                const uint32_t m = sh.c_win[t], tbm = sh.c_tob[t], below = m & ((1u << d) - 1u);
                const int D = (tbm >> d) & 1u;
                const uint32_t r = D ? sh.c_rB[t] + __popc(below & tbm) : sh.c_rA[t] + __popc(below & ~tbm);
                const uint32_t sc = sh.c_cell[t];
                int x, y, z;
                decode(a, sc & 0x7FFFFFFFu, x, y, z);
                uint32_t tgt;
                bool inter;
                target_of(a, (int)(sc >> 31), x, y, z, d, tgt, inter);
                const uint32_t gt = a.grid[tgt];
                const DFront& dst = a.f[D];
                const uint32_t nrec = D ? nrec1 : nrec0;
                const uint32_t ns = r < nrec ? dst.recyc[r] : (D ? n1 : n0) + (r - nrec);
                if (ns >= dst.cap) { atomicOr(&st->err, kErrCapacity); continue; }
                if (D == 1 && a.border_policy == 0 && r >= nrec && ns >= a.border_ref_cap) atomicOr(&st->err, kErrBorderRef);
                new_cell<FP32>(a, dst, ns, tgt, gt, sh.c_rs[t], sh.c_over[t], d, pmax, ntag);
            }
            if (i < F) {  // the full cell is now recrystallized
                const DFront& src = a.f[key >> 31];
                const uint32_t slot = key & 0x7FFFFFFFu;
                a.grid[cell] = a.ndefg + rs;
                src.dir[slot] = kInactive;
                if (!FP32) ((double*)src.fill)[slot] = 0.0;
                else { ((float*)src.fill)[slot] = 0.0f; src.comp[slot] = 0.0f; }
            }
            if (gk && gold == gk) {
                const uint32_t q = atomicAdd(&st->ndepleted, 1u);
                if (q < a.ndefg) a.depleted[q] = gs;
            }
            ca += ta; cb += tb;
            __syncthreads();
        }
        if (__any_sync(0xFFFFFFFFu, pmax > 0.0 || ntag)) flush_new(a, pmax, ntag);
        arrived += G;
        if (!group_barrier(sh, &fd->bar, G, arrived, first)) { if (threadIdx.x == 0) fuse_gave_up(st, 4u, rank, arrived); return; }
        // the lists' ends after this step, the same in every block
        const uint32_t p0 = n0, p1 = n1;
        if (W0 > nrec0) n0 += W0 - nrec0;
        if (W1 > nrec1) n1 += W1 - nrec1;
        bool over_cap = false;
        if (n0 > a.f[0].cap) { n0 = a.f[0].cap; over_cap = true; }
        if (n1 > a.f[1].cap) { n1 = a.f[1].cap; over_cap = true; }

        // ---- D: the step to the host
        if (first) {
            HostBox* const box = a.box;
            const uint32_t nm = min(min(__ldcg(&st->nmiss), a.misscap), kBoxMiss), nd = min(min(__ldcg(&st->ndepleted), a.ndefg), kBoxDep);
            for (uint32_t i = threadIdx.x; i < nm; i += kFuse) box->miss[i] = __ldcg(&a.miss[i]);
            for (uint32_t i = threadIdx.x; i < nd; i += kFuse) box->depleted[i] = __ldcg(&a.depleted[i]);
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
        seq = (seq + 1u) & kCmdSeqMask;
    }
}

}  // namespace score
