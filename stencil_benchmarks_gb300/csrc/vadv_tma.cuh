// Vertical advection with float32 compute: columns staged by the tensor memory
// accelerator, factors in tensor memory (TMEM).
//
// One warp solves 32 consecutive columns (i unit-stride), one per lane.  A
// field is described to the TMA as a 2D tensor: x = element offset inside a
// level (i + j * sj flattened), y = level.  One cp.async.bulk.tensor brings a
// box of 8 levels x (32 columns + the rest of their 16-byte granules) of one
// field, so a warp issues five instructions (six when wcon is read at j + 1)
// per 8 levels, and a level costs its lanes six shared loads, the arithmetic
// and an eighth of a TMEM store, against the copies, addresses and predicates
// of per-lane cp.async rows (stencil_core.cuh:vadv_tmem_column).  A tensor
// copy's operands live in uniform registers: everything it needs is computed
// from warp-uniform values, or each copy costs about 18 instructions.
//
// A tensor stride is a multiple of 16 bytes.  Where the level stride is not,
// the map's stride is the multiple below it and level k starts drift = stride
// mod 16 bytes further right than level k - 1: the boxes are 7 * drift bytes
// wider, a stage's box starts 8 * drift bytes (a multiple of 16) further right
// than the one before, and row q of a box begins q * drift bytes into it.
// (512x512x80 bfloat16 with drift 8 at 11 warps: 77 us; with two maps of every other level
// instead, twice the copies, 91 us.)
//
// Stages form a ring per warp that runs on across solves: a freed stage is
// refilled with a level block further up, which near the end of a column group
// is the start of the warp's next one, so its first loads pass during the
// backward sweep.  pos returns for the backward sweep through a second ring.
// The factors of a warp's first nt level blocks live in TMEM, those of the
// others in shared memory: TMEM alone would hold 12 warps per SM at 80 levels
// and 4 from 137 levels on.  The last block's stay in registers, as the backward
// sweep starts with them; the 2 KB a warp that this frees let 14 warps of two
// stages share an SM at 80 levels (8192 column groups in 4 rounds instead of 5:
// bfloat16 76 -> 72 us, float32 100 either way).
// All waits are bounded (see TmaPipe::wait).
// Bound, 512x512x80: float32 HBM (5.0 TB/s of compulsory bytes, 75% of the
// measured copy rate; fewer warps or deeper rings change it by 2%), bfloat16 the
// issue slots and the recurrence's latency at 14 warps per SM.  Against the
// cp.async form: float32 131 -> 100 us (odd planes 153 -> 110), bfloat16
// 113 -> 72 (odd planes 151 -> 84; aligned rows 85 -> 40 at 510x254x80),
// 400x300x137 170 -> 99 and 189 -> 89, u, v, w of 256x256x80 fused 144 -> 83.
#pragma once

#include <algorithm>

#include "stencil_core.cuh"
#include "tensor_map.cuh"

namespace sb {

constexpr int kTmaLevels = 8;     // levels per stage
constexpr int kTmaMaxStages = 3;  // stages of the forward ring: 2 or 3
constexpr int kTmaMaxWarps = 16;  // of a block: four per lane quarter of TMEM
constexpr int kTmaPosStages = 2;  // stages of the pos ring of the backward sweep
constexpr int kTmaBlockCols = 2 * kTmaLevels;            // TMEM columns of a block's factors
constexpr int kTmaBlockBytes = 2 * kTmaLevels * 32 * 4;  // shared memory of a block's factors
// the ring may run `stages` blocks into the next column group, and the first block has no last level
__host__ __device__ constexpr int tma_min_levels(int stages) { return kTmaLevels * (stages - 1) + 1; }
constexpr int kTmaFields = 5;     // maps in the order wcon(k+1), stage(k+1), pos(k), tens(k), tensstage(k)

// Geometry of the boxes for a drift of R bytes; R < 0: any drift, a run-time value.
template <class S, int R>
struct TmaBox {
    static constexpr int ES = (int)sizeof(S);
    static constexpr int EPG = 16 / ES;  // elements per 16-byte granule
    // 32 columns and wcon's i + 1, any granule offset, any row's drift
    static constexpr int ROWB = (33 * ES + (16 - ES) + (kTmaLevels - 1) * (R < 0 ? 16 - ES : R) + 15) / 16 * 16;
    static constexpr int W = ROWB / ES;
    static constexpr int BOXB = (ROWB * kTmaLevels + 127) / 128 * 128;  // boxes start on 128-byte boundaries
    static constexpr int POSB = BOXB;                                    // a stage of the pos ring
    static constexpr int BAR_BYTES = (kTmaMaxStages + kTmaPosStages) * 8;  // mbarriers of one warp
    // one stage: five boxes, six when wcon(j + 1) has its own
    static __host__ __device__ constexpr int stage_bytes(bool far) { return (kTmaFields + (far ? 1 : 0)) * BOXB; }
    static __host__ __device__ constexpr int rings_bytes(bool far, int stages) {
        return stages * stage_bytes(far) + kTmaPosStages * POSB;
    }
    // dynamic shared memory of a block: 16 bytes for the TMEM address, the warps'
    // mbarriers, then (here) the warps' rings and factor blocks
    static __host__ __device__ constexpr int ring_offset(int nwarps) { return (16 + nwarps * BAR_BYTES + 127) / 128 * 128; }
};
static_assert(TmaBox<float, 0>::W == 36 && TmaBox<bf16, 0>::W == 40 && TmaBox<bf16, -1>::W <= 256, "box widths");

// a warp-uniform value, in a form that the compiler keeps in a uniform register
__device__ __forceinline__ int uniform(int v) { return __reduce_max_sync(0xffffffffu, v); }

// one solve of 32 columns: everything a warp needs to stage and compute it
template <class S>
struct TmaSolve {
    const CUtensorMap* maps;  // [kTmaFields]
    int x[kTmaFields + 1];    // x of column col0 in each map, and of wcon's at the shift
    const S* stage;
    S* out;
    int col0, nvalid, nk, sk, wsh;
    int drift;  // bytes
    bool live;
    __device__ __forceinline__ int blocks() const { return (nk + kTmaLevels - 1) / kTmaLevels; }
};

__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint32_t dst, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
            dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// the maps of a domain that a copy in the same stream brought to global memory
__device__ __forceinline__ void acquire_maps(const CUtensorMap* maps) {
#pragma unroll
    for (int f = 0; f < kTmaFields; ++f)
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"((uint64_t)(maps + f)) : "memory");
}

// one lane of the (converged) warp, the same each time
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one)::"memory");
    return one != 0u;
}

// 16 consecutive TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&f)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
        "r"(__float_as_uint(f[0])), "r"(__float_as_uint(f[1])), "r"(__float_as_uint(f[2])), "r"(__float_as_uint(f[3])), "r"(__float_as_uint(f[4])), "r"(__float_as_uint(f[5])), "r"(__float_as_uint(f[6])), "r"(__float_as_uint(f[7])), "r"(__float_as_uint(f[8])), "r"(__float_as_uint(f[9])), "r"(__float_as_uint(f[10])), "r"(__float_as_uint(f[11])), "r"(__float_as_uint(f[12])), "r"(__float_as_uint(f[13])), "r"(__float_as_uint(f[14])), "r"(__float_as_uint(f[15]))
        : "memory");
}
// issue only: the registers are valid after tmem_wait_ld
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// ties the registers to the wait, so that no use moves above it
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// The two rings of one warp.  Fill and drain positions run on across solves;
// each is a stage index and the parity of its pass over the ring.
struct TmaRing {
    uint32_t stage, parity;
    __device__ __forceinline__ void next(uint32_t n) {
        if (++stage == n) {
            stage = 0;
            parity ^= 1u;
        }
    }
};

template <class S, int R>
struct TmaPipe {
    using B = TmaBox<S, R>;
    unsigned char* mem;  // forward stages, then pos stages
    uint32_t mem_s, bar_s;
    uint32_t stage_b;  // bytes of one forward stage
    int lane, polls;
    uint32_t stages;  // of the forward ring
    TmaRing fillr, drainr, pfillr, pdrainr;

    __device__ __forceinline__ void init(unsigned char* m, unsigned char* bars, int lane_, uint32_t stages_, int stage_bytes,
                                         int polls_) {
        mem = m;
        mem_s = (uint32_t)uniform((int)__cvta_generic_to_shared(m));
        bar_s = (uint32_t)uniform((int)__cvta_generic_to_shared(bars));
        stage_b = stage_bytes;
        lane = lane_;
        stages = stages_;
        polls = polls_;
        fillr = drainr = pfillr = pdrainr = TmaRing{0u, 0u};
        if (lane == 0) {
            for (int q = 0; q < kTmaMaxStages + kTmaPosStages; ++q)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_s + 8 * q) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
    }
    static __device__ __forceinline__ void expect(uint32_t bar, uint32_t bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
    }
    // granule that holds x (the granule offset of a field plus a column), moved to block blk's levels
    static __device__ __forceinline__ int box_x(const TmaSolve<S>& v, int x, int blk) {
        const int drift = R < 0 ? v.drift : R;
        return (x & ~(B::EPG - 1)) + blk * (kTmaLevels * drift / B::ES);
    }
    // level block `blk` of solve `v` into the next forward stage
    __device__ __forceinline__ void fill(const TmaSolve<S>& v, int blk) {
        const uint32_t bar = bar_s + 8 * fillr.stage, dst = mem_s + fillr.stage * stage_b;
        fillr.next(stages);
        const bool far = v.wsh > 1;  // wcon(i, j + 1): a box of its own
        if (elect_one()) {
            expect(bar, (uint32_t)((far ? kTmaFields + 1 : kTmaFields) * (B::ROWB * kTmaLevels)));
#pragma unroll
            for (int f = 0; f < kTmaFields; ++f)
                tma_load_2d(v.maps + f, dst + (uint32_t)(f * B::BOXB), bar, box_x(v, v.x[f], blk), blk * kTmaLevels);
            if (far)
                tma_load_2d(v.maps, dst + (uint32_t)(kTmaFields * B::BOXB), bar, box_x(v, v.x[kTmaFields], blk),
                            blk * kTmaLevels);
        }
    }
    // pos of level block `blk` into the next stage of the backward ring
    __device__ __forceinline__ void fill_pos(const TmaSolve<S>& v, int blk) {
        const uint32_t bar = bar_s + 8 * (kTmaMaxStages + pfillr.stage);
        const uint32_t dst = mem_s + stages * stage_b + pfillr.stage * B::POSB;
        pfillr.next(kTmaPosStages);
        if (elect_one()) {
            expect(bar, (uint32_t)(B::ROWB * kTmaLevels));
            tma_load_2d(v.maps + 2, dst, bar, box_x(v, v.x[2], blk), blk * kTmaLevels);
        }
    }
    // Wait for the stage at position r of the ring whose first barrier is `bar`,
    // at most `tries` polls; the decision is the whole warp's.
    __device__ __forceinline__ bool wait(uint32_t bar, const TmaRing& r, int tries) const {
        return __all_sync(0xffffffffu, mbar_wait(bar + 8 * r.stage, r.parity, tries));
    }
    // wait for the next full stage of each ring; its memory
    __device__ __forceinline__ bool ready() const { return wait(bar_s, drainr, polls); }
    __device__ __forceinline__ const unsigned char* stage() const { return mem + drainr.stage * stage_b; }
    __device__ __forceinline__ bool ready_pos() const { return wait(bar_s + 8 * kTmaMaxStages, pdrainr, polls); }
    __device__ __forceinline__ const unsigned char* stage_pos() const {
        return mem + stages * stage_b + pdrainr.stage * B::POSB;
    }
    // every lane has read the stage: its memory may be filled again
    __device__ __forceinline__ void release(TmaRing& r, uint32_t n) {
        r.next(n);
        __syncwarp();
    }
    // After a wait that gave up: wait (bounded) for every copy still in flight,
    // so that none lands in memory the block no longer owns, and set the status
    // word.  Neither ring ever holds more than its stages, so the fills in
    // flight are those from the drain position to the fill position.
    __device__ __forceinline__ void abandon(int* status, int nfwd, int npos) {
        for (; nfwd > 0; --nfwd, drainr.next(stages)) wait(bar_s, drainr, kDefaultWaitPolls);
        for (; npos > 0; --npos, pdrainr.next(kTmaPosStages)) wait(bar_s + 8 * kTmaMaxStages, pdrainr, kDefaultWaitPolls);
        if (lane == 0) {
            *(volatile int*)status = 1;
            __threadfence_system();
        }
    }
};

// 1 / d correctly rounded, for 2^-125 <= |d| <= 2^125: the hardware's approximate
// reciprocal and one Newton step on its exact remainder (P. Markstein, IA-64 and
// Elementary Functions, 2000, ch. 3; the exhaustive comparison with __frcp_rn
// over every such float32 is sb_debug_rcp_f32).  Unlike __frcp_rn it has no
// branch, so the levels of a block are one basic block and their shared loads
// and independent arithmetic overlap the recurrence.
constexpr float kRcpLo = 0x1p-125f, kRcpHi = 0x1p125f;
__device__ __forceinline__ float rcp_in_range(float d) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return __fmaf_rn(y, __fmaf_rn(-d, y, 1.0f), y);
}

// Solve `v` (its first `stages` level blocks are in the ring or on their
// way); `next` is the warp's next solve, `FillNext(blk)` fills its block.
// stage0: stage(k = 0) of this lane's column, on return that of `next`.
// Factors of block b: registers for the last block, TMEM columns tcol + 16 * b
// for b < nt, else shared memory fmem + (b - nt) * 2 KB.  Returns false when a wait gave up: nothing is in the
// rings then.
template <class S, int R, class FillNext>
__device__ __forceinline__ bool vadv_tma_solve(TmaPipe<S, R>& pipe, const TmaSolve<S>& v, const TmaSolve<S>& next,
                                               FillNext&& fill_next, float& stage0, uint32_t tcol, int nt, float* fmem, int* status) {
    using A = Ar<float>;
    using B = TmaBox<S, R>;
    constexpr int L = kTmaLevels;
    const float dtr = konst<float>(3.0 / 20.0);
    const int lane = pipe.lane, nk = v.nk, nblk = v.blocks();
    // this lane's element of each field's box, before the stage's and the row's offset
    const int drift = R < 0 ? v.drift : R;
    int el[kTmaFields + 1];
#pragma unroll
    for (int f = 0; f < kTmaFields; ++f) el[f] = f * B::BOXB + ((v.x[f] & (B::EPG - 1)) + lane) * B::ES;
    el[kTmaFields] = v.wsh > 1 ? kTmaFields * B::BOXB + ((v.x[kTmaFields] & (B::EPG - 1)) + lane) * B::ES
                               : el[0] + v.wsh * B::ES;
    auto rd = [&](const unsigned char* st, int f, int q) -> float {  // field f at level q of the stage
        return cvt<float, S>(*reinterpret_cast<const S*>(st + el[f] + q * (B::ROWB + drift)));
    };
#pragma unroll
    for (int q = 0; q < kTmaPosStages; ++q) pipe.fill_pos(v, nblk - 1 - q);

    // ---- forward sweep
    float cs = 0.f, sprev = 0.f, scur = stage0, cp = 0.f, dp = 0.f, plast = 0.f;
    float fac[2 * L];
    float dlo, dhi;  // magnitudes of the pivots since they were reset
    auto level = [&](const unsigned char* st, int q, auto in_range) {  // 0 < k < nk - 1
        const float w1 = rd(st, kTmaFields, q), w0 = rd(st, 0, q), snext = rd(st, 1, q);
        const float p0 = rd(st, 2, q), t0 = rd(st, 3, q), ts0 = rd(st, 4, q);
        const float csp = cs;  // cs(k-1) = -acol(k)
        cs = A::scale2<-1>(A::scale2<-2>(A::add(w1, w0)));
        const float ddown = A::sub(sprev, scur);
        const float dup = A::sub(snext, scur);
        const float bcol = A::sub(A::add(dtr, csp), cs);
        const float corr = A::sub(A::mul(csp, ddown), A::mul(cs, dup));
        const float dv = A::add(A::add(A::add(A::mul(dtr, p0), t0), ts0), corr);
        const float pivot = A::add(bcol, A::mul(cp, csp));
        float divided;
        if constexpr (decltype(in_range)::value) {
            divided = rcp_in_range(pivot);
            dlo = fminf(dlo, fabsf(pivot));
            dhi = fmaxf(dhi, fabsf(pivot));
        } else {
            divided = A::rcp(pivot);
        }
        cp = A::mul(cs, divided);
        dp = A::mul(A::add(dv, A::mul(dp, csp)), divided);
        sprev = scur;
        scur = snext;
        fac[2 * q] = cp;
        fac[2 * q + 1] = dp;
    };
    // levels q0 .. L-1 of a stage, none the last one: once more with the general
    // reciprocal where a lane met a pivot outside rcp_in_range's range
    auto levels = [&](const unsigned char* st, auto q0) {
        const float cs_ = cs, sprev_ = sprev, scur_ = scur, cp_ = cp, dp_ = dp;
        dlo = dhi = 1.0f;
#pragma unroll
        for (int q = decltype(q0)::value; q < L; ++q) level(st, q, std::true_type{});
        if (__any_sync(0xffffffffu, !(dlo >= kRcpLo && dhi <= kRcpHi))) {
            cs = cs_, sprev = sprev_, scur = scur_, cp = cp_, dp = dp_;
#pragma unroll
            for (int q = decltype(q0)::value; q < L; ++q) level(st, q, std::false_type{});
        }
    };
    for (int b = 0; b < nblk; ++b) {
        if (!pipe.ready()) {
            pipe.abandon(status, next.live ? (int)pipe.stages : min((int)pipe.stages, nblk - b), kTmaPosStages);
            return false;
        }
        const unsigned char* const st = pipe.stage();
        const int k0 = b * L;
        if (b == 0) {
            const float w1 = rd(st, kTmaFields, 0), w0 = rd(st, 0, 0), snext = rd(st, 1, 0);
            cs = A::scale2<-1>(A::scale2<-2>(A::add(w1, w0)));
            const float dup = A::sub(snext, scur);
            const float bcol = A::sub(dtr, cs);
            const float corr = A::mul(-cs, dup);
            const float dv = A::add(A::add(A::add(A::mul(dtr, rd(st, 2, 0)), rd(st, 3, 0)), rd(st, 4, 0)), corr);
            cp = A::div(cs, bcol);
            dp = A::div(dv, bcol);
            fac[0] = cp;
            fac[1] = dp;
            sprev = scur;
            scur = snext;
            levels(st, std::integral_constant<int, 1>{});
        } else if (k0 + L < nk) {
            levels(st, std::integral_constant<int, 0>{});
        } else {
            // the block of the last level; factors past it are never read
#pragma unroll
            for (int q = 0; q < L; ++q) {
                if (k0 + q < nk - 1) {
                    level(st, q, std::false_type{});
                } else if (k0 + q == nk - 1) {
                    const float bcol = A::add(dtr, cs);  // acol = -cs(nk-2)
                    const float corr = A::mul(cs, A::sub(sprev, scur));
                    plast = rd(st, 2, q);
                    const float dv = A::add(A::add(A::add(A::mul(dtr, plast), rd(st, 3, q)), rd(st, 4, q)), corr);
                    dp = A::div(A::add(dv, A::mul(dp, cs)), A::add(bcol, A::mul(cp, cs)));
                    fac[2 * q] = fac[2 * q + 1] = 0.f;
                } else {
                    fac[2 * q] = fac[2 * q + 1] = 0.f;
                }
            }
        }
        if (b == nblk - 1) {
            // the backward sweep starts with them
        } else if (b < nt) {
            tmem_st16(tcol + (uint32_t)(kTmaBlockCols * b), fac);
        } else {
#pragma unroll
            for (int q = 0; q < 2 * L; ++q) fmem[((b - nt) * 2 * L + q) * 32 + lane] = fac[q];
        }
        pipe.release(pipe.drainr, pipe.stages);
        const int ahead = b + (int)pipe.stages;
        if (ahead < nblk)
            pipe.fill(v, ahead);
        else if (next.live)
            fill_next(ahead - nblk);
    }
    tmem_wait_st();

    // ---- backward sweep
    if (next.live)
        stage0 = ld<float, S>(next.stage + next.col0 + min(lane, next.nvalid - 1));
    const bool valid = lane < v.nvalid;
    S* const out = v.out + v.col0 + lane;
    float data = dp;
    if (valid) st<S, float>(out + (nk - 1) * v.sk, A::mul(dtr, A::sub(data, plast)));
    uint32_t fr[2 * L];
#pragma unroll
    for (int q = 0; q < 2 * L; ++q) fr[q] = __float_as_uint(fac[q]);
    auto factors = [&](int b) {  // on their way into fr
        if (b < nt) {
            tmem_ld16_issue(tcol + (uint32_t)(kTmaBlockCols * b), fr);
        } else {
#pragma unroll
            for (int q = 0; q < 2 * L; ++q) fr[q] = __float_as_uint(fmem[((b - nt) * 2 * L + q) * 32 + lane]);
        }
    };
    for (int b = nblk - 1; b >= 0; --b) {
        if (!pipe.ready_pos()) {
            pipe.abandon(status, next.live ? (int)pipe.stages : 0, min(kTmaPosStages, b + 1));
            return false;
        }
        const unsigned char* const sp = pipe.stage_pos() - 2 * B::BOXB;  // as if a whole stage
        tmem_wait_ld(fr);
        float f[2 * L];
#pragma unroll
        for (int q = 0; q < 2 * L; ++q) f[q] = __uint_as_float(fr[q]);
        if (b > 0) factors(b - 1);  // while this block is solved
        const int k0 = b * L;
        const bool full = k0 + L < nk;
#pragma unroll
        for (int q = L - 1; q >= 0; --q) {
            if (full || k0 + q < nk - 1) {
                const float p0 = rd(sp, 2, q);
                data = A::sub(f[2 * q + 1], A::mul(f[2 * q], data));
                if (valid) st<S, float>(out + (k0 + q) * v.sk, A::mul(dtr, A::sub(data, p0)));
            }
        }
        pipe.release(pipe.pdrainr, kTmaPosStages);
        if (b >= kTmaPosStages) pipe.fill_pos(v, b - kTmaPosStages);
    }
    return true;
}

// ---- host side

// The maps of one component and their granule offsets: field f as a 2D tensor
// of (element offset in a level, level) based at the granule that holds its
// first element; wcon and stage start at level 1, as level k uses k + 1.  Every
// byte inside the tensor lies between the field's first and last element (or
// in their granules): x runs to the end of the last level, which lies drift
// bytes further right per level.  false where the driver refuses a map.
template <class S, int R>
inline bool encode_tma_maps(CUtensorMap* maps, int* off, const void* const (&field)[kTmaFields], int64_t ni, int64_t nj,
                     int64_t nk, int64_t sj, int64_t sk, int64_t wsh) {
    auto encode = tensor_map_encoder();
    if (!encode) return false;
    constexpr int ES = (int)sizeof(S);
    const int64_t drift = sk * ES % 16;
    for (int f = 0; f < kTmaFields; ++f) {
        const int first = f < 2 ? 1 : 0;
        const uintptr_t at = (uintptr_t)field[f] + (uintptr_t)(first * sk) * ES;
        off[f] = (int)((at & 15) / ES);
        const int64_t rows = nk - first, span = (ni - 1) + (nj - 1) * sj + 1 + (f == 0 ? wsh : 0);
        const cuuint64_t dims[2] = {(cuuint64_t)(off[f] + span + (rows - 1) * drift / ES), (cuuint64_t)rows};
        const cuuint64_t strides[1] = {(cuuint64_t)(sk * ES - drift)};
        const cuuint32_t box[2] = {(cuuint32_t)TmaBox<S, R>::W, (cuuint32_t)kTmaLevels};
        const cuuint32_t estride[2] = {1, 1};
        if (encode(&maps[f], tma_type<S>(), 2, (void*)(at & ~(uintptr_t)15), dims, strides, box, estride,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

// Warps per block, ring stages and TMEM blocks per warp of a solve of `ngroups`
// column groups on `sms` SMs.  Warps beyond what TMEM holds whole columns for
// keep their last level blocks in shared memory (137 levels: 8 warps instead of
// 4, 400x300 float32 99 us against 170 for the cp.async form's 4).  The fewest
// rounds win (a round is one column group per warp), then three stages over two
// (512x512x80: the same, 0-2%), then the fewest warps that keep the number of
// rounds, as they share the SM with fewer others.
struct TmaShape {
    int warps, stages, nt, warp_bytes;
    bool operator==(const TmaShape& o) const {
        return warps == o.warps && stages == o.stages && nt == o.nt && warp_bytes == o.warp_bytes;
    }
};
// min_nk: levels of the shortest column that the launch solves; max_warps: warps per block at most.
template <class S, int R>
inline TmaShape tma_shape(bool far, int64_t nk, int64_t min_nk, int64_t ngroups, int max_warps, int sms, int smem_optin) {
    using B = TmaBox<S, R>;
    const int nblk = (int)ceil_div(nk, (int64_t)kTmaLevels);
    TmaShape best{0, 0, 0, 0};
    int64_t best_rounds = 0;
    for (int stages = kTmaMaxStages; stages >= 2; --stages) {
        if (min_nk < tma_min_levels(stages)) continue;
        for (int quarter = 1; quarter <= 4; ++quarter) {  // warps that share a lane quarter of TMEM
            const int nt = std::min(nblk - 1, 512 / kTmaBlockCols / quarter);  // the last block's stay in registers
            const int bytes = B::rings_bytes(far, stages) + (nblk - 1 - nt) * kTmaBlockBytes;
            const int64_t fit = std::min<int64_t>(std::min(4 * quarter, max_warps), (smem_optin - 16 - 128) / (bytes + B::BAR_BYTES));
            if (fit < 1) continue;
            const int64_t rounds = ceil_div(ngroups, sms * fit);
            if (best.warps && rounds >= best_rounds) continue;
            best = {(int)ceil_div(ngroups, sms * rounds), stages, nt, bytes};
            best_rounds = rounds;
        }
    }
    return best;
}

}  // namespace sb
