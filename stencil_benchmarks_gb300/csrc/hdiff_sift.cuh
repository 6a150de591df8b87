// Horizontal diffusion, exact float64, that computes in fp64 only what the flux
// limiter lets through.
//
// GB300's fp64 pipe takes the same time for an instruction whatever the number
// of active lanes and is what bounds exact hdiff: 11 rounded operations per
// point.  But a flux whose sign equals that of the gradient is limited to zero,
// and most are (89% on uniform random fields, nearly all on smooth ones: the
// limited flux is the one against the gradient of a field whose Laplacian
// follows it).  A point whose four fluxes are zero keeps its value.  So a warp
//   1. reads a tile of inp into shared memory, stores it as the result and finds
//      the tile's largest exponent;
//   2. marches over the tile in 32-bit fixed point (unit 2^-27 of the largest
//      value) and closes every flux whose sign is certain and equals that of the
//      gradient; the others stay open;
//   3. computes the open fluxes exactly, 32 at a time in full warps, and limits
//      them with the exact test;
//   4. computes the points with an open flux exactly, likewise; one open flux
//      needs no sum, only the coefficient product and the update.
// Results are bit-identical to evaluating everything.
//
// When a flux may be closed.  With the unit u = 2^(E-1049), E the largest biased
// exponent, A = trunc(x / u) satisfies |A| < 2^27, so a fixed-point Laplacian is
// below 2^30 and a flux below 2^31 in magnitude, and they differ from the exact
// ones by less than 8 and 16 units; the fp64 evaluation rounds each Laplacian by
// less than 2^-20 units.  A fixed-point flux beyond +-kSiftSure therefore has
// the sign of the fp64 flux, which is then at least a unit.  Truncation is
// monotone, so different A(+1) and A have the sign of the fp64 difference, which
// is at least 2^-54 u.  The product of the two is positive and, for u >= 2^-500,
// does not underflow: the limiter makes the flux +0.
// When a point keeps its value: x - coeff * (+-0) is x unless coeff is not
// finite or x is -0.
// Tiles with an inf or nan, a value of 2^1017 or more, all values below 2^-474,
// a -0, a coefficient that is not finite, or more than kSiftCap open fluxes (a
// quarter) are computed in full (hdiff_dense_tile).  So is every tile where out
// is coeff itself (hdiff_in_place_tile): step 1 would overwrite the coefficients
// that step 4 reads; computed in full, each is read by the lane that then writes
// its point.
//
// 512x512x80, U[0, 1): 189 us against 547 for the TMA tile, which computes
// everything; 3.1 fp64 instructions per point instead of 11.6, that pipe 56% and
// the issue slots 71% busy.  128x128x64: 18.5 us against 36.7.  On other fields,
// 512x512x40, against the tile's 278 us: 105 on U[0, 1) and U[-1, 1), 91 on a
// smooth field, 116 to 163 on ramps with noise.  Where every tile is computed in
// full after all: 271 where half the fluxes pass, 282 on a smooth field with noise,
// 298 on a constant one (TMA tile 272), 338 on zeros with smooth blobs (328);
// 128x128x64, one wave of blocks, 42-52 (34-41).
#pragma once

#include "stencil_core.cuh"

namespace sb {

// Warps and rows of a tile, 512x512x80 / 128x128x64 in us: 1, 2, 3, 4 warps on 16
// rows 254 / 22.0, 198 / 21.3, 194 / 18.9, 195 / 18.7; 4 warps on 20, 24, 30 rows
// 189 / 18.9, 191 / 19.0, 202 / 20.8; 8 warps on 31 rows 226 / 22.7.  Longer tiles
// read fewer rows twice, but fewer of them fit an SM.
constexpr int kSiftWarps = 4;
constexpr int kSiftRows = 20;                 // output rows of a tile
constexpr int kSiftCols = 64, kSiftOut = 60;  // columns read and written
constexpr int kSiftSure = 17;                 // units beyond which a fixed-point flux has a certain sign
constexpr int kSiftCap = 640;                 // open fluxes of a tile at most

struct SiftTile {
    double x[(kSiftRows + 4) * kSiftCols];  // row t: j0 - 2 + t, column c: cs + c
    double flux[kSiftCap];
    alignas(16) uint32_t open[(kSiftRows + 1) * 4];    // per row j0 - 1 + r: open flx of even / odd columns, open fly of even / odd
    uint16_t first[(kSiftRows + 1) * 4];   // where each of these masks' fluxes start in flux[]
    uint16_t list[kSiftRows * kSiftOut];   // open fluxes (row * 128 + direction * 64 + column), later points (row * 64 + column)
    unsigned emax[kSiftWarps];             // per warp: largest exponent field, 2^32 - 1 where the tile must be computed in full
};

// x as an integer multiple of 2^(E-1049), truncated toward zero (E: the largest
// biased exponent; the shift is at least 5, and clamps at 32)
__device__ __forceinline__ int sift_fix(double x, int E) {
    const int hi = __double2hiint(x);
    const unsigned m = __funnelshift_l((unsigned)__double2loint(x), ((unsigned)hi & 0xfffffu) | 0x100000u, 11);
    unsigned a;
    asm("shr.u32 %0, %1, %2;" : "=r"(a) : "r"(m), "r"(E + 5 - ((hi >> 20) & 0x7ff)));
    const int s = hi >> 31;
    return ((int)a ^ s) - s;
}

// the limiter certainly makes the flux +0: same sign as the gradient d
__device__ __forceinline__ bool sift_closed(int flux, int d) {
    const int s = d >> 31;
    return d != 0 && (flux ^ s) - s > kSiftSure;
}

// Every point of the tile in fp64: the march of hdiff_vscan_strip with two columns
// per lane, on the tile's rows, which the warps divide: each piece computes the
// Laplacians of two rows and the fluxes of one more besides, so kSiftDenseWarps
// warps take long pieces, as these operations fill the pipe.  A tile of few columns
// (the last one along i) takes 8 or 16 lanes a row and 4 or 2 pieces a warp.
// Half the fluxes open, 512x512x40 / 128x128x64 in us: four warps 282 / 44.4, two
// 271 / 42.4, one 277 / 43.9.
constexpr int kSiftDenseWarps = 2;
template <class IDX>
__device__ __noinline__ void hdiff_dense_tile(const double* tile, const double* __restrict__ coeff, double* __restrict__ out,
                                              int whi, IDX si, IDX sj, IDX base, int warp, int lane, int nrow) {
    using A = Ar<double>;
    const int across = whi - 2 <= 12 ? 8 : whi - 2 <= 28 ? 16 : 32;  // lanes of a row
    const int pieces = kSiftDenseWarps * (32 / across), piece = (nrow + pieces - 1) / pieces;
    const int r0 = (warp * (32 / across) + lane / across) * piece, n = min(piece, nrow - r0);
    if (warp * (32 / across) * piece >= nrow) return;  // whole warp
    const int c0 = 2 * (lane % across);
    auto row = [&](int t, double(&o)[2]) {  // row r0 + t of the tile
        const double2 v = *reinterpret_cast<const double2*>(tile + min(r0 + t, nrow + 3) * kSiftCols + c0);
        o[0] = v.x;
        o[1] = v.y;
    };
    // (lanes at the edge of a piece see the next piece's values; no written column depends on them)
    auto lap_row = [&](const double(&b)[2], const double(&c)[2], const double(&a)[2], double(&o)[2], double& right) {
        const double left = shfl_up(c[1], 1);
        right = shfl_down(c[0], 1);
        o[0] = A::sub(A::scale2<2>(c[0]), A::add(A::add(A::add(c[1], left), a[0]), b[0]));
        o[1] = A::sub(A::scale2<2>(c[1]), A::add(A::add(A::add(right, c[0]), a[1]), b[1]));
    };
    double below[2], a0[2], a1[2], a2[2], lap_m1[2], lap0[2], lap1[2], fly_m1[2], rnb0, rnb1;
    row(0, below);
    row(1, a0);
    row(2, a1);
    row(3, a2);
    lap_row(below, a0, a1, lap_m1, rnb0);
    lap_row(a0, a1, a2, lap0, rnb0);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        fly_m1[q] = A::limit(A::sub(lap0[q], lap_m1[q]), a1[q], a0[q]);
        a0[q] = a1[q];
        a1[q] = a2[q];
    }
    for (int r = 0; r < piece; ++r) {
        row(r + 4, a2);
        lap_row(a0, a1, a2, lap1, rnb1);
        const double lapR = shfl_down(lap0[0], 1);
        double fly0[2], flx0[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            fly0[q] = A::limit(A::sub(lap1[q], lap0[q]), a1[q], a0[q]);
            flx0[q] = A::limit(A::sub(q ? lapR : lap0[1], lap0[q]), q ? rnb0 : a0[1], a0[q]);
        }
        const double flxL = shfl_up(flx0[1], 1);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int c = c0 + q;
            if (r < n && c >= 2 && c < whi) {
                const IDX o = base + (IDX)c * si + (IDX)(r0 + r) * sj;
                const double d = A::sub(A::add(A::sub(flx0[q], q ? flx0[0] : flxL), fly0[q]), fly_m1[q]);
                out[o] = A::sub(a0[q], A::mul(__ldg(coeff + o), d));
            }
            a0[q] = a1[q];
            a1[q] = a2[q];
            lap0[q] = lap1[q];
            fly_m1[q] = fly0[q];
        }
        rnb0 = rnb1;
    }
}

// A tile of hdiff_sift_tile's shape where out is coeff.  A function of its own: a
// run-time condition on the store in hdiff_sift_tile's first step made every call
// slower (512x512x80: 254 us instead of 189).
template <int NW, class IDX>
__device__ __noinline__ void hdiff_in_place_tile(SiftTile& s, const double* __restrict__ inp, double* out, int ni, int nj,
                                                 IDX si, IDX sj, IDX sk, int cs, int j0, int k, int warp, int lane) {
    const int nrow = min(kSiftRows, nj - j0);
    const IDX base = (IDX)k * sk + (IDX)cs * si + (IDX)j0 * sj;
    for (int t = warp; t < nrow + 4; t += NW)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = lane + 32 * h;
            s.x[t * kSiftCols + c] = cs + c <= ni + 1 ? __ldg(inp + (base + (IDX)c * si + (IDX)(t - 2) * sj)) : 0.0;
        }
    __syncthreads();
    if (warp < kSiftDenseWarps)
        hdiff_dense_tile<IDX>(s.x, out, out, min(2 + kSiftOut, ni - cs), si, sj, base, warp, lane, nrow);
}

// The NW warps of a block, columns [cs + 2, cs + 62) and rows [j0, j0 + 20) of plane k; out is not coeff.
template <int NW, class IDX>
__device__ __forceinline__ void hdiff_sift_tile(SiftTile& s, const double* __restrict__ inp,
                                                const double* __restrict__ coeff, double* __restrict__ out, int ni, int nj,
                                                IDX si, IDX sj, IDX sk, int cs, int j0, int k, int warp, int lane) {
    using A = Ar<double>;
    constexpr int TY = kSiftRows, W = kSiftCols;
    const int nrow = min(TY, nj - j0);
    const IDX base = (IDX)k * sk + (IDX)cs * si + (IDX)j0 * sj;  // of tile column 0, row j0
    const int whi = min(2 + kSiftOut, ni - cs);                  // written columns: [2, whi)

    // ---- 1: the tile, its largest exponent, the values as the result
    unsigned emax = 0;
    {
        unsigned negzero = ~0u, cmax = 0;
#pragma unroll 4
        for (int t = warp; t < nrow + 4; t += NW) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                const IDX o = base + (IDX)c * si + (IDX)(t - 2) * sj;
                const double x = cs + c <= ni + 1 ? __ldg(inp + o) : 0.0;
                s.x[t * W + c] = x;
                const unsigned hi = (unsigned)__double2hiint(x);
                emax = max(emax, hi & 0x7ff00000u);
                negzero = min(negzero, (hi ^ 0x80000000u) | (unsigned)__double2loint(x));
                if (t >= 2 && t < nrow + 2 && c >= 2 && c < whi) {
                    cmax = max(cmax, (unsigned)__double2hiint(__ldg(coeff + o)) & 0x7fffffffu);
                    out[o] = x;
                }
            }
        }
        emax = __reduce_max_sync(0xffffffffu, emax);
        if (__any_sync(0xffffffffu, negzero == 0u || cmax >= 0x7ff00000u)) emax = ~0u;
        if (lane == 0) s.emax[warp] = emax;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NW; ++w) emax = max(emax, s.emax[w]);
    const bool plain = emax >= (549u << 20) && emax < (2040u << 20);

    // ---- 2: which fluxes stay open, row r standing for j0 - 1 + r; each warp takes a piece of the rows
    if (plain) {
        const int E = (int)(emax >> 20), c0 = 2 * lane;
        const double2* rows = reinterpret_cast<const double2*>(s.x) + lane;
        auto fix_row = [&](int t, int(&o)[2]) {
            const double2 v = rows[t * (W / 2)];
            o[0] = sift_fix(v.x, E);
            o[1] = sift_fix(v.y, E);
        };
        const bool vx0 = c0 >= 1 && c0 < whi, vx1 = c0 + 1 < whi;  // flx(c) feeds points c and c + 1
        const bool vy0 = c0 >= 2 && c0 < whi, vy1 = c0 >= 1 && c0 + 1 < whi;
        const int piece = (nrow + 1 + NW - 1) / NW, r0 = warp * piece, r1 = min(nrow + 1, r0 + piece);
        if (r0 < r1) {
            int am[2], a[2], ap[2], lm[2] = {0, 0};
            uint32_t x0m = 0, x1m = 0;
            fix_row(r0, am);
            fix_row(r0 + 1, a);
#pragma unroll 2
            for (int t = r0 + 1; t <= r1 + 1; ++t) {
                fix_row(t + 1, ap);
                const int left = __shfl_up_sync(0xffffffffu, a[1], 1), right = __shfl_down_sync(0xffffffffu, a[0], 1);
                const int l0 = 4 * a[0] - (a[1] + left + ap[0] + am[0]);
                const int l1 = 4 * a[1] - (right + a[0] + ap[1] + am[1]);
                const int lr = __shfl_down_sync(0xffffffffu, l0, 1);
                // flx of row r = t - 1, fly of row r = t - 2
                const uint32_t x0 = __ballot_sync(0xffffffffu, vx0 && !sift_closed(l1 - l0, a[1] - a[0]));
                const uint32_t x1 = __ballot_sync(0xffffffffu, vx1 && !sift_closed(lr - l1, right - a[1]));
                const uint32_t y0 = __ballot_sync(0xffffffffu, vy0 && !sift_closed(l0 - lm[0], a[0] - am[0]));
                const uint32_t y1 = __ballot_sync(0xffffffffu, vy1 && !sift_closed(l1 - lm[1], a[1] - am[1]));
                if (lane == 0 && t > r0 + 1)
                    *reinterpret_cast<uint4*>(s.open + 4 * (t - 2)) = t == 2 ? make_uint4(0u, 0u, y0, y1)  // row 0: fly only
                                                                             : make_uint4(x0m, x1m, y0, y1);
                x0m = x0;
                x1m = x1;
                lm[0] = l0;
                lm[1] = l1;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    am[q] = a[q];
                    a[q] = ap[q];
                }
            }
        }
    }
    __syncthreads();

    // ---- 3: the open fluxes; lane r has the masks of row r
    uint32_t open[4] = {0u, 0u, 0u, 0u};
    if (plain && lane <= nrow) {
        const uint4 m = *reinterpret_cast<const uint4*>(s.open + 4 * lane);
        open[0] = m.x;
        open[1] = m.y;
        open[2] = m.z;
        open[3] = m.w;
    }
    const int mine = __popc(open[0]) + __popc(open[1]) + __popc(open[2]) + __popc(open[3]);
    int sum = mine;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int v = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += v;
    }
    const int total = __shfl_sync(0xffffffffu, sum, 31);
    if (!plain || total > kSiftCap) {
        if (warp < kSiftDenseWarps) hdiff_dense_tile<IDX>(s.x, coeff, out, whi, si, sj, base, warp, lane, nrow);
        return;
    }
    if (total == 0) return;
    if (lane <= nrow && lane % NW == warp) {
        int at = sum - mine;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s.first[lane * 4 + q] = (uint16_t)at;
            for (uint32_t m = open[q]; m; m &= m - 1)
                s.list[at++] = (uint16_t)(lane * 128 + (q >> 1) * 64 + 2 * (__ffs((int)m) - 1) + (q & 1));
        }
    }
    __syncthreads();
    auto lap_at = [&](int c) {
        const double* x = s.x + c;
        return A::sub(A::scale2<2>(x[0]), A::add(A::add(A::add(x[1], x[-1]), x[W]), x[-W]));
    };
    for (int n0 = 32 * warp; n0 < total; n0 += 32 * NW) {
        const int n = n0 + lane, code = s.list[min(n, total - 1)];
        const int a0 = (code >> 7) * W + W + (code & 63), a1 = a0 + ((code & 64) ? W : 1);
        const double f = A::limit<true>(A::sub(lap_at(a1), lap_at(a0)), s.x[a1], s.x[a0]);
        if (n < total) s.flux[n] = f;
    }
    __syncthreads();

    // ---- 4: the points that have an open flux, those with one first
    const uint32_t fy0 = __shfl_up_sync(0xffffffffu, open[2], 1), fy1 = __shfl_up_sync(0xffffffffu, open[3], 1);
    const uint32_t w0 = __ballot_sync(0xffffffffu, 2 * lane >= 2 && 2 * lane < whi);
    const uint32_t w1 = __ballot_sync(0xffffffffu, 2 * lane >= 1 && 2 * lane + 1 < whi);
    uint32_t one[2] = {0u, 0u}, more[2] = {0u, 0u};
    if (lane >= 1 && lane <= nrow) {
        auto split = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t w, uint32_t& single, uint32_t& multi) {
            multi = ((a & b) | (c & d) | ((a | b) & (c | d))) & w;
            single = (a | b | c | d) & w & ~multi;
        };
        split(open[0], open[1] << 1, open[2], fy0, w0, one[0], more[0]);
        split(open[1], open[0], open[3], fy1, w1, one[1], more[1]);
    }
    // both counts scanned at once: at most 960 each
    const int counts = __popc(one[0]) + __popc(one[1]) + ((__popc(more[0]) + __popc(more[1])) << 16);
    sum = counts;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int v = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += v;
    }
    const int all = __shfl_sync(0xffffffffu, sum, 31), nsingle = all & 0xffff, nmulti = all >> 16;
    if (lane % NW == warp) {
        int at = (sum - counts) & 0xffff, am = nsingle + ((sum - counts) >> 16);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            for (uint32_t m = one[q]; m; m &= m - 1) s.list[at++] = (uint16_t)(lane * 64 + 2 * (__ffs((int)m) - 1) + q);
            for (uint32_t m = more[q]; m; m &= m - 1) s.list[am++] = (uint16_t)(lane * 64 + 2 * (__ffs((int)m) - 1) + q);
        }
    }
    __syncthreads();
    // position in flux[] of bit b of mask `slot`
    auto flux_at = [&](int slot, int b) { return s.flux[s.first[slot] + __popc(s.open[slot] & ((1u << b) - 1u))]; };
    for (int n0 = 32 * warp; n0 < nsingle; n0 += 32 * NW) {
        const int n = n0 + lane, code = s.list[min(n, nsingle - 1)];
        const int r = code >> 6, c = code & 63, odd = c & 1, b = c >> 1, bl = b - 1 + odd;  // bl: bit of column c - 1
        const IDX o = base + (IDX)c * si + (IDX)(r - 1) * sj;
        const double cf = __ldg(coeff + o);
        const bool right = (s.open[r * 4 + odd] >> b) & 1u, leftf = (s.open[r * 4 + (odd ^ 1)] >> bl) & 1u;
        const bool up = (s.open[r * 4 + 2 + odd] >> b) & 1u;
        const int slot = right ? r * 4 + odd : leftf ? r * 4 + (odd ^ 1) : up ? r * 4 + 2 + odd : (r - 1) * 4 + 2 + odd;
        const double f = flux_at(slot, leftf && !right ? bl : b);
        const double d = right || (up && !leftf) ? f : A::neg(f);
        const double v = A::sub(s.x[(r + 1) * W + c], A::mul(cf, d));
        if (n < nsingle) out[o] = v;
    }
    // (the last warp first, so that the remainders of the two loops meet different warps)
    for (int n0 = 32 * (NW - 1 - warp); n0 < nmulti; n0 += 32 * NW) {
        const int n = n0 + lane, code = s.list[nsingle + min(n, nmulti - 1)];
        const int r = code >> 6, c = code & 63, odd = c & 1, b = c >> 1, bl = b - 1 + odd;
        const IDX o = base + (IDX)c * si + (IDX)(r - 1) * sj;
        const double cf = __ldg(coeff + o);
        auto flux_or_zero = [&](int slot, int bit) { return ((s.open[slot] >> bit) & 1u) ? flux_at(slot, bit) : 0.0; };
        const double fx1 = flux_or_zero(r * 4 + odd, b), fx0 = flux_or_zero(r * 4 + (odd ^ 1), bl);
        const double fy1_ = flux_or_zero(r * 4 + 2 + odd, b), fy0_ = flux_or_zero((r - 1) * 4 + 2 + odd, b);
        const double d = A::sub(A::add(A::sub(fx1, fx0), fy1_), fy0_);
        const double v = A::sub(s.x[(r + 1) * W + c], A::mul(cf, d));
        if (n < nmulti) out[o] = v;
    }
}

}  // namespace sb
