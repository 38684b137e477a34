// Sifting kernels of the ICEEMDAN engine (sm_100a, FP64).
//
// One sift iteration over all realizations of a stage is:
//   k_tile_knots     strict extrema of every tile (find_extrema_shfl_* :93-148,
//                    select_extrema_* :151-207), the knots' slopes and the end relations of the
//                    chunks of the canonical partitioned spline solve (tridiagonal_setup
//                    :311-343); knot bitmaps and the rows of the separator system are written
//   k_spline_solve   per spline: scan of the tile counts (CUB scan :1582-1604), end-knot
//                    extrapolation where it spans tiles (setBoundaryMax/Min :210-291), the
//                    separator system (with the tile kernels: cusparseDgtsv2_nopivot :1622-1641)
//   k_tile_sift      chunk interiors and segment coefficients (spline_coefficients :383-401),
//                    envelopes, mean envelope, sx statistics (interpolate :404-439,
//                    averageUppperLower :442-454, produceSX :457-467, thresholdJudge :470-492),
//                    the update h -= m (updateRealizations :528-544), and after a row's last
//                    tile its stop test (meanD/multiplyD on sx :1851, siftingCriterion :495-525,
//                    checkBreak :547-580)
// Spline values and coefficients live in shared memory only; k_tile_knots hands the knots'
// positions and slopes over.  An iteration moves 8 N bytes in k_tile_knots and 24 N in k_tile_sift
// (h, next h, mean envelope) plus N/2 of bitmaps, and per knot 20 bytes of positions and slopes
// and about 6 of separator rows.  Line numbers refer to the reference's cudaICEEMDAN.cu.
#include <cuda_runtime.h>

#include <cstdint>

#include "canon.cuh"
#include "kernels.h"
#include "spline_device.cuh"

namespace ceemdan {

namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = kTileSamples / kTileThreads;  // samples per thread in a tile
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kWarpSamples = 32 * kPerThread;
// a thread's samples in the knot bitmaps
using TileBits = unsigned short;
static_assert(8 * sizeof(TileBits) == kPerThread, "one bit per sample");
constexpr int kWords = kTileSamples / 32;            // bitmap words per tile (64)

// ---------------------------------------------------------------------------------------
// Geometry of the ragged multi-channel layout (kernels.h: Chan, SiftArgs).
// ---------------------------------------------------------------------------------------
struct Geo {
    int c, r, g;       // channel, realization within the channel, global row
    int n, ntiles;     // samples and tiles of the row
    int tile0;         // first global tile of the row
    size_t base;       // first sample of the row in the padded planes (h, mean envelope)
};

__device__ __forceinline__ Geo geo(const SiftArgs& a, int c, int r) {
    Geo q;
    if (a.nchan == 1) {  // channel 0's geometry from the launch parameters
        q.c = 0;
        q.r = r;
        q.g = r;
        q.n = a.n1;
        q.ntiles = a.ntiles1;
        q.tile0 = r * a.ntiles1;
        q.base = (size_t)r * (size_t)row_ld(a.n1);
        return q;
    }
    const Chan* ch = a.chan + c;
    q.c = c;
    q.r = r;
    q.n = __ldg(&ch->n);
    q.ntiles = __ldg(&ch->ntiles);
    q.g = __ldg(&ch->row0) + r;
    q.tile0 = __ldg(&ch->tile0) + r * q.ntiles;
    q.base = (size_t)__ldg(&ch->samp0) + (size_t)r * (size_t)row_ld(q.n);
    return q;
}

// last channel c with pre[c] <= v (pre: nondecreasing exclusive prefix, pre[0] = 0): the
// channel whose range [pre[c], pre[c+1]) holds v
__device__ __forceinline__ int plan_find(const int* pre, int nchan, int v) {
    int lo = 0, hi = nchan - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(pre + mid) <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Rows and tiles of the channels that sift in this iteration.
__device__ __forceinline__ int active_rows(const SiftArgs& a) {
    if (a.nchan == 1) return a.cs[0].done ? 0 : a.nr1;
    return __ldg(a.plan + a.nchan);
}
__device__ __forceinline__ int active_tiles(const SiftArgs& a) {
    if (a.nchan == 1) return a.cs[0].done ? 0 : a.nr1 * a.ntiles1;
    return __ldg(a.plan + 2 * a.nchan + 1);
}

// Active row v -> its geometry.
__device__ __forceinline__ Geo row_geo(const SiftArgs& a, int v) {
    if (a.nchan == 1) return geo(a, 0, v);
    const int c = plan_find(a.plan, a.nchan, v);
    return geo(a, c, v - __ldg(a.plan + c));
}

// Active tile v -> the geometry of its row and its tile index t within the row.
__device__ __forceinline__ Geo tile_geo(const SiftArgs& a, int v, int& t) {
    int c = 0, local = v;
    if (a.nchan > 1) {
        const int* pt = a.plan + a.nchan + 1;
        c = plan_find(pt, a.nchan, v);
        local = v - __ldg(pt + c);
    }
    const int nt = a.nchan == 1 ? a.ntiles1 : __ldg(&a.chan[c].ntiles);
    const int r = local / nt;
    t = local - r * nt;
    return geo(a, c, r);
}

// Active spline v (the maxima splines of the ra active rows, then their minima splines).
__device__ __forceinline__ Geo spline_geo(const SiftArgs& a, int v, int ra, int& e) {
    e = v >= ra ? 1 : 0;
    return row_geo(a, v - e * ra);
}

// Index of tile t of row q's spline e in the per-tile arrays (tile_cnt, bitmap words / 64, lists,
// headers, edges, separator rows), and of the row's first tile in the arrays with one entry more a
// row (sep_off, tile_rank, tile_list).
__device__ __forceinline__ size_t tix(const SiftArgs& a, int e, const Geo& q, int t) {
    return (size_t)e * a.ntot + (size_t)(q.tile0 + t);
}
__device__ __forceinline__ size_t oix(const SiftArgs& a, int e, const Geo& q) {
    return (size_t)e * (size_t)(a.ntot + a.nrows) + (size_t)(q.tile0 + q.g);
}
__device__ __forceinline__ int spline_id(const SiftArgs& a, int e, const Geo& q) {
    return e * a.nrows + q.g;
}
// record / separator-value offset and reduced-workspace offset of row q's spline e
__device__ __forceinline__ size_t rec_base(const SiftArgs& a, int e, const Geo& q) {
    if (a.nchan == 1) return (size_t)e * (size_t)a.rec_total + (size_t)q.r * (size_t)a.rs1;
    const Chan* ch = a.chan + q.c;
    return (size_t)e * (size_t)a.rec_total + (size_t)__ldg(&ch->rec0) +
           (size_t)q.r * (size_t)__ldg(&ch->rec_stride);
}
__device__ __forceinline__ size_t red_base(const SiftArgs& a, int e, const Geo& q) {
    if (a.nchan == 1)
        return (size_t)e * (size_t)a.red_total + (size_t)q.r * (size_t)red_stride_of(a.rs1);
    const Chan* ch = a.chan + q.c;
    return (size_t)e * (size_t)a.red_total + (size_t)__ldg(&ch->red0) +
           (size_t)q.r * (size_t)red_stride_of(__ldg(&ch->rec_stride));
}

// Entry of k_tile_sift's arrays where the segment of a sample with r knots before it in the tile
// starts: the knot before the tile at 0, in-tile knot m at 2 + kq(m).  An envelope's entries start
// kLead past a multiple of eight, so that its list of in-tile knots starts at one (the 16-byte
// copies of the positions).
__device__ __forceinline__ int seg_at(int r) { return r + ((r + 15) >> 4); }
constexpr int kLead = 6;
// With both envelopes there: where envelope 1's entries start, and the entries that takes (the
// copies round up to eight), given the most knots a tile of the row has.
__device__ __forceinline__ int sift_base1(int cm0) { return kLead + ((seg_at(cm0 + 1) + 8) & ~7); }
__device__ __forceinline__ int sift_need(int cm0, int cm1) {
    return sift_base1(cm0) + seg_at(cm1 + 1) + 8;
}

// Four doubles to a 32-byte aligned address, as one access.
__device__ __forceinline__ void store4(double* p, const double* v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
                 "d"(v[2]), "d"(v[3])
                 : "memory");
}

// The tile kernels run as persistent CTAs: CTA b works on the b-th of gridDim.x contiguous ranges
// of the active tiles, and copies the next tile's samples to shared memory while it computes on
// the current one.  TileIter walks the range; mark and par are the row's (loaded once a row).
// kList: the rows of k_tile_sift's class cls, as k_spline_solve listed them (contiguous ranges of
// all rows would leave most CTAs idle while a few work on the rows of the other class).
template <bool kList, int cls>
struct TileIter {
    int v, end;  // active tile, end of the range
    int tile;
    int cm;      // knots of the row's densest tile (of the envelope whose list the thread fetches)
    int base1;   // k_tile_sift: envelope 1's entries when both envelopes are there at once
    unsigned flags;  // above four bits of the row: its position in the list (kList)
    Geo q;
    __device__ __forceinline__ void row(const SiftArgs& a) {
        if (kList) {
            const int4 w = a.cls_row[(size_t)cls * a.nrows + (flags >> 4)];
            q = geo(a, w.x, w.y);
            tile = v - w.z;
        } else {
            q = tile_geo(a, v, tile);
        }
        const int cm0 = a.cmax[q.g], cm1 = a.cmax[a.nrows + q.g];
        cm = threadIdx.x < kTileThreads / 2 ? cm0 : cm1;
        base1 = sift_base1(cm0);
        const int need = sift_need(cm0, cm1);
        flags = (flags & ~15u) | (a.par[q.g] != 0 ? 1u : 0u) | (a.mark[q.g] != 0 ? 2u : 0u) |
                (min(a.kcount[q.g], a.kcount[a.nrows + q.g]) > 3 ? 4u : 0u) |
                (need > kSiftDense ? 8u : 0u);
    }
    __device__ __forceinline__ explicit TileIter(const SiftArgs& a) {
        const unsigned long long word = kList ? a.cls_count[cls] : 0ull;
        const int total = kList ? (int)(word & 0xffffffffull) : active_tiles(a);
        v = (int)((long long)total * blockIdx.x / gridDim.x);
        end = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
        tile = cm = base1 = 0;
        flags = 0u;
        if (v >= end) return;
        if (kList) {  // the last row that starts at v or before: 32 of them a look
            const int lane = threadIdx.x & 31;
            int pos = 0;
            for (int n = (int)(word >> 32); n > 1;) {
                const int step = (n + 31) >> 5, i = lane * step;
                const bool le = i < n && a.cls_row[(size_t)cls * a.nrows + pos + i].z <= v;
                const int last = (31 - __clz(__ballot_sync(0xffffffffu, le))) * step;
                pos += last;
                n = min(step, n - last);
            }
            flags = (unsigned)pos << 4;
        }
        row(a);
    }
    __device__ __forceinline__ int par() const { return (int)(flags & 1u); }
    __device__ __forceinline__ bool live() const { return flags & 2u; }  // else: repeats
    // averageUppperLower: the mean envelope keeps its previous value unless both envelopes have
    // more than 3 knots
    __device__ __forceinline__ bool mean() const { return flags & 4u; }
    // k_tile_sift: more entries than the dense form has
    __device__ __forceinline__ bool two() const { return flags & 8u; }
    __device__ __forceinline__ bool more() const { return v < end; }
    __device__ __forceinline__ void next(const SiftArgs& a) {
        ++v;
        if (++tile == q.ntiles) {
            if (kList) flags += 16u;
            if (v < end) row(a);
        }
    }
    // past the rest of the row while it does not satisfy pred
    template <class Pred>
    __device__ __forceinline__ void to_row(const SiftArgs& a, Pred pred) {
        while (v < end && !pred(*this)) {
            v += q.ntiles - tile;
            if (kList) flags += 16u;
            if (v < end) row(a);
        }
    }
};

// The samples of a tile in shared memory, 16-byte piece u at stage_piece(u): a warp copies its
// own samples coalesced (pieces l, l + 32, ...), then thread t reads its consecutive pieces without
// bank conflicts.  Every warp stages and reads only its own pieces.
__device__ __forceinline__ int stage_piece(int u) { return u ^ ((u >> 3) & 7); }

__device__ __forceinline__ void stage_tile(double2* st, const double* h, int m, int tid) {
    const int u0 = (tid & ~31) * (kPerThread / 2) + (tid & 31);
    // 32 pieces on, the swizzle changes in its third bit only
    double2* const s0 = st + stage_piece(u0);
    double2* const s1 = st + (stage_piece(u0) ^ 4);
    const double* src = h + 2 * u0;
    if (m == kTileSamples) {
#pragma unroll
        for (int g = 0; g < kPerThread / 2; ++g) cp_async16((g & 1 ? s1 : s0) + 32 * g, src + 64 * g);
    } else {
        const int m4 = (m + 3) & ~3;  // rows are padded to a multiple of four samples
#pragma unroll
        for (int g = 0; g < kPerThread / 2; ++g)
            if (2 * (u0 + 32 * g) < m4) cp_async16((g & 1 ? s1 : s0) + 32 * g, src + 64 * g);
    }
}
// piece g of the thread's own samples (g < 8)
__device__ __forceinline__ double2* own_piece(double2* st, int tid, int g) {
    return st + ((kPerThread / 2 * tid + (tid & 7)) ^ g);
}
// sample j of the tile
__device__ __forceinline__ double staged(const double2* st, int j) {
    return reinterpret_cast<const double*>(st + stage_piece(j >> 1))[j & 1];
}
// the thread's samples (zeros past the row)
__device__ __forceinline__ void unstage_tile(double* h, double2* st, int m, int tid) {
#pragma unroll
    for (int g = 0; g < kPerThread / 2; ++g) {
        const double2 w = *own_piece(st, tid, g);
        h[2 * g] = w.x;
        h[2 * g + 1] = w.y;
    }
    if (m < kTileSamples) {
#pragma unroll
        for (int i = 0; i < kPerThread; ++i)
            if (kPerThread * tid + i >= m) h[i] = 0.0;
    }
}

// The chunk a thread sweeps, given the separators of the tile's two envelopes: the chunks of
// envelope 0, then envelope 1, on consecutive threads (at most 128).  k: the separator closing
// the chunk.
__device__ __forceinline__ bool sweep_lane(int tid, int ns0, int ns1, int& e, int& k) {
    const int m0 = max(ns0 - 1, 0), m1 = max(ns1 - 1, 0);
    e = tid >= m0 ? 1 : 0;
    k = tid - (e ? m0 : 0) + 1;
    return tid < m0 + m1;
}

// Shared memory of k_tile_knots: per envelope the knots' positions within the tile and the slopes
// of the segments starting at them (padded positions kq), and the tile's samples.  41.5 KB: five
// CTAs per SM.
struct KnotSmem {
    double s[2][kListSlots];
    double ex[2][3][kRowSlots];       // first-row end relations of chunk k
    double2 stage[kTileSamples / 2];  // the samples
    double halo[kTileWarps][2];       // each warp's neighbours
    double yend[2][2];                // the row's end values
    alignas(16) short x[2][kListSlots];
};
static_assert(kListSlots % 8 == 0 &&
                  kListSlots >= kTileSamples / 2 + 1 + (kTileSamples / 2 + 1) / kChunk + 1,
              "a tile's knots of one envelope, padded, in 16-byte pieces");

}  // namespace

size_t tile_knots_smem() { return sizeof(KnotSmem); }

// =======================================================================================
// k_tile_knots: persistent CTAs over the 2048-sample tiles, both envelopes; thread t holds samples
// 16t..16t+15.  Strict extrema from the signs of neighbour differences, a bit each in the knot
// bitmaps; the knots compacted into shared memory; the segment slopes; the end relations of the
// chunks between separators (one thread per chunk) and from them the rows of the separator system
// inside the tile.  What the tile's first and last separators need from other tiles goes into the
// tile's header for k_spline_solve.
//
// Bound by instructions and the barriers between short phases (half of the issue slots used):
// sixteen samples to a thread share signs between neighbours and one scan step, where one sample
// to a lane took four times the instructions.  B200, N=244032 NR=100: 104 us at K/N = 0.18, 61 us
// at 0.001 (3.2 TB/s of its 8 N bytes), where the separate extrema, end-rule and chunk kernels took
// 178 us on average.  Six CTAs per SM instead of five change nothing.
//
// kExtrema: the knots alone (bitmaps, counts, headers' knots, end values), their values in place of
// the slopes in the lists, for the extrema entry.
// =======================================================================================
template <bool kExtrema>
__global__ void __launch_bounds__(kTileThreads, 5)
k_tile_knots(const __grid_constant__ SiftArgs a) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    KnotSmem& S = *reinterpret_cast<KnotSmem*>(dyn_smem);
    __shared__ int s_w[kTileWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && threadIdx.x < 2) a.cls_count[threadIdx.x] = 0ull;  // (k_spline_solve)
    using Iter = TileIter<false, 0>;
    Iter it(a);
    auto live = [](const Iter& t) { return t.live(); };
    auto prefetch = [&]() {
        if (!it.more()) return;
        const int n0 = it.tile * kTileSamples, left = it.q.n - n0;
        const double* h = a.h[it.par()] + it.q.base + n0;
        stage_tile(S.stage, h, min(kTileSamples, left), tid);
        const int j = warp * kWarpSamples;  // the neighbours of the warp's samples
        if (lane == 0 && n0 + j > 0 && j <= left) cp_async8(&S.halo[warp][0], h + j - 1);
        if (lane == 31 && j + kWarpSamples < left)
            cp_async8(&S.halo[warp][1], h + j + kWarpSamples);
    };
    it.to_row(a, live);
    prefetch();
    while (it.more()) {
    const Geo q = it.q;
    const int tile = it.tile;
    const int n0 = tile * kTileSamples;
    const int left = q.n - n0;               // samples of the row from the tile on
    const int m = min(kTileSamples, left);   // samples of the tile
    const int j0 = kPerThread * tid;
    cp_async_wait_all();
    __syncwarp();
    unsigned b0, b1;
    {
        double h[kPerThread + 1];
        unstage_tile(h, S.stage, m, tid);
        double nb = 0.0;
        if (lane == 0) nb = S.halo[warp][0];
        if (lane == 31) nb = S.halo[warp][1];
        h[kPerThread] = __shfl_down_sync(0xffffffffu, h[0], 1);
        if (lane == 31) h[kPerThread] = nb;
        unsigned rise = 0u, fall = 0u;  // bit i: h[i] < h[i+1], h[i] > h[i+1]
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            if (h[i] < h[i + 1]) rise |= 1u << i;
            if (h[i] > h[i + 1]) fall |= 1u << i;
        }
        unsigned before = (rise >> (kPerThread - 1)) | (fall >> (kPerThread - 1)) << 1;
        before = __shfl_up_sync(0xffffffffu, before, 1);
        if (lane == 0) before = (nb < h[0] ? 1u : 0u) | (nb > h[0] ? 2u : 0u);
        b0 = ((rise << 1) | (before & 1u)) & fall;
        b1 = ((fall << 1) | (before >> 1)) & rise;
    }
    b0 &= (1u << kPerThread) - 1u;
    b1 &= (1u << kPerThread) - 1u;
    // both end samples of the row are knots of both envelopes; none past the row
    if (n0 + j0 == 0) {
        b0 |= 1u;
        b1 |= 1u;
    }
    const int e1 = left - 1 - j0;  // bit of sample n-1
    if (e1 < kPerThread) {
        const unsigned in = e1 > 0 ? (1u << e1) - 1u : 0u, end = e1 >= 0 ? 1u << e1 : 0u;
        b0 = (b0 & in) | end;
        b1 = (b1 & in) | end;
    }
    reinterpret_cast<TileBits*>(a.bitmap + tix(a, 0, q, tile) * kWords)[tid] = (TileBits)b0;
    reinterpret_cast<TileBits*>(a.bitmap + tix(a, 1, q, tile) * kWords)[tid] = (TileBits)b1;
    // knots before the thread (both envelopes in one word): the warp's scan, and the other warps'
    // totals; k_tile_sift takes the warps' prefixes from the tile's TileScan
    const int own = __popc(b0) | __popc(b1) << 16;
    const int incl = warp_scan(own, lane);
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    int wb = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < kTileWarps; ++i) {
        if (i < warp) wb += s_w[i];
        tot += s_w[i];
    }
    if (lane == 0) {
        TileScan& sc = a.scan[q.tile0 + tile];
        sc.before[warp] = wb;
        if (warp == 0) sc.total = tot;
    }
    const int c0 = tot & 0xffff, c1 = tot >> 16;
    {
        const int ex = wb + incl - own;
        int p0 = ex & 0xffff, p1 = ex >> 16;
        // one knot of each envelope a turn: as many turns as the warp's fullest thread has knots
        unsigned w0 = b0, w1 = b1;
        while (w0 | w1) {
            if (w0) S.x[0][kq(p0++)] = (short)(j0 + __ffs(w0) - 1);
            if (w1) S.x[1][kq(p1++)] = (short)(j0 + __ffs(w1) - 1);
            w0 &= w0 - 1u;
            w1 &= w1 - 1u;
        }
    }
    __syncthreads();
    // End rule (setBoundaryMax/Min): applied here when the tile's own knots decide it (six or
    // more), else by k_spline_solve from the knots of several tiles.
    const bool first = tile == 0, last = tile == q.ntiles - 1;
    if (first || last) {
        if (tid < 64 && lane < 2) {
            const int e = tid >> 5, c = e ? c1 : c0, side = lane;
            const int sp = spline_id(a, e, q);
            const short* x = S.x[e];
            auto y = [&](int i) { return staged(S.stage, x[kq(i)]); };
            if (side == 0 ? first : last) {
                double v0 = side == 0 ? y(0) : y(c - 1);
                if (c >= 6) {
                    v0 = side == 0
                             ? boundary_left(e, x[0], x[1], x[2], y(0), y(1), y(2))
                             : boundary_right(e, x[kq(c - 3)], x[kq(c - 2)], x[kq(c - 1)],
                                              y(c - 3), y(c - 2), y(c - 1));
                } else {
                    for (int i = 0; i < c; ++i) {
                        a.end_x[(size_t)(2 * sp + side) * kEndKnots + i] = n0 + x[kq(i)];
                        a.end_y[(size_t)(2 * sp + side) * kEndKnots + i] = y(i);
                    }
                }
                a.yend[2 * sp + side] = S.yend[e][side] = v0;
            }
        }
        __syncthreads();
    }
    {
        constexpr int kHalf = kTileThreads / 2;  // threads per envelope
        const int e = tid / kHalf;
        const int c = e ? c1 : c0;
        const short* x = S.x[e];
        // value of knot i (at padded position p)
        auto y = [&](int i, int p) {
            double v = staged(S.stage, x[p]);
            if (first && i == 0) v = S.yend[e][0];
            if (last && i == c - 1) v = S.yend[e][1];
            return v;
        };
        // (the knots' own values where the slopes go)
        for (int i = tid % kHalf, p = kq(i); i < c && kExtrema; i += kHalf, p += kq(kHalf))
            S.s[e][p] = staged(S.stage, x[p]);
        // 16 knots on, the padded positions advance by 17; the segments at the row's ends take
        // the end values
        for (int i = tid % kHalf, p0 = kq(i), p1 = kq(i + 1); i + 1 < c && !kExtrema;
             i += kHalf, p0 += kq(kHalf), p1 += kq(kHalf)) {
            const int x0 = x[p0], x1 = x[p1];
            S.s[e][p0] = div_int(staged(S.stage, x1) - staged(S.stage, x0), (double)(x1 - x0));
        }
        for (int side = 0; side < 2 && !kExtrema; ++side) {
            const int i = side == 0 ? 0 : c - 2;  // written by the same thread above
            if ((side == 0 ? first : last) && c > 1 && tid % kHalf == i % kHalf)
                S.s[e][kq(i)] = div_int(y(i + 1, kq(i + 1)) - y(i, kq(i)),
                                        (double)(x[kq(i + 1)] - x[kq(i)]));
        }
        if (tid % kHalf == kHalf - 1) {
            if (c > 0) {
                TileHdr& hd = a.hdr[tix(a, e, q, tile)];
                const int i1 = c > 1 ? 1 : 0, pb = kq(c - 1), ia = c > 1 ? c - 2 : 0, pa = kq(ia);
                hd.x0 = n0 + x[0];
                hd.x1 = n0 + x[i1];
                hd.xa = n0 + x[pa];
                hd.xb = n0 + x[pb];
                hd.y0 = y(0, 0);
                hd.y1 = y(i1, i1);
                hd.ya = y(ia, pa);
                hd.yb = y(c - 1, pb);
            }
            a.tile_cnt[tix(a, e, q, tile)] = c;
        }
    }
    __syncthreads();
    // the samples are done with: the next tile's land during the sweeps
    const size_t sl0 = tix(a, 0, q, tile) * kListSlots, sl1 = tix(a, 1, q, tile) * kListSlots;
    it.next(a);
    it.to_row(a, live);
    prefetch();
    {  // the knots' positions and slopes for k_tile_sift, as they lie here
        const int e = warp >> 1, c = e ? c1 : c0, n = c > 0 ? kq(c - 1) + 1 : 0;
        const size_t sl = e ? sl1 : sl0;
        const int4* xs = reinterpret_cast<const int4*>(S.x[e]);
        const double2* ss = reinterpret_cast<const double2*>(S.s[e]);
        int4* xo = reinterpret_cast<int4*>(a.list_x + sl);
        double2* so = reinterpret_cast<double2*>(a.list_s + sl);
        for (int i = tid & 63; i < (n + 7) >> 3; i += kTileThreads / 2) xo[i] = xs[i];
        for (int i = tid & 63; i < (n + 1) >> 1; i += kTileThreads / 2) so[i] = ss[i];
    }
    if (kExtrema) continue;  // (the next tile's first barrier separates these reads, too)
    int e, k;
    const bool act = sweep_lane(tid, tile_seps(c0), tile_seps(c1), e, k);
    const int c = e ? c1 : c0;
    const int js = min(k * kChunk, c - 1);  // the separator's knot
    ChunkEnds ce;
    if (act) {
        const int jb = (k - 1) * kChunk;
        const int len = js - jb - 1;
        if (len > 0) {
            ce = chunk_ends_knots(S.x[e] + kq(jb), S.s[e] + kq(jb), len);
        } else {
            ce.ga = 0.0; ce.aa = 0.0; ce.ba = 1.0;
            ce.gb = 0.0; ce.ab = 1.0; ce.bb = 0.0;
        }
        S.ex[e][0][k] = ce.ga;
        S.ex[e][1][k] = ce.aa;
        S.ex[e][2][k] = ce.ba;
    }
    __syncthreads();
    if (act) {
        TileHdr& hd = a.hdr[tix(a, e, q, tile)];
        if (k == 1) {
            hd.ga = ce.ga;
            hd.aa = ce.aa;
            hd.ba = ce.ba;
        }
        if (js == c - 1) {
            hd.gb = ce.gb;
            hd.ab = ce.ab;
            hd.bb = ce.bb;
        } else {
            const int im = kq(js - 1), i0 = kq(js), ip = kq(js + 1);
            const Row sr = spline_row(S.x[e][im], S.x[e][i0], S.x[e][ip], S.s[e][im], S.s[e][i0]);
            const Row o = reduced_row(sr, ce.gb, ce.ab, ce.bb, S.ex[e][0][k + 1],
                                      S.ex[e][1][k + 1], S.ex[e][2][k + 1]);
            const double w[4] = {o.l, o.m, o.u, o.r};
            store4(a.rows + (tix(a, e, q, tile) * kRowSlots + k) * 4, w);
        }
    }
    // (the next tile's first barrier separates these reads of s, x and ex from its writes)
    }
}
template __global__ void k_tile_knots<false>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_knots<true>(const __grid_constant__ SiftArgs a);

// Compacted copy of the knots (stage-level entry point, one channel; blockIdx.z: envelope): row r's
// knots to kx/ky[r*n + i], from k_tile_knots<true>'s lists and the end values.  (From the bitmaps and
// the samples it took 97 us at N=244032 NR=50, from the lists 62, and k_tile_knots 50 instead of
// 35.)
__global__ void __launch_bounds__(kThreads)
k_gather_knots(const __grid_constant__ SiftArgs a, int32_t* kx_max, double* ky_max,
               int32_t* kx_min, double* ky_min) {
    __shared__ int s_before[kThreads / 32];
    const int e = blockIdx.z, tile = blockIdx.x, tid = threadIdx.x;
    const Geo q = geo(a, 0, blockIdx.y);
    int before = 0;  // knots of the tiles before this one
    for (int t = tid; t < tile; t += kThreads) before += a.tile_cnt[tix(a, e, q, t)];
    before = __reduce_add_sync(0xffffffffu, before);
    if ((tid & 31) == 0) s_before[tid >> 5] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) before += s_before[w];
    const int c = a.tile_cnt[tix(a, e, q, tile)], n0 = tile * kTileSamples;
    const short* x = a.list_x + tix(a, e, q, tile) * kListSlots;
    const double* y = a.list_s + tix(a, e, q, tile) * kListSlots;
    const double* yend = a.yend + 2 * spline_id(a, e, q);
    const size_t o = (size_t)q.r * q.n + before;
    int32_t* const kx = (e ? kx_min : kx_max) + o;
    double* const ky = (e ? ky_min : ky_max) + o;
#pragma unroll 4
    for (int m = tid; m < c; m += kThreads) {
        const int s = n0 + x[kq(m)];
        kx[m] = s;
        ky[m] = s == 0 ? yend[0] : (s == q.n - 1 ? yend[1] : y[kq(m)]);
    }
}

// =======================================================================================
// canonical partitioned solve of explicit systems
// =======================================================================================
namespace {

struct GlobalRowFn {
    const double *l, *m, *u, *r;
    int first;
    __device__ __forceinline__ Row operator()(int k) const {
        const int i = first + k;
        Row w;
        w.l = l[i];
        w.m = m[i];
        w.u = u[i];
        w.r = r[i];
        return w;
    }
};

// In-CTA canonical partitioned solve of an explicit system in global memory (its sweeps keep their
// factors in registers: a factor read back from memory would cost a round trip a row) stored at sys
// (4 planes of `plane` doubles: l, m, u, r), solution to x.  ws: workspace for the deeper levels
// (<= 0.75*n + 16 doubles).  All threads of the CTA must call it.
template <class Pivot>
__device__ void cta_partitioned_global(int n, const double* sys, int plane, double* x, double* ws) {
    int sizes[8];
    int depth = 0;
    sizes[0] = n;
    while (sizes[depth] > kChunk && depth < 7) {
        sizes[depth + 1] = (sizes[depth] - 1) / kChunk;
        ++depth;
    }
    const double* lv[8];
    double* xv[8];
    int off = 0;
    lv[0] = sys;
    for (int k = 1; k <= depth; ++k) {
        lv[k] = ws + off;
        off += 4 * sizes[k];
    }
    xv[0] = x;
    for (int k = 1; k <= depth; ++k) {
        xv[k] = ws + off;
        off += sizes[k];
    }
    double* ends = ws + off;  // 6 * (chunks of the widest level)
    for (int k = 0; k < depth; ++k) {
        const int nk = sizes[k];
        const int P = sizes[k + 1];
        const int pl = (k == 0) ? plane : nk;
        const double* L = lv[k];
        for (int q = threadIdx.x; q <= P; q += blockDim.x) {
            const int first = q * kChunk;
            const int len = (q < P) ? kChunk - 1 : nk - first;
            GlobalRowFn fn{L, L + pl, L + 2 * pl, L + 3 * pl, first};
            const ChunkEnds ce = chunk_ends<Pivot>(len, fn, NoIw());
            ends[6 * q + 0] = ce.ga;
            ends[6 * q + 1] = ce.aa;
            ends[6 * q + 2] = ce.ba;
            ends[6 * q + 3] = ce.gb;
            ends[6 * q + 4] = ce.ab;
            ends[6 * q + 5] = ce.bb;
        }
        __syncthreads();
        double* R = const_cast<double*>(lv[k + 1]);
        for (int p = threadIdx.x; p < P; p += blockDim.x) {
            const int s = p * kChunk + kChunk - 1;
            Row sr;
            sr.l = L[s];
            sr.m = L[pl + s];
            sr.u = L[2 * pl + s];
            sr.r = L[3 * pl + s];
            const Row o = reduced_row(sr, ends[6 * p + 3], ends[6 * p + 4], ends[6 * p + 5],
                                      ends[6 * (p + 1) + 0], ends[6 * (p + 1) + 1],
                                      ends[6 * (p + 1) + 2]);
            R[p] = o.l;
            R[P + p] = o.m;
            R[2 * P + p] = o.u;
            R[3 * P + p] = o.r;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const int nb = sizes[depth];
        const int pl = (depth == 0) ? plane : nb;
        const double* L = lv[depth];
        GlobalRowFn fn{L, L + pl, L + 2 * pl, L + 3 * pl, 0};
        thomas_small<Pivot>(nb, fn, xv[depth], 1);
    }
    __syncthreads();
    for (int k = depth - 1; k >= 0; --k) {
        const int nk = sizes[k];
        const int P = sizes[k + 1];
        const int pl = (k == 0) ? plane : nk;
        const double* L = lv[k];
        const double* Xs = xv[k + 1];
        double* xo = xv[k];
        for (int q = threadIdx.x; q <= P; q += blockDim.x) {
            const int first = q * kChunk;
            const int len = (q < P) ? kChunk - 1 : nk - first;
            GlobalRowFn fn{L, L + pl, L + 2 * pl, L + 3 * pl, first};
            const double xl = (q > 0) ? Xs[q - 1] : 0.0;
            const double xr = (q < P) ? Xs[q] : 0.0;
            chunk_interior<true, Pivot>(len, fn, xl, xr, xo + first, 1);
            if (q < P) xo[first + kChunk - 1] = xr;
        }
        __syncthreads();
    }
}

}  // namespace

__device__ void cta_spline_tridiag(int n, const double* sys, int plane, double* x, double* ws) {
    cta_partitioned_global<SplinePivot>(n, sys, plane, x, ws);
}

// ---------------------------------------------------------------------------------------
// The same canonical partitioned solve for many systems at once, one level per launch, the
// chunks of every system spread over the grid (blockIdx.y = system, x = chunk): system s has
// nrows[s] rows (0: skipped) at sys + 4*plane*s (planes l, m, u, r), solution to
// x + plane*s, deeper levels in ws + ws_stride*s with cta_partitioned_global's layout.  Every
// chunk performs its operations in the same order, so the solution is identical to
// cta_spline_tridiag's; the launches replace its in-CTA barriers.  For long systems whose one CTA
// would otherwise walk thousands of chunks.
// ---------------------------------------------------------------------------------------
namespace {

struct PLevels {
    int depth;
    int sizes[8];
    size_t lv[8], xv[8], ends;  // offsets into the system's workspace (lv[0], xv[0] unused)
};

// Level-0 rows of a spline system rebuilt from its knot positions and right-hand side (the
// adjoint's systems: identity end rows with zero right-hand side, interior rows
// l = x_i - x_{i-1}, m = 2(l + u), u = x_{i+1} - x_i): the values k_adj_rows stores in the
// l, m, u planes, read as 4 bytes per row instead of 24.
struct KnotSysRows {
    const int32_t* x;
    const double* r;
    int K, first;
    __device__ __forceinline__ Row operator()(int k) const {
        const int i = first + k;
        Row w;
        if (i == 0 || i == K - 1) {
            w.l = 0.0;
            w.m = 1.0;
            w.u = 0.0;
            w.r = 0.0;
        } else {
            const int dl = x[i] - x[i - 1], du = x[i + 1] - x[i];
            w.l = (double)dl;
            w.m = (double)(2 * (dl + du));
            w.u = (double)du;
            w.r = r[i];
        }
        return w;
    }
};

__device__ __forceinline__ PLevels plevels(int n) {
    PLevels v;
    v.depth = 0;
    v.sizes[0] = n;
    while (v.sizes[v.depth] > kChunk && v.depth < 7) {
        v.sizes[v.depth + 1] = (v.sizes[v.depth] - 1) / kChunk;
        ++v.depth;
    }
    size_t off = 0;
    for (int k = 1; k <= v.depth; ++k) {
        v.lv[k] = off;
        off += 4 * (size_t)v.sizes[k];
    }
    for (int k = 1; k <= v.depth; ++k) {
        v.xv[k] = off;
        off += (size_t)v.sizes[k];
    }
    v.ends = off;
    return v;
}

}  // namespace

__global__ void __launch_bounds__(kThreads)
k_psolve_ends(int k, const int* nrows, const double* sys, int plane, double* ws,
              size_t ws_stride, const int32_t* kx) {
    const int sidx = blockIdx.y;
    const int n = nrows[sidx];
    if (n <= 0) return;
    const PLevels v = plevels(n);
    if (k >= v.depth) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int nk = v.sizes[k], P = v.sizes[k + 1];
    if (q > P) return;
    double* w = ws + ws_stride * sidx;
    const double* L = k == 0 ? sys + (size_t)4 * plane * sidx : w + v.lv[k];
    const int pl = k == 0 ? plane : nk;
    const int first = q * kChunk;
    const int len = (q < P) ? kChunk - 1 : nk - first;
    const ChunkEnds ce =
        (k == 0 && kx) ? chunk_ends(len, KnotSysRows{kx + (size_t)plane * sidx, L + 3 * pl, n,
                                                     first}, NoIw())
                       : chunk_ends(len, GlobalRowFn{L, L + pl, L + 2 * pl, L + 3 * pl, first},
                                    NoIw());
    double* ends = w + v.ends;
    ends[6 * q + 0] = ce.ga;
    ends[6 * q + 1] = ce.aa;
    ends[6 * q + 2] = ce.ba;
    ends[6 * q + 3] = ce.gb;
    ends[6 * q + 4] = ce.ab;
    ends[6 * q + 5] = ce.bb;
}

__global__ void __launch_bounds__(kThreads)
k_psolve_rows(int k, const int* nrows, const double* sys, int plane, double* ws,
              size_t ws_stride, const int32_t* kx) {
    const int sidx = blockIdx.y;
    const int n = nrows[sidx];
    if (n <= 0) return;
    const PLevels v = plevels(n);
    if (k >= v.depth) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int nk = v.sizes[k], P = v.sizes[k + 1];
    if (p >= P) return;
    double* w = ws + ws_stride * sidx;
    const double* L = k == 0 ? sys + (size_t)4 * plane * sidx : w + v.lv[k];
    const int pl = k == 0 ? plane : nk;
    const double* ends = w + v.ends;
    const int s = p * kChunk + kChunk - 1;
    Row sr;
    if (k == 0 && kx) {
        sr = KnotSysRows{kx + (size_t)plane * sidx, L + 3 * pl, n, 0}(s);
    } else {
        sr.l = L[s];
        sr.m = L[pl + s];
        sr.u = L[2 * pl + s];
        sr.r = L[3 * pl + s];
    }
    const Row o = reduced_row(sr, ends[6 * p + 3], ends[6 * p + 4], ends[6 * p + 5],
                              ends[6 * (p + 1) + 0], ends[6 * (p + 1) + 1],
                              ends[6 * (p + 1) + 2]);
    double* R = w + v.lv[k + 1];
    R[p] = o.l;
    R[P + p] = o.m;
    R[2 * P + p] = o.u;
    R[3 * P + p] = o.r;
}

__global__ void __launch_bounds__(kThreads)
k_psolve_base(int nsys, const int* nrows, const double* sys, int plane, double* x, double* ws,
              size_t ws_stride, const int32_t* kx) {
    const int sidx = blockIdx.x * blockDim.x + threadIdx.x;
    if (sidx >= nsys) return;
    const int n = nrows[sidx];
    if (n <= 0) return;
    const PLevels v = plevels(n);
    double* w = ws + ws_stride * sidx;
    const int nb = v.sizes[v.depth];
    const double* L = v.depth == 0 ? sys + (size_t)4 * plane * sidx : w + v.lv[v.depth];
    const int pl = v.depth == 0 ? plane : nb;
    double* xo = v.depth == 0 ? x + (size_t)plane * sidx : w + v.xv[v.depth];
    if (v.depth == 0 && kx)
        thomas_small(nb, KnotSysRows{kx + (size_t)plane * sidx, L + 3 * pl, n, 0}, xo, 1);
    else
        thomas_small(nb, GlobalRowFn{L, L + pl, L + 2 * pl, L + 3 * pl, 0}, xo, 1);
}

__global__ void __launch_bounds__(kThreads)
k_psolve_back(int k, const int* nrows, const double* sys, int plane, double* x, double* ws,
              size_t ws_stride, const int32_t* kx) {
    const int sidx = blockIdx.y;
    const int n = nrows[sidx];
    if (n <= 0) return;
    const PLevels v = plevels(n);
    if (k >= v.depth) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int nk = v.sizes[k], P = v.sizes[k + 1];
    if (q > P) return;
    double* w = ws + ws_stride * sidx;
    const double* L = k == 0 ? sys + (size_t)4 * plane * sidx : w + v.lv[k];
    const int pl = k == 0 ? plane : nk;
    const double* Xs = w + v.xv[k + 1];
    double* xo = k == 0 ? x + (size_t)plane * sidx : w + v.xv[k];
    const int first = q * kChunk;
    const int len = (q < P) ? kChunk - 1 : nk - first;
    const double xl = (q > 0) ? Xs[q - 1] : 0.0;
    const double xr = (q < P) ? Xs[q] : 0.0;
    if (k == 0 && kx)
        chunk_interior(len, KnotSysRows{kx + (size_t)plane * sidx, L + 3 * pl, n, first}, xl,
                       xr, xo + first, 1);
    else
        chunk_interior(len, GlobalRowFn{L, L + pl, L + 2 * pl, L + 3 * pl, first}, xl, xr,
                       xo + first, 1);
    if (q < P) xo[first + kChunk - 1] = xr;
}

// Launch sequence of the level kernels for nsys systems of at most max_rows rows (kx: the
// systems' knot positions, plane-strided, when their level-0 rows are spline rows rebuilt from
// the knots and only the right-hand-side plane is stored; null: all four planes stored).
cudaError_t psolve_launch(int nsys, int max_rows, const int* nrows, const double* sys, int plane,
                          double* x, double* ws, size_t ws_stride, cudaStream_t st,
                          int* launches, const int32_t* kx) {
    int sizes[8], depth = 0;
    sizes[0] = max_rows;
    while (sizes[depth] > kChunk && depth < 7) {
        sizes[depth + 1] = (sizes[depth] - 1) / kChunk;
        ++depth;
    }
    int nl = 0;
    for (int k = 0; k < depth; ++k) {
        const dim3 g((unsigned)((sizes[k + 1] + 1 + kThreads - 1) / kThreads), (unsigned)nsys);
        k_psolve_ends<<<g, kThreads, 0, st>>>(k, nrows, sys, plane, ws, ws_stride, kx);
        k_psolve_rows<<<g, kThreads, 0, st>>>(k, nrows, sys, plane, ws, ws_stride, kx);
        nl += 2;
    }
    k_psolve_base<<<(unsigned)((nsys + kThreads - 1) / kThreads), kThreads, 0, st>>>(
        nsys, nrows, sys, plane, x, ws, ws_stride, kx);
    ++nl;
    for (int k = depth - 1; k >= 0; --k) {
        const dim3 g((unsigned)((sizes[k + 1] + 1 + kThreads - 1) / kThreads), (unsigned)nsys);
        k_psolve_back<<<g, kThreads, 0, st>>>(k, nrows, sys, plane, x, ws, ws_stride, kx);
        ++nl;
    }
    if (launches) *launches = nl;
    return cudaGetLastError();
}

namespace {

constexpr int kSolvePass = kSolveChunks * kChunk;                 // level-2 rows per pass
constexpr int kSolveSlots = kSolvePass + (kSolvePass >> 4) + 1;  // padded
constexpr int kTabTiles = 256;  // rows of up to this many tiles keep their tables in shared memory

// Level-2 rows staged in shared memory.
struct RedStage {
    SepRow row[kSolveSlots];
    double x[kSolveSlots + 1];  // reciprocal pivots, then the solution
};
static_assert(2 * kSolveChunks == kSolveThreads && kSolveChunks % 32 == 0,
              "a thread per chunk and direction");
static_assert(sizeof(RedStage) == kSolveStage, "the host sizes the workspace after it");

// Rows of a spline's transposed system from its knot positions and right-hand side in padded
// shared memory (KnotSysRows' values).
struct StagedKnotRows {
    const int* x;
    const double* r;
    int K, first;
    __device__ __forceinline__ Row operator()(int k) const {
        const int i = first + k;
        if (i == 0 || i == K - 1) return identity_row();
        const int x0 = x[kq(i)], dl = x0 - x[kq(i - 1)], du = x[kq(i + 1)] - x0;
        Row w;
        w.l = (double)dl;
        w.m = (double)(2 * (dl + du));
        w.u = (double)du;
        w.r = r[kq(i)];
        return w;
    }
};
struct PadSlots17 {
    double* p;  // padded array
    int first;
    __device__ __forceinline__ double& operator()(int k) const { return p[kq(first + k)]; }
};

// Asynchronous copies of the rows p0 .. p0 + kSolvePass - 1 of a spline's separator system from
// their tiles' slots (separator p is separator p - soff[t] of tile t) into the stage: eight
// threads per tile.  kInner: without the tiles' first and last rows.
template <bool kInner>
__device__ __forceinline__ void stage_rows(RedStage& st, const double* rows, const int* soff,
                                           int ntiles, int p0) {
    int t = 0;
    if (p0 > 0) {  // the tile of row p0: the last one with soff[t] <= p0
        int hi = ntiles - 1;
        while (t < hi) {
            const int mid = (t + hi + 1) >> 1;
            if (soff[mid] <= p0) t = mid;
            else hi = mid - 1;
        }
    }
    const int end = p0 + kSolvePass;
    for (t += threadIdx.x >> 3; t < ntiles && soff[t] < end; t += kSolveThreads >> 3) {
        const int s0 = soff[t];
        const int a = max(s0 + (kInner ? 1 : 0), p0), b = min(soff[t + 1] - (kInner ? 1 : 0), end);
        const double* src = rows + ((size_t)t * kRowSlots - s0) * 4;
        for (int p = a + (threadIdx.x & 7); p < b; p += 8) {
            SepRow* dst = st.row + kq(p - p0);
            cp_async16(dst, src + (size_t)p * 4);
            cp_async16(&dst->u, src + (size_t)p * 4 + 2);
        }
    }
}

// The separator system of one spline (P rows), solution to X.  One pass (P <= kSolvePass): the
// rows are staged already.  wg: global workspace, used when the level-3 system does not fit the
// wcap doubles of shared memory after the stage.  Every thread of the CTA calls it, after a
// barrier.
__device__ __forceinline__ void solve_separators(RedStage& st, int wcap, const double* rows,
                                                 const int* soff, int ntiles, int P, double* X,
                                                 double* wg) {
    const bool one = P <= kSolvePass;
    if (P <= kChunk) {
        if (threadIdx.x == 0) thomas_rows(st.row, P, st.x);
        __syncthreads();
        if (threadIdx.x < P) X[threadIdx.x] = st.x[threadIdx.x];
        return;
    }
    const int Q = (P - 1) / kChunk;  // level-3 size
    // One pass: the level-3 workspace follows the stage.  More: the stage is filled again for the
    // second sweep, so its x plane (the reciprocals would not last) and what follows the stage
    // hold the end relations and separator rows, and the level-3 system takes the staged rows'
    // place in between.
    const int deep = 5 * padded(Q) + Q + 64;  // level-3 rows, solution and below
    const bool fits = one ? 6 * (Q + 1) + deep <= wcap
                          : 10 * (Q + 1) <= wcap + kSolveSlots && deep <= 4 * kSolveSlots;
    double* ends = !fits ? wg : (one ? reinterpret_cast<double*>(&st + 1) : st.x);
    SepRow* sep = reinterpret_cast<SepRow*>(ends + 6 * (size_t)(Q + 1));  // (several passes)
    SepRow* r3 = one ? sep : (fits ? st.row : sep + (Q + 1));
    double* x3 = reinterpret_cast<double*>(r3 + padded(Q));
    double* ws3 = x3 + ((padded(Q) + 1) & ~1);  // deeper levels
    for (int p0 = 0; p0 < P; p0 += kSolvePass) {
        if (!one) {
            __syncthreads();
            stage_rows<false>(st, rows, soff, ntiles, p0);
            cp_async_wait_all();
            __syncthreads();
        }
        int lane_q;
        const bool top = ends_item(threadIdx.x, kSolveChunks, lane_q);
        const int q = p0 / kChunk + lane_q;
        if (q <= Q) {
            const int first = q * kChunk;
            const int len = (q < Q) ? kChunk - 1 : P - first;
            const int i = kq(first - p0);
            if (!top) {
                ends_rows<false>(st.row + i, len, nullptr, ends + 6 * q);
                if (!one && q < Q) sep[q] = load_row(st.row + i + kChunk - 1);
            } else {
                ends_rows<true>(st.row + i, len, one ? st.x + i : nullptr, ends + 6 * q);
            }
        }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < Q; p += kSolveThreads)
        r3[kq(p)] = next_row(load_row(one ? st.row + kq(p * kChunk + kChunk - 1) : sep + p),
                             ends + 6 * p);
    __syncthreads();
    partition_rows(CtaGroup(), Q, r3, x3, ws3);
    if (fits && !one) {  // the stage is filled again: the level-3 solution moves out of it
        for (int p = threadIdx.x; p < Q; p += kSolveThreads) ends[kq(p)] = x3[kq(p)];
        x3 = ends;
    }
    for (int p0 = 0; p0 < P; p0 += kSolvePass) {
        if (!one) {
            __syncthreads();
            stage_rows<false>(st, rows, soff, ntiles, p0);
            cp_async_wait_all();
            __syncthreads();
        }
        const int q = p0 / kChunk + threadIdx.x;
        if (threadIdx.x < kSolveChunks && q <= Q) {
            const int first = q * kChunk;
            const int len = (q < Q) ? kChunk - 1 : P - first;
            const double xl = (q > 0) ? x3[kq(q - 1)] : 0.0;
            const double xr = (q < Q) ? x3[kq(q)] : 0.0;
            SepRow* r = st.row + kq(first - p0);
            if (one) {
                double* x = st.x + kq(first);
                interior_rows(r, len, xl, xr, x);
                if (q < Q) x[kChunk - 1] = xr;
            } else {  // the x plane is taken: the solution goes straight to X, row by row
                double cp = 0.0, gp = 0.0;
#pragma unroll 1
                for (int k = 0; k < len; ++k) {
                    const SepRow a = load_row(r + k);
                    double ri = a.r;
                    if (k == 0) ri = fma(-a.l, xl, ri);
                    if (k == len - 1) ri = fma(-a.u, xr, ri);
                    const double iw = pivot_inv(k == 0 ? a.m : fma(-a.l, cp, a.m));
                    gp = (k == 0 ? ri : fma(-a.l, gp, ri)) * iw;
                    cp = a.u * iw;
                    r[k].u = cp;
                    r[k].r = gp;
                }
                double xv = gp;
                X[first + len - 1] = xv;
#pragma unroll 1
                for (int k = len - 2; k >= 0; --k) {
                    xv = fma(-r[k].u, xv, r[k].r);
                    X[first + k] = xv;
                }
                if (q < Q) X[first + kChunk - 1] = xr;
            }
        }
    }
    if (one) {
        __syncthreads();
        for (int p = threadIdx.x; p < P; p += kSolveThreads) X[p] = st.x[kq(p)];
    }
}

}  // namespace

// Transposed spline solve of the reverse pass in shared memory, one CTA per spline of nrows[s]
// knots (0: none): positions kx, right-hand side rhs (rows s of `stride` doubles), solution to z;
// cta_partitioned_global's operations in the same order.  The global-memory form spends its time in
// round trips of its sweeps (N = 8192, NR = 50: 45 us a launch in the first stage and 23 in the
// eighth, 15 and 9 here).
size_t adj_solve_smem(int cap) {
    const int P = cap / kChunk + 1;
    return sizeof(double) * (2 * (size_t)padded(cap) + 5 * (size_t)padded(P) + 6 * (size_t)(P + 1) +
                             (size_t)P + 80) +
           sizeof(int) * ((size_t)padded(cap) + 4);
}

__global__ void __launch_bounds__(kThreads)
k_adj_solve_smem(const int* nrows, int cap, const int32_t* kx, const double* rhs, size_t stride,
                 double* z) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int sp = blockIdx.x;
    const int K = nrows[sp];
    if (K <= 0) return;
    const int P = (K - 1) / kChunk;
    SepRow* r2 = reinterpret_cast<SepRow*>(dyn_smem);
    const int cp2 = cap / kChunk + 1;
    double* x2 = reinterpret_cast<double*>(r2 + padded(cp2));
    double* ends = x2 + ((padded(cp2) + 1) & ~1);
    double* ws = ends + 6 * (cp2 + 1);
    double* R = ws + ((cp2 + 65) & ~1);
    double* Z = R + padded(cap);
    int* X = reinterpret_cast<int*>(Z + padded(cap));
    const int32_t* x = kx + (size_t)sp * cap;
    const double* r = rhs + (size_t)sp * stride;
    for (int i = threadIdx.x; i < K; i += kThreads) {
        X[kq(i)] = x[i];
        R[kq(i)] = r[i];
    }
    __syncthreads();
    if (K <= kChunk) {
        if (threadIdx.x == 0)
            thomas_rolled(K, StagedKnotRows{X, R, K, 0}, PadSlots17{Z, 0}, PadSlots17{R, 0});
    } else {
        for (int q = threadIdx.x; q <= P; q += kThreads) {
            const int first = q * kChunk, len = (q < P) ? kChunk - 1 : K - first;
            const ChunkEnds e =
                chunk_ends(len, StagedKnotRows{X, R, K, first}, PadSlots17{Z, first});
            double* o = ends + 6 * q;
            o[0] = e.ga;
            o[1] = e.aa;
            o[2] = e.ba;
            o[3] = e.gb;
            o[4] = e.ab;
            o[5] = e.bb;
        }
        __syncthreads();
        for (int p = threadIdx.x; p < P; p += kThreads)
            r2[kq(p)] = next_row(
                sep_row(StagedKnotRows{X, R, K, 0}(p * kChunk + kChunk - 1)), ends + 6 * p);
        __syncthreads();
        partition_rows(CtaGroup(), P, r2, x2, ws);
        for (int q = threadIdx.x; q <= P; q += kThreads) {
            const int first = q * kChunk, len = (q < P) ? kChunk - 1 : K - first;
            const double xl = (q > 0) ? x2[kq(q - 1)] : 0.0, xr = (q < P) ? x2[kq(q)] : 0.0;
            chunk_interior_iw(len, StagedKnotRows{X, R, K, first}, xl, xr, PadSlots17{Z, first},
                              PadSlots17{R, first});
            if (q < P) Z[kq(first + kChunk - 1)] = xr;
        }
    }
    __syncthreads();
    double* out = z + (size_t)sp * cap;
    for (int i = threadIdx.x; i < K; i += kThreads) out[i] = Z[kq(i)];
}

namespace {

// The end rule of a spline whose first (side 0) or last (side 1) tile holds fewer than six
// knots: the three end knots come from the tiles' headers, the tile's chunk is eliminated again
// with the new end value.  ne: the tiles with knots, in order (NE of them); hd: the spline's
// headers; cnt: the tiles' knot counts.  kExtrema: the end value alone.
template <bool kExtrema>
__device__ __noinline__ void end_rule_sparse(const SiftArgs& a, int e, int sp, int side,
                                             const int* ne, int NE, const int* cnt, TileHdr* hd) {
    const int te = ne[side == 0 ? 0 : NE - 1];
    TileHdr& h0 = hd[te];
    const int c = cnt[te];
    int x[5];
    double y[5];
    for (int i = 0; i < c && i < 5; ++i) {
        x[i] = a.end_x[(size_t)(2 * sp + side) * kEndKnots + i];
        y[i] = a.end_y[(size_t)(2 * sp + side) * kEndKnots + i];
    }
    int ex[3];
    double ey[3];  // the three knots from the end inwards
    int got = 0;
    for (; got < 3 && got < c; ++got) {
        const int i = side == 0 ? got : c - 1 - got;
        ex[got] = x[i];
        ey[got] = y[i];
    }
    for (int r = 1; got < 3 && r < NE; ++r) {
        const int t = ne[side == 0 ? r : NE - 1 - r];
        const TileHdr& h = hd[t];
        ex[got] = side == 0 ? h.x0 : h.xb;
        ey[got] = side == 0 ? h.y0 : h.yb;
        ++got;
        if (got < 3 && cnt[t] > 1) {
            ex[got] = side == 0 ? h.x1 : h.xa;
            ey[got] = side == 0 ? h.y1 : h.ya;
            ++got;
        }
    }
    const double v = side == 0 ? boundary_left(e, ex[0], ex[1], ex[2], ey[0], ey[1], ey[2])
                               : boundary_right(e, ex[2], ex[1], ex[0], ey[2], ey[1], ey[0]);
    a.yend[2 * sp + side] = v;
    if (kExtrema) return;
    if (side == 0) {
        h0.y0 = v;
        if (c == 1) h0.yb = v;
        if (c == 2) h0.ya = v;
    } else {
        h0.yb = v;
        if (c == 1) h0.y0 = v;
        if (c == 2) h0.y1 = v;
    }
    y[side == 0 ? 0 : c - 1] = v;
    double s[4];
    for (int i = 0; i + 1 < c; ++i) s[i] = seg_slope(x[i], x[i + 1], y[i], y[i + 1]);
    if (c > 1) {  // k_tile_sift's slope of the end segment
        const int i = side == 0 ? 0 : c - 2;
        a.list_s[(size_t)(&h0 - a.hdr) * kListSlots + i] = s[i];
    }
    if (c < 3) return;  // no rows between the tile's separators
    const ChunkEnds ce = chunk_ends_knots(x, s, c - 2);
    h0.ga = ce.ga;
    h0.aa = ce.aa;
    h0.ba = ce.ba;
    h0.gb = ce.gb;
    h0.ab = ce.ab;
    h0.bb = ce.bb;
}

}  // namespace

// =======================================================================================
// k_spline_solve: one CTA per spline (envelope, realization): prefix sums over its tiles (knots,
// separators, tiles with knots), the end rule where one tile could not decide it, the rows of the
// separators at the tiles' edges, the separator system (levels >= 2 of the canonical partitioned
// solve), and for every tile the knots just outside it with their spline values.  The system's
// rows are staged once when they fit a pass (2048 rows).  Latency bound (a chain of short sweeps
// per CTA): two CTAs per SM with the level-3 system in shared memory.  B200, N=244032 NR=100: 24
// us at K/N = 0.18, 55 us for white noise; the two kernels before it took 42 us on average.
//
// kExtrema: the counts and the end rule alone, for the extrema entry (no shared memory but the
// tables).
// =======================================================================================
template <bool kExtrema>
__global__ void __launch_bounds__(kSolveThreads, 2)
k_spline_solve(const __grid_constant__ SiftArgs a) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int s_tab[3][kTabTiles + 1];
    __shared__ int s_scan[kSolveThreads / 32], s_k[kSolveThreads / 32], s_m[kSolveThreads / 32];
    RedStage& st = *reinterpret_cast<RedStage*>(dyn_smem);
    const int vs = blockIdx.x;
    // one channel: the grid is its splines, and every load below is under way before the
    // channel's done word is looked at
    const int ra = a.nchan == 1 ? a.nr1 : active_rows(a);
    if (vs >= 2 * ra) return;
    int e;
    const Geo q = spline_geo(a, vs, ra, e);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int done = a.nchan == 1 ? a.cs[0].done : 0, mark = a.mark[q.g];
    const int c_first = tid < q.ntiles ? a.tile_cnt[tix(a, e, q, 0) + tid] : 0;
    if (done) return;
    // the row to the list of its class of k_tile_sift
    auto list_row = [&](int cls) {
        const unsigned long long w =
            atomicAdd(&a.cls_count[cls], 1ull << 32 | (unsigned long long)q.ntiles);
        a.cls_row[(size_t)cls * a.nrows + (size_t)(w >> 32)] =
            make_int4(q.c, q.r, (int)(w & 0xffffffffull), 0);
    };
    if (mark == 0) {  // the row repeats its last iteration (k_tile_sift)
        if (e == 0 && tid == 0 && a.sift_split) list_row(0);
        return;
    }
    const int sp = spline_id(a, e, q);
    const int ntiles = q.ntiles;
    const size_t te0 = tix(a, e, q, 0);
    const int* cnt = a.tile_cnt + te0;
    TileHdr* hd = a.hdr + te0;
    double* rows = a.rows + te0 * (size_t)(kRowSlots * 4);
    const bool small = ntiles <= kTabTiles;
    const size_t o1 = oix(a, e, q);
    int* soff = small ? s_tab[0] : a.sep_off + o1;    // separators before each tile
    int* rank = small ? s_tab[1] : a.tile_rank + o1;  // tiles with knots before each tile
    int* ne = small ? s_tab[2] : a.tile_list + o1;    // the tiles with knots
    int P = 0, NE = 0, K = 0, cm = 0;
    for (int t0 = 0; t0 < ntiles; t0 += kSolveThreads) {
        const int t = t0 + tid;
        const int c = t0 == 0 ? c_first : (t < ntiles ? cnt[t] : 0);
        const int own = tile_seps(c) | (c > 0 ? 0x10000 : 0);  // both sums stay below 2^16
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        const int kw = __reduce_add_sync(0xffffffffu, c);
        const int mw = __reduce_max_sync(0xffffffffu, c);
        if (lane == 31) {
            s_scan[warp] = incl;
            s_k[warp] = kw;
            s_m[warp] = mw;
        }
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kSolveThreads / 32; ++w) {
            if (w < warp) before += s_scan[w];
            all += s_scan[w];
            K += s_k[w];
            cm = max(cm, s_m[w]);
        }
        const int ex = before + incl - own;
        if (t < ntiles) {
            soff[t] = P + (ex & 0xffff);
            rank[t] = NE + (ex >> 16);
            if (c > 0) ne[NE + (ex >> 16)] = t;
        }
        P += all & 0xffff;
        NE += all >> 16;
        __syncthreads();  // s_scan and s_k are reused
    }
    if (tid == 0) {
        soff[ntiles] = P;
        a.kcount[sp] = K;
        a.cmax[sp] = cm;
        if (a.sift_split && !kExtrema) {  // the spline that comes second knows both counts
            const unsigned other = atomicExch(&a.cls_wait[q.g], (unsigned)cm + 1u);
            if (other != 0u) {
                a.cls_wait[q.g] = 0u;
                const int co = (int)other - 1;
                list_row(sift_need(e ? co : cm, e ? cm : co) > kSiftSparse ? 1 : 0);
            }
        }
    }
    __syncthreads();
    const bool one = P <= kSolvePass;
    if (one && !kExtrema) stage_rows<true>(st, rows, soff, ntiles, 0);
    // the first tile holds sample 0 and the last one sample n-1, so both have knots
    if (K > 5) {
        const bool l = cnt[0] < 6, r = cnt[ntiles - 1] < 6;
        if (l || r) {
            if (tid == 0 && l) end_rule_sparse<kExtrema>(a, e, sp, 0, ne, NE, cnt, hd);
            if (tid == 32 && r) end_rule_sparse<kExtrema>(a, e, sp, 1, ne, NE, cnt, hd);
            __syncthreads();
        }
    }
    if (kExtrema) return;
    if (a.bflags && tid == 0) {
        // a replaced end value differs from the sample in its bits (t > y or t < y)
        const double* h = a.h[a.par[q.g]] + q.base;
        a.bflags[sp] = (unsigned char)(
            (__double_as_longlong(a.yend[2 * sp]) != __double_as_longlong(h[0]) ? 1 : 0) |
            (__double_as_longlong(a.yend[2 * sp + 1]) != __double_as_longlong(h[q.n - 1]) ? 2
                                                                                          : 0));
    }
    // rows of the first and last separator of every tile with knots
    for (int i = tid; i < NE; i += kSolveThreads) {
        const int t = ne[i], c = cnt[t];
        const TileHdr h = hd[t];
        TileHdr hp, hn;
        if (i > 0) hp = hd[ne[i - 1]];
        if (i + 1 < NE) hn = hd[ne[i + 1]];
        const int k = tile_seps(c) - 1;
        // (one pass: straight into the stage)
        SepRow* row0 = one ? st.row + kq(soff[t])
                           : reinterpret_cast<SepRow*>(rows) + (size_t)t * kRowSlots;
        SepRow* row1 = one ? st.row + kq(soff[t] + k) : row0 + k;
        Row sr = identity_row();
        if (i > 0 && (c > 1 || i + 1 < NE)) {
            const int xp = c > 1 ? h.x1 : hn.x0;
            const double yp = c > 1 ? h.y1 : hn.y0;
            sr = spline_row(hp.xb, h.x0, xp, div_int(h.y0 - hp.yb, (double)(h.x0 - hp.xb)),
                            div_int(yp - h.y0, (double)(xp - h.x0)));
        }
        Row o = c > 1 ? reduced_row(sr, 0.0, 1.0, 0.0, h.ga, h.aa, h.ba)
                      : reduced_row(sr, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0);
        *row0 = sep_row(o);
        if (c > 1) {
            sr = identity_row();
            if (i + 1 < NE)
                sr = spline_row(h.xa, h.xb, hn.x0, div_int(h.yb - h.ya, (double)(h.xb - h.xa)),
                                div_int(hn.y0 - h.yb, (double)(hn.x0 - h.xb)));
            o = reduced_row(sr, h.gb, h.ab, h.bb, 0.0, 0.0, 1.0);
            *row1 = sep_row(o);
        }
    }
    if (one) cp_async_wait_all();
    __syncthreads();
    double* X = a.xsep + rec_base(a, e, q);
    solve_separators(st, a.solve_wcap, rows, soff, ntiles, P, X, a.red + red_base(a, e, q));
    __syncthreads();
    // the knots just before and after every tile
    TileEdge* ed = a.edge + te0;
    for (int t = tid; t < ntiles; t += kSolveThreads) {
        const int s0 = soff[t], s1 = soff[t + 1], r = rank[t];
        TileEdge w;
        w.sep0 = s0;
        w.pad = 0;
        w.px = w.nx = 0;
        w.py = w.pc = w.ny = w.nc = 0.0;
        if (r > 0) {
            const TileHdr& h = hd[ne[r - 1]];
            w.px = h.xb;
            w.py = h.yb;
            w.pc = X[s0 - 1];
        }
        const int rn = r + (s1 > s0 ? 1 : 0);
        if (rn < NE) {
            const TileHdr& h = hd[ne[rn]];
            w.nx = h.x0;
            w.ny = h.y0;
            w.nc = X[s1];
        }
        ed[t] = w;
    }
}
template __global__ void k_spline_solve<false>(const __grid_constant__ SiftArgs a);
template __global__ void k_spline_solve<true>(const __grid_constant__ SiftArgs a);

// =======================================================================================
// k_tile_sift: persistent CTAs over the tiles: the spline values of the tile's knots (chunk
// interiors, one thread per chunk), the segment coefficients in shared memory, both envelopes at
// every sample, the mean envelope, the sx statistics, and the sample's next value h - m written to
// the other h plane.  The stop decision comes after a row's last tile (criterion below); it either takes the
// new plane as the row's h (mark 1) or keeps the old one (mark 0, the realization has finished:
// its mode is h).  A row marked 0 repeats its iteration: h, knots and envelopes are the same, so
// the next launch only exports the mode and counts the iteration; the new plane is already what
// that iteration's update gives.  The knots of both envelopes fit the shared-memory arrays at
// white-noise density (about 1440 a tile); denser rows take one envelope after the other.
//
// Bound by latency: a tile is a chain of short phases between barriers, so what counts is how many
// CTAs an SM holds.  Registers are kept under 96 (flags and counts read anew in the rare paths,
// two samples at a time, row words packed): five CTAs per SM with room for 736 knots, three with
// room for 1928; a row goes by its densest tile.  Knots and slopes come from k_tile_knots' lists
// instead of being found again, a row's counts are added once per CTA, not per tile, and both
// planes are stored coalesced out of shared memory (a thread's 32 bytes in a line each took 32
// cycles of the load/store unit, half of all it did).  B200, N=244032 NR=100, K/N = 0.18: 262 ->
// 205 us (2.9 TB/s of its 24 N bytes); K/N = 0.001: 167 -> 138 us; white noise: 381 -> 312 us.
// Four CTAs with room for 1184 were 225, 153 and 321 us where five were 206, 142 and 314.  Each class's launch takes the tiles of its
// own rows in even shares: with rows of both classes (K/N = 0.23) 398 -> 234 us.
// =======================================================================================
namespace {

// The row's stop decision after an iteration (sifting fraction carry, siftingCriterion,
// checkBreak), by one thread once all its tiles are counted (cn samples with sx > sd, any: some
// sx > sd2); the channel's last row closes the channel's iteration.
__device__ __noinline__ void row_criterion(const SiftArgs& a, int c, int g, int r, int n,
                                           unsigned cn, int any) {
    ChanState& cst = a.cs[c];
    const int nr = a.nchan == 1 ? a.nr1 : __ldg(&a.chan[c].nr);
    const double inv_n = 1.0 / (double)n;
    const int j = cst.iter, cap = cst.cap;
    const int kk = a.kcount[g] + a.kcount[a.nrows + g];
    const double fr = (a.frac[g] + (double)cn) * inv_n;
    a.frac[g] = fr;
    const bool crit = fr > a.tol || (any != 0 && kk > 6);
    int fin = a.finish[g];
    int mark = 1;
    if (fin == 0 && (!crit || j == cap - 1)) {
        mark = 0;
        fin = 1;
    }
    a.mark[g] = mark;
    a.finish[g] = fin;
    if (a.tape_mark) a.tape_mark[r] = (signed char)mark;
    if (mark == 1) {
        a.par[g] ^= 1;
    } else {  // the row's repeated iteration has the same counts
        a.cnt[g] = cn;
        a.any[g] = any;
    }
    atomicAdd(&cst.knots, (unsigned long long)kk);
    // rows counted (low word) and finished (high word); the thread that completes the count
    // knows both from the one sum
    const unsigned long long add = 1ull | (unsigned long long)fin << 32;
    const unsigned long long sum = atomicAdd(&cst.rows, add) + add;
    if ((unsigned)sum == (unsigned)nr) {
        cst.rows = 0ull;
        cst.iter = j + 1;
        cst.iters += 1ull;
        if (a.forced > 0 ? j + 1 >= a.forced : (int)(sum >> 32) == nr) cst.done = 1;
    }
}

// Adds the counts of some tiles (of one CTA's range) to their row's: one 64-bit sum of tiles,
// additions with some sx > sd2, and samples with sx > sd, so that the thread that completes the row
// has them all from its own addition, without a fence between counts and ticket (a fence here waits for the tile's stores:
// about a microsecond of every CTA).  Rows of 2^17 tiles and more (2^28 samples) do not fit one
// word: they are counted in separate words, ordered by fences.  Returns true to the thread that
// completes the row.
__device__ __forceinline__ bool count_tiles(const SiftArgs& a, const Geo& q, unsigned tiles,
                                            unsigned& cn, int& any) {
    const int bits = 32 - __clz(q.ntiles);
    if (bits <= a.count_bits) {
        const int s1 = bits + 12, s2 = s1 + bits;
        const unsigned long long add = (unsigned long long)cn | (unsigned long long)any << s1 |
                                       (unsigned long long)tiles << s2;
        const unsigned long long sum = atomicAdd(&a.acc[q.g], add) + add;
        if ((int)(sum >> s2) != q.ntiles) return false;
        a.acc[q.g] = 0ull;
        cn = (unsigned)(sum & ((1ull << s1) - 1ull));
        any = (sum >> s1 & ((1ull << bits) - 1ull)) != 0ull ? 1 : 0;
        return true;
    }
    unsigned* w = reinterpret_cast<unsigned*>(a.acc_wide + 2 * (size_t)q.g);
    if (cn) atomicAdd(w, cn);
    if (any) atomicOr(w + 1, 1u);
    __threadfence();
    if (atomicAdd(w + 2, tiles) + tiles != (unsigned)q.ntiles) return false;
    __threadfence();
    cn = atomicExch(w, 0u);
    any = (int)atomicExch(w + 1, 0u);
    w[2] = 0u;
    return true;
}

// chunk_interior (same operations, same order) of the chunk whose knots 0..len+1 sit in the
// padded arrays from the chunk's base on: x positions, s slopes; c receives the spline values of
// knots 1..len, d[k] the factor of row k meanwhile.  One new knot and slope a row, read ahead.
template <class Pivot>
__device__ __forceinline__ void chunk_interior_sweep(Pivot& pv, const short* x, const double* s,
                                                     double* c, double* d, int len, double xl,
                                                     double xr) {
    // row k: lengths x[k+1] - x[k], x[k+2] - x[k+1], slopes s[k], s[k+1]; row 0 takes xl, row
    // len-1 takes xr
    int xt = x[2];
    double l = (double)(x[1] - x[0]), u = (double)(xt - x[1]), un = 0.0, st = s[1], sn = 0.0;
    double ri = fma(-l, xl, 3.0 * (st - s[0]));
    if (len == 1) ri = fma(-u, xr, ri);
    if (len > 1) {
        const int xn = x[kq(3)];
        un = (double)(xn - xt);
        xt = xn;
        sn = s[2];
    }
    double iw = pv.inv(2.0 * (l + u));
    double cp = u * iw, gp = ri * iw;
    d[0] = cp;
#pragma unroll 2
    for (int k = 1; k < len; ++k) {
        c[k] = gp;
        l = u;
        u = un;
        ri = 3.0 * (sn - st);
        st = sn;
        if (k + 1 < len) {
            const int xn = x[kq(k + 3)];
            un = (double)(xn - xt);
            xt = xn;
            sn = s[k + 2];
        }
        if (k == len - 1) ri = fma(-u, xr, ri);
        iw = pv.inv(fma(-l, cp, 2.0 * (l + u)));
        gp = fma(-l, gp, ri) * iw;
        cp = u * iw;
        d[k] = cp;
    }
    c[len] = gp;
    double xv = gp;
#pragma unroll 4
    for (int k = len - 2; k >= 0; --k) {
        xv = fma(-d[k], xv, c[k + 1]);
        c[k + 1] = xv;
    }
}
__device__ __noinline__ void chunk_interior_checked(const short* x, const double* s, double* c,
                                                    double* d, int len, double xl, double xr) {
    CheckedPivot pv;
    chunk_interior_sweep(pv, x, s, c, d, len, xl, xr);
}
__device__ __forceinline__ void chunk_interior_knots(const short* x, const double* s, double* c,
                                                     double* d, int len, double xl, double xr) {
    RawPivot pv;
    chunk_interior_sweep(pv, x, s, c, d, len, xl, xr);
    if (pv.ones) chunk_interior_checked(x, s, c, d, len, xl, xr);
}

// Shared memory of k_tile_sift: kCap entries each for the knots' positions and segments (seg_at;
// envelope 1 after envelope 0; the knot after the tile where in-tile knot `count` would be), the
// tile's samples, and small pieces.  b holds the slopes at first.
template <int kCap>
struct SiftSmem {
    double b[kCap], c[kCap], d[kCap];
    double2 stage[kTileSamples / 2];  // the samples, in the end their next values
    double2 mean[kTileSamples / 4];   // half of every thread's mean envelope
    TileEdge edge[2];                 // and edges (envelopes 0, 1)
    unsigned bits[2][kWords];         // and bitmaps
    TileScan scan;                    // and knot counts
    double xs[2][kRowSlots];          // the tile's separator values
    alignas(16) short x[kCap];
};

}  // namespace

size_t tile_sift_smem(bool dense) {
    return dense ? sizeof(SiftSmem<kSiftDense>) : sizeof(SiftSmem<kSiftSparse>);
}

template <bool kDense, bool kSplit, bool kEnv>
__global__ void __launch_bounds__(kTileThreads, kDense ? 3 : 5)
k_tile_sift(const __grid_constant__ SiftArgs a) {
    constexpr int kCap = kDense ? kSiftDense : kSiftSparse;
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    SiftSmem<kCap>& S = *reinterpret_cast<SiftSmem<kCap>*>(dyn_smem);
    __shared__ int s_w[kTileWarps], s_begin;  // (s_begin: thread 0's own)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    TileIter<kSplit, kDense ? 1 : 0> it(a);
    // the knots' positions and slopes of envelope e of the tile, to the entries from base on
    auto fetch_list = [&](int e, int cm, int base, int th, int wh) {
        if (cm == 0) return;
        const size_t sl = tix(a, e, it.q, it.tile) * kListSlots;
        const int n = kq(cm - 1) + 1;  // (of the row's densest tile)
        for (int i = th; i < (n + 7) >> 3; i += wh)
            cp_async16(&S.x[base + 2 + 8 * i], a.list_x + sl + 8 * i);
        for (int i = th; i < (n + 1) >> 1; i += wh)
            cp_async16(&S.b[base + 2 + 2 * i], a.list_s + sl + 2 * i);
    };
    constexpr int kHalf = kTileThreads / 2;  // threads per envelope
    int sep = 0;  // the tile's first separator (of the envelope the thread fetches)
    // the tile's pieces, in two groups: what the sweeps read, then the samples
    auto prefetch = [&]() {
        if (!it.more()) return;
        if (it.live()) {
            const int e = tid / kHalf, th = tid % kHalf;
            const size_t te = tix(a, e, it.q, it.tile);
            if (th < kWords / 4) cp_async16(&S.bits[e][4 * th], a.bitmap + te * kWords + 4 * th);
            if (th >= 16 && th < 16 + (int)sizeof(TileEdge) / 16)
                cp_async16(reinterpret_cast<char*>(&S.edge[e]) + 16 * (th - 16),
                           reinterpret_cast<const char*>(a.edge + te) + 16 * (th - 16));
            if (tid >= 24 && tid < 24 + (int)sizeof(TileScan) / 16)
                cp_async16(reinterpret_cast<char*>(&S.scan) + 16 * (tid - 24),
                           reinterpret_cast<const char*>(a.scan + it.q.tile0 + it.tile) +
                               16 * (tid - 24));
            if (e == 0 || !(kDense && it.two()))
                fetch_list(e, it.cm, e ? it.base1 : kLead, th, kHalf);
            const double* X = a.xsep + rec_base(a, e, it.q) + sep;
            for (int i = th; i < kRowSlots; i += kHalf) cp_async8(&S.xs[e][i], X + i);
        }
        cp_async_commit();
        const int n0 = it.tile * kTileSamples;
        stage_tile(S.stage, a.h[it.par()] + it.q.base + n0, min(kTileSamples, it.q.n - n0), tid);
        cp_async_commit();
    };
    if (tid == 0) s_begin = it.v;
    if (it.more() && it.tile > 0) sep = a.edge[tix(a, tid / kHalf, it.q, it.tile)].sep0;
    prefetch();
    // samples with sx > sd of the row's tiles so far, and in the sign bit whether some sx > sd2
    unsigned cnt_row = 0u;
    while (it.more()) {
    const Geo& q = it.q;
    const int tile = it.tile;
    const bool repeat = !it.live(), write_mean = it.mean();
    ChanState& cst = a.cs[q.c];
    const int n0 = tile * kTileSamples;
    const int m = min(kTileSamples, q.n - n0);  // samples of the tile
    // the tile in the current plane and in the next one (kEnv: in the upper envelope)
    auto hin = [&]() -> const double* { return a.h[it.par()] + q.base + n0; };
    auto hout = [&]() -> double* {
        return kEnv ? a.dbg_upper + (size_t)q.r * q.n + n0 : a.h[it.par() ^ 1] + q.base + n0;
    };
    const int j0 = kPerThread * tid;
    const int lim = m - j0;  // the thread's samples in the row
    if (repeat) cp_async_wait_all();
    else cp_async_wait_but_one();  // (the samples are waited for after the sweeps)
    __syncthreads();
    unsigned cnt = 0u;  // samples with sx > sd
    int any = 0;        // some sx > sd2
    if (repeat) {
        // repeated iteration of a finished row: its mode is h
        double* mo = cst.mode_out + (size_t)q.r * q.n + n0;
        const int w0 = warp * kWarpSamples;
        for (int j = w0 + lane; j < min(m, w0 + kWarpSamples); j += 32) mo[j] = staged(S.stage, j);
    } else {
    const TileEdge* ed0 = &S.edge[0];
    const TileEdge* ed1 = &S.edge[1];
    const unsigned b0 = reinterpret_cast<const TileBits*>(S.bits[0])[tid];
    const unsigned b1 = reinterpret_cast<const TileBits*>(S.bits[1])[tid];
    const int tot = S.scan.total;
    const int own = __popc(b0) | __popc(b1) << 16;
    const int ex = S.scan.before[warp] + warp_scan(own, lane) - own;
    const bool first = tile == 0, last = tile == q.ntiles - 1;
    const int c0 = tot & 0xffff, c1 = tot >> 16;
    // (only the densest rows of the dense launch)
    const bool two = kDense && it.two();
    const int base0 = kLead, base1 = two ? kLead : it.base1;
    sep += tile_seps(tid < kHalf ? c0 : c1);  // the next tile's, unless a row starts there
    // knots before the thread's first sample (sample 0 of the row lies in the first segment)
    const bool origin = first && tid == 0;
    const int rA0 = origin ? 1 : ex & 0xffff, rA1 = origin ? 1 : ex >> 16;
    // position and value of knot r of envelope e (r = 0 before the tile, 1 .. count in it,
    // count + 1 after it) at entry p
    auto knot_x = [&](int e, int r, int p) -> int {
        const TileEdge* ed = e ? ed1 : ed0;
        if (r == 0) return ed->px - n0;
        if (r > (e ? c1 : c0)) return ed->nx - n0;
        return S.x[p];
    };
    auto knot_y = [&](int e, int r, int x) -> double {
        const TileEdge* ed = e ? ed1 : ed0;
        const int c = e ? c1 : c0;
        if (r == 0) return ed->py;
        if (r > c) return ed->ny;
        if (first && r == 1) return a.yend[2 * (e * a.nrows + q.g)];
        if (last && r == c) return a.yend[2 * (e * a.nrows + q.g) + 1];
        return staged(S.stage, x);
    };
    // envelope e at the thread's sample i, one at a time (the paths that are not the common one);
    // values from h itself: other warps may have refilled the stage
    auto env_one = [&](int e, int i, unsigned flags, int before) -> double {
        int r = (e ? before >> 16 : before & 0xffff) + __popc(flags & ((1u << i) - 1u));
        if (first && j0 + i == 0) r = 1;
        const int p = (e ? base1 : base0) + seg_at(r);
        const int x = knot_x(e, r, p);
        double y;
        if (r == 0) y = (e ? ed1 : ed0)->py;
        else if (first && r == 1) y = a.yend[2 * (e * a.nrows + q.g)];
        else y = hin()[x];
        return seg_eval(y, S.b[p], S.c[p], S.d[p], (double)(j0 + i - x));
    };
    // the thread's first segments: their first knots' values (read before the first next samples
    // replace them), and the first sample's place in them
    double yu = 0.0, yv = 0.0, tu = 0.0, tv = 0.0;
    for (int pass = 0; pass < (two ? 2 : 1); ++pass) {
        if (pass) {  // the upper envelope waits in the tile's part of the output plane
            double* up = hout();
            for (int i = 0; i < kPerThread && i < lim; ++i) up[j0 + i] = env_one(0, i, b0, ex);
            __syncthreads();
            fetch_list(1, a.cmax[a.nrows + q.g], base1, tid, kTileThreads);
            cp_async_wait_all();
            __syncthreads();
        }
        const int eh = two ? pass : tid / kHalf, th = two ? tid : tid % kHalf;
        const int wh = two ? kTileThreads : kHalf;
        const int ch = eh ? c1 : c0, bh = eh ? base1 : base0;
        const int step = kq(wh);  // seg_at advances by 17 for 16 segments
        {
            const int ns0 = two && pass ? 0 : tile_seps(c0);
            const int ns1 = two && !pass ? 0 : tile_seps(c1);
            int e, k;
            if (sweep_lane(tid, ns0, ns1, e, k)) {
                const double xl = S.xs[e][k - 1], xr = S.xs[e][k];
                const int jb = (k - 1) * kChunk, js = min(k * kChunk, (e ? c1 : c0) - 1);
                const int base = (e ? base1 : base0) + 2, i = base + kq(jb);
                if (js - jb > 1)
                    chunk_interior_knots(S.x + i, S.b + i, S.c + i, S.d + i, js - jb - 1, xl,
                                         xr);
                S.c[base + kq(js)] = xr;
                if (k == 1) S.c[base] = xl;
            }
            const TileEdge* ed = eh ? ed1 : ed0;
            if (th == wh - 1) S.c[bh] = ed->pc;
            if (th == wh - 2) S.c[bh + 2 + kq(ch)] = ed->nc;
            if (th == wh - 3 && ch == 1) S.c[bh + 2] = S.xs[eh][0];
        }
        if (!pass) cp_async_wait_all();  // the samples
        __syncthreads();
        // segment r starts at seg_at(r)
        for (int r = 1 + th, i0 = bh + seg_at(r), i1 = bh + seg_at(r + 1); r < ch;
             r += wh, i0 += step, i1 += step) {
            double b, d;
            seg_coeffs_int((double)(S.x[i1] - S.x[i0]), S.b[i0], S.c[i0], S.c[i1], b, d);
            S.b[i0] = b;
            S.d[i0] = d;
        }
        // the segments that enter and leave the tile (one and the same without a knot in it)
        if (th == wh - 1 ? !first : th == wh - 2 && !last && ch > 0) {
            const int r = th == wh - 1 ? 0 : ch, i0 = bh + seg_at(r), i1 = bh + seg_at(r + 1);
            const int x0 = knot_x(eh, r, i0), x1 = knot_x(eh, r + 1, i1);
            const double len = (double)(x1 - x0);
            double b, d;
            seg_coeffs_int(len, div_int(knot_y(eh, r + 1, x1) - knot_y(eh, r, x0), len), S.c[i0],
                           S.c[i1], b, d);
            S.b[i0] = b;
            S.d[i0] = d;
        } else if (th == wh - 2 && last) {
            // The samples past the row, in the warp that holds its end: envelopes of opposite
            // sign so large that the end knot's value vanishes in them, so sx = 0, which counts
            // nowhere (where it would not vanish, NaN: its thread does its samples again).
            const int i0 = bh + seg_at(ch);
            const double big = fabs(staged(S.stage, m - 1)) < 0x1p+900 ? 0x1p+1000 : NAN;
            S.b[i0] = eh ? -big : big;
            S.d[i0] = 0.0;
        }
        if (!two) {
            const int xu = rA0 == 0 ? ed0->px - n0 : S.x[base0 + seg_at(rA0)];
            const int xv = rA1 == 0 ? ed1->px - n0 : S.x[base1 + seg_at(rA1)];
            yu = rA0 == 0 ? ed0->py : staged(S.stage, xu);
            yv = rA1 == 0 ? ed1->py : staged(S.stage, xv);
            if (first) {  // the end value (the last segment starts before the other one)
                if (rA0 == 1) yu = a.yend[2 * q.g];
                if (rA1 == 1) yv = a.yend[2 * (a.nrows + q.g)];
            }
            tu = (double)(j0 - xu);
            tv = (double)(j0 - xv);
        }
        __syncthreads();
    }
    // kEnv: the envelopes themselves go to the caller's arrays in place of the next h and the
    // mean envelope (contiguous rows, aligned to 32 bytes or not: then a sample to a
    // lane, and the padded copy of the rows in: 61441 x 50 281 us a call, 61440 x 50 260)
    auto mean = [&]() -> double* {
        return kEnv ? a.dbg_lower + (size_t)q.r * q.n + n0 : a.menv + q.base + n0;
    };
    const bool wide = !kEnv || (((size_t)a.dbg_upper | (size_t)a.dbg_lower) & 31) == 0 &&
                                   (q.n & 3) == 0;
    bool redo = false;
    // samples of the row in the warp's part of the tile (warp-uniform)
    const int in_row = m - warp * kWarpSamples;
    const bool full = in_row >= kWarpSamples;
    const bool common = !two && (kEnv || write_mean) && in_row > 0;
    if (common) {
        // Both envelopes along the thread's samples: a segment's coefficients are loaded when the
        // samples pass its first knot (whose value is that sample's).  sx > t is decided by the
        // signs of p - q t for bounds t around the threshold (sx_bounds; one fma rounds to zero or
        // to the exact sign, over- and underflow included); a thread with an undecided sample
        // or a NaN redoes its samples with the division.  Once the warp has seen some sx > sd2 in
        // the row it only counts.
        const bool known = __any_sync(0xffffffffu, cnt_row >> 31 != 0u);
        int ru = rA0, rv = rA1;
        double bu, cu, du, bv, cv, dv;
        auto load_u = [&]() {
            const int p = base0 + seg_at(ru);
            bu = S.b[p];
            cu = S.c[p];
            du = S.d[p];
        };
        auto load_v = [&]() {
            const int p = base1 + seg_at(rv);
            bv = S.b[p];
            cv = S.c[p];
            dv = S.d[p];
        };
        load_u();
        load_v();
        const unsigned f0 = origin ? b0 & ~1u : b0, f1 = origin ? b1 & ~1u : b1;
        const unsigned wf = __reduce_or_sync(0xffffffffu, f0 | f1);
        int und = 0, smax = 0, amax = -1, bmax = -1;
        double2* mean_w = S.mean + warp * (kTileSamples / 4 / kTileWarps);
        // two samples at a time: without a knot among them in the whole warp one set of
        // coefficients serves both, and nothing splits the instruction stream
#pragma unroll 1
        for (int i0 = 0; i0 < kPerThread; i0 += 4) {
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
            double2* const pa = own_piece(S.stage, tid, (i0 + k) / 2);
            double eu[2], ev[2];
            if (!(wf >> (i0 + k) & 3u)) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    eu[i] = seg_eval(yu, bu, cu, du, tu + (double)i);
                    ev[i] = seg_eval(yv, bv, cv, dv, tv + (double)i);
                }
                tu += 2.0;
                tv += 2.0;
            } else {
                const double2 hk = *pa;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    eu[i] = seg_eval(yu, bu, cu, du, tu);
                    ev[i] = seg_eval(yv, bv, cv, dv, tv);
                    tu += 1.0;
                    tv += 1.0;
                    if (f0 >> (i0 + k + i) & 1u) {
                        ++ru;
                        load_u();
                        yu = i ? hk.y : hk.x;
                        tu = 1.0;
                    }
                    if (f1 >> (i0 + k + i) & 1u) {
                        ++rv;
                        load_v();
                        yv = i ? hk.y : hk.x;
                        tv = 1.0;
                    }
                }
            }
            double2* const pm = mean_w + (stage_piece(4 * lane) ^ ((i0 + k) / 2 & 3));
            if (kEnv) {
                *pa = make_double2(eu[0], eu[1]);
                *pm = make_double2(ev[0], ev[1]);
                continue;
            }
            const double2 hk = *pa;
            double mv[2], hn[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double s = eu[i] + ev[i], p = fabs(s), w = fabs(eu[i] - ev[i]);
                mv[i] = s / 2.0;
                hn[i] = (i ? hk.y : hk.x) - mv[i];
                const int s1 = __double2hiint(fma(-a.sd_hi, w, p));
                const int s0 = __double2hiint(fma(-a.sd_lo, w, p));
                und |= (s1 - 1) & ~s0;  // sign bit: neither bound decides
                cnt += 1u - ((unsigned)s0 >> 31);  // (when decided, not below means above)
                smax = max(smax, s1);
                if (!known) {
                    amax = max(amax, __double2hiint(fma(-a.sd2_hi, w, p)));
                    bmax = max(bmax, __double2hiint(fma(-a.sd2_lo, w, p)));
                }
            }
            *pa = make_double2(hn[0], hn[1]);
            *pm = make_double2(mv[0], mv[1]);
            }
            if (i0 & 4) {  // 64 bytes of every lane's samples
                __syncwarp();
                if (!wide) {
                    double* const out = mean() + warp * kWarpSamples;
                    for (int g = 0; g < 8; ++g) {
                        const int i = lane + 32 * g, o = kPerThread * (i >> 3) + (i0 & 8) + (i & 7);
                        if (o < in_row) out[o] = staged(mean_w, i);
                    }
                } else
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int j = lane + 32 * g;
                    const int u = stage_piece(2 * j);
                    const double2 p0 = mean_w[u], p1 = mean_w[u ^ 1];
                    const double w[4] = {p0.x, p0.y, p1.x, p1.y};
                    const int o = kPerThread * (j >> 1) + (i0 & 8) + 4 * (j & 1);
                    if (full || o < in_row) store4(mean() + warp * kWarpSamples + o, w);
                }
                __syncwarp();
            }
        }
        if (!wide) {
            for (int i = lane; i < min(in_row, kWarpSamples); i += 32)
                hout()[warp * kWarpSamples + i] = staged(S.stage, warp * kWarpSamples + i);
        } else {
#pragma unroll
            for (int g = 0; g < kPerThread / 4; ++g) {
                const int u = (tid & ~31) * (kPerThread / 2) + 2 * (lane + 32 * g);
                const double2 p0 = S.stage[stage_piece(u)], p1 = S.stage[stage_piece(u) ^ 1];
                const double w[4] = {p0.x, p0.y, p1.x, p1.y};
                if (full || 2 * u < m) store4(hout() + 2 * u, w);  // (rows are padded to four)
            }
        }
        any = amax > 0 ? 1 : 0;
        // undecided, a NaN, or no sample surely above sd2 and not all surely below
        redo = und < 0 || smax > 0x7ff00000 || (amax <= 0 && bmax >= 0);
    }
    if (__any_sync(0xffffffffu, !common || (redo && !kEnv))) {
        // (the flags and counts anew: kept, they would cost the common path registers)
        const unsigned f0 = reinterpret_cast<const TileBits*>(S.bits[0])[tid];
        const unsigned f1 = reinterpret_cast<const TileBits*>(S.bits[1])[tid];
        const int mine = __popc(f0) | __popc(f1) << 16;
        const int before = S.scan.before[warp] + warp_scan(mine, lane) - mine;
        if (!common || redo) {
        cnt = 0u;
        any = 0;
        double* ho = hout() + j0;
        double* me = mean() + j0;
        const double* hi = hin() + j0;
#pragma unroll 1
        for (int i = 0; i < kPerThread && i < lim; ++i) {
            const double u = two ? ho[i] : env_one(0, i, f0, before);
            const double v = env_one(1, i, f1, before);
            if (kEnv) {
                ho[i] = u;
                me[i] = v;
                continue;
            }
            if (!common) {
                double mv = (u + v) / 2.0;
                if (write_mean) me[i] = mv;
                else mv = me[i];
                ho[i] = hi[i] - mv;
            }
            any |= sx_greater(u, v, a.sd2) ? 1 : 0;
            cnt += sx_greater(u, v, a.sd) ? 1 : 0;
        }
        }
    }
    }
    cnt_row = ((cnt_row & 0x7fffffffu) + cnt) | (cnt_row & 0x80000000u) |
              (any != 0 ? 0x80000000u : 0u);
    // the CTA's last tile of the row: the counts of the warps, then the row's
    const bool leave = !kEnv && (tile + 1 == q.ntiles || it.v + 1 == it.end);
    if (leave) {
        const bool y = __any_sync(0xffffffffu, cnt_row >> 31 != 0u);
        cnt_row = __reduce_add_sync(0xffffffffu, cnt_row & 0x7fffffffu);
        if (lane == 0) s_w[warp] = (int)(cnt_row | (y ? 1u << 30 : 0u));
    }
    __syncthreads();
    if (leave) {
        if (tid == 0) {
            unsigned t = 0u;
            int y = 0;
#pragma unroll
            for (int w = 0; w < kTileWarps; ++w) {
                t += (unsigned)s_w[w] & 0x3fffffffu;
                y |= s_w[w] >> 30;
            }
            // (since the start of the row or of the CTA's range)
            const int tiles = it.v + 1 - max(it.v - tile, s_begin);
            if (count_tiles(a, q, (unsigned)tiles, t, y)) {
                if (repeat) {
                    t = a.cnt[q.g];
                    y = a.any[q.g];
                }
                row_criterion(a, q.c, q.g, q.r, q.n, t, y);
            }
        }
        cnt_row = 0u;
    }
    // every warp is done with the tile: the next one's pieces take its place
    it.next(a);
    if (it.tile == 0) sep = 0;
    prefetch();
    }
}

template __global__ void k_tile_sift<true, false, false>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_sift<true, true, false>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_sift<false, true, false>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_sift<true, false, true>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_sift<true, true, true>(const __grid_constant__ SiftArgs a);
template __global__ void k_tile_sift<false, true, true>(const __grid_constant__ SiftArgs a);

// Mode export of channel c's realizations that finished in the last executed iteration
// (blockIdx.y = realization).
__global__ void k_export_final(SiftArgs a, int c) {
    const Geo q = geo(a, c, blockIdx.y);
    if (a.mark[q.g] != 0) return;
    const ChanState& cst = a.cs[c];
    const double* h = a.h[a.par[q.g]] + q.base;
    double* mo = cst.mode_out + (size_t)q.r * q.n;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < q.n; s += gridDim.x * blockDim.x)
        mo[s] = h[s];
}

// Start of a stage of channel c (one CTA): the stage's sift cap and mode buffer, iteration 0,
// no realization finished, no update pending.
__global__ void k_begin_stage(SiftArgs a, int c, int cap, double* mode_out) {
    const Chan* ch = a.chan + c;
    const int nr = __ldg(&ch->nr), row0 = __ldg(&ch->row0);
    for (int r = threadIdx.x; r < nr; r += blockDim.x) {
        a.mark[row0 + r] = -1;
        a.finish[row0 + r] = 0;
        a.par[row0 + r] = 0;
        a.cnt[row0 + r] = 0u;
        a.any[row0 + r] = 0;
    }
    if (threadIdx.x == 0) {
        ChanState& cst = a.cs[c];
        cst.done = 0;
        cst.iter = 0;
        cst.cap = cap;
        cst.mode_out = mode_out;
    }
}

// Active-channel plan of the iteration (several channels): one CTA.  plan[c] = rows and
// plan[nchan+1+c] = tiles of the channels before c whose stage is running (done == 0);
// plan[nchan] and plan[2*nchan+1] are the totals.
__device__ void plan_block(const SiftArgs& a) {
    __shared__ int s_rows[32], s_tiles[32];
    const int m = a.nchan;
    const int per = (m + 1023) / 1024;
    const int i0 = threadIdx.x * per;
    int rows = 0, tiles = 0;
    for (int i = i0; i < min(i0 + per, m); ++i) {
        if (a.cs[i].done) continue;
        const int nr = a.chan[i].nr;
        rows += nr;
        tiles += nr * a.chan[i].ntiles;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int ir = rows, itl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, ir, o);
        const int w = __shfl_up_sync(0xffffffffu, itl, o);
        if (lane >= o) {
            ir += u;
            itl += w;
        }
    }
    if (lane == 31) {
        s_rows[warp] = ir;
        s_tiles[warp] = itl;
    }
    __syncthreads();
    if (warp == 0) {
        int u = s_rows[lane], w = s_tiles[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int pu = __shfl_up_sync(0xffffffffu, u, o);
            const int pw = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) {
                u += pu;
                w += pw;
            }
        }
        s_rows[lane] = u;
        s_tiles[lane] = w;
    }
    __syncthreads();
    int pr = (warp > 0 ? s_rows[warp - 1] : 0) + ir - rows;
    int pt = (warp > 0 ? s_tiles[warp - 1] : 0) + itl - tiles;
    for (int i = i0; i < min(i0 + per, m); ++i) {
        a.plan[i] = pr;
        a.plan[m + 1 + i] = pt;
        if (a.cs[i].done) continue;
        const int nr = a.chan[i].nr;
        pr += nr;
        pt += nr * a.chan[i].ntiles;
    }
    if (threadIdx.x == 1023) {
        a.plan[m] = s_rows[31];
        a.plan[2 * m + 1] = s_tiles[31];
    }
}

__global__ void __launch_bounds__(1024)
k_plan(SiftArgs a) {
    plan_block(a);
}

// =======================================================================================
// generic batched tridiagonal solve (stage-level entry point): one CTA per system
// =======================================================================================
__global__ void __launch_bounds__(kTridiagThreads)
k_tridiag_batched(int n, const double* l, const double* m, const double* u, const double* r,
                  double* x, double* sys, double* ws, size_t ws_stride) {
    const size_t b = blockIdx.x;
    double* S = sys + b * 4 * (size_t)n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        S[i] = l[b * n + i];
        S[n + i] = m[b * n + i];
        S[2 * n + i] = u[b * n + i];
        S[3 * n + i] = r[b * n + i];
    }
    __syncthreads();
    cta_partitioned_global<AnyPivot>(n, S, n, x + b * n, ws + b * ws_stride);
}

}  // namespace ceemdan
