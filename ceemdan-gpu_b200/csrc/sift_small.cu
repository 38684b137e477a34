// k_sift_small: the whole lock-step sift of one stage for rows of at most kSmallMaxN samples, in
// one cooperative launch that keeps every realization's h in shared memory.  An iteration on chip:
// the deferred update, extrema and compaction, the end-knot rule, the canonical tile-aligned
// spline solve (chunk end relations, separator rows, the separator system by the index-based
// partition, chunk interiors), segment coefficients, both envelopes, the mean envelope, the sx
// statistics and the stop test.  Every operation is the one the three-kernel iteration of
// sift_kernels.cu performs, in the same order, so the results are bit-identical.  Channel 0 only;
// the reference loop it replaces is cudaICEEMDAN.cu:1752-1867 (per iteration ~25 kernel launches
// and library calls, and a host round trip).
//
// An iteration is a chain of short phases, so what counts is latency: a sweep over 15 rows is one
// lane's serial work, a phase ends at a barrier, and everything else is parallel over the samples
// or knots.  Three forms, by what the GPU holds (enable_small):
//   kPair    two CTAs (a cluster) per realization, one envelope each.  After the coefficients each
//            CTA evaluates its envelope for the other's half of the row into the other's shared
//            memory, then its own half; each combines one half, and the mean envelope's other half
//            comes back through L2.
//   kDual    one CTA, two groups of 256 threads with a barrier each, one envelope per group.
//   kSingle  one CTA, one envelope after the other; the upper one waits in global memory.
// All realizations meet once per iteration at the lock-step test, one 64-bit count per iteration
// (arrivals and, in the high word, finished realizations).  Nothing else passes between
// realizations, so the test of iteration j is awaited in the middle of iteration j + 1, whose
// work until then changes nothing that outlives the stage; the wait polls at most spin_limit
// times, then the CTA sets CEEMDAN_ERR_TIMEOUT in the channel's error word and the stage ends.
//
// B200, one iteration of the first stages, the previous form (one kernel, unrolled sweeps, the
// upper envelope handed over through L2, the stop test awaited at once) and this one: N=4096 NR=50
// 37.6 -> 14.2 us, N=8192 NR=50 49.1 -> 19.2 (kPair); N=2501 NR=100 54.5 -> 14.9, N=5000 NR=100
// 65.0 -> 20.8 (kDual); N=7680 NR=100 79.6 -> 33.7 (kSingle).  The code of an iteration has to stay
// in the instruction cache: with a copy of build_envelope for each group kDual took 18.2 and 26.5.
// At N=4096 NR=50 a quarter of the 28,000 cycles is the separator system (two sweeps of 15 rows at
// 80 cycles a reciprocal, and their barriers), a quarter the evaluation and the exchange.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "canon.cuh"
#include "kernels.h"
#include "spline_device.cuh"

namespace ceemdan {

namespace cg = cooperative_groups;

namespace {

constexpr int kMaxTiles = kSmallMaxN / kTileSamples;
constexpr int kSmallWords = kSmallMaxN / 32;
static_assert(kSmallMaxN % kTileSamples == 0 && kTileSamples == 64 * 32, "two warps of words a tile");

// What a CTA's wait at the lock-step test came to.
constexpr int kGoOn = 0, kStop = 1, kGaveUp = 2;

// The threads that build one envelope: the whole CTA, or half of it with its own barrier.
template <int kSize>
struct SmallGroup {
    int id, t;
    __device__ __forceinline__ int tid() const { return t; }
    __device__ __forceinline__ int size() const { return kSize; }
    __device__ __forceinline__ void sync() const {
        if (kSize == kSmallThreads) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + id), "r"(kSize) : "memory");
    }
};

// One envelope's arrays.  Knot m of tile t sits at base[t] + kq(m): a tile's knots start at a new
// slot, with one pad slot per 16, so that a chunk's knots are consecutive and the lanes that sweep
// neighbouring chunks read different banks.
struct EnvSmem {
    double *S, *C, *D;  // slopes -> b; reciprocal pivots -> spline values; lengths -> factors -> d
    short* X;           // knot positions
    SepRow* R2;         // separator system (padded rows), its solution, end relations, workspace
    double *X2, *ends, *ws;
    int2* W;            // words of the knot bitmap with the tile's knots before them
    struct Info {
        int cnt[kMaxTiles], base[kMaxTiles];   // knots, first slot
        int soff[kMaxTiles + 1];               // separators before the tile
        int prev[kMaxTiles], next[kMaxTiles];  // slots of the last knot before / first after it
        int K;
        double yend[2];
    }* I;
};

struct SmallLayout {
    size_t H, S, C, D, X, R2, X2, ends, ws, W, info, warp;  // offsets (env arrays: within a set)
    size_t set, total;  // bytes of one envelope's set, of everything
    size_t recv;        // kPair: doubles for the other CTA's envelope, over the solve's workspace
};

__host__ __device__ inline SmallLayout small_layout(int n, int mode) {
    const int ntiles = (n + kTileSamples - 1) / kTileSamples;
    const int kcap = n / 2 + 2;
    const int slots = kcap + kcap / 16 + 2 * ntiles;
    const int pcap = kcap / kChunk + 2 * ntiles + 8;
    SmallLayout L;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 15) & ~(size_t)15;
        return o;
    };
    L.S = take(sizeof(double) * slots);
    L.C = take(sizeof(double) * slots);
    L.D = take(sizeof(double) * slots);
    L.R2 = L.recv = off;
    take(sizeof(SepRow) * padded(pcap));
    L.X2 = take(sizeof(double) * padded(pcap));
    L.ends = take(sizeof(double) * 6 * (pcap + 1));
    L.ws = take(sizeof(double) * (pcap + 64));
    if (mode == kSmallPair) {  // at least half a row for the exchanged envelope
        const size_t need = L.recv + sizeof(double) * (size_t)small_half(n);
        if (off < need) off = (need + 15) & ~(size_t)15;
    }
    L.X = take(sizeof(short) * slots);
    L.W = take(sizeof(int2) * ((n + 31) / 32 + 1));
    L.info = take(sizeof(EnvSmem::Info));
    L.warp = take(sizeof(int) * (kSmallWords / 32));
    L.set = off;
    off = 0;
    L.H = take(sizeof(double) * n);
    L.total = L.H + off + L.set * (mode == kSmallDual ? 2 : 1);
    return L;
}

__device__ __forceinline__ EnvSmem env_smem(const SmallLayout& L, unsigned char* set) {
    EnvSmem E;
    E.S = reinterpret_cast<double*>(set + L.S);
    E.C = reinterpret_cast<double*>(set + L.C);
    E.D = reinterpret_cast<double*>(set + L.D);
    E.X = reinterpret_cast<short*>(set + L.X);
    E.R2 = reinterpret_cast<SepRow*>(set + L.R2);
    E.X2 = reinterpret_cast<double*>(set + L.X2);
    E.ends = reinterpret_cast<double*>(set + L.ends);
    E.ws = reinterpret_cast<double*>(set + L.ws);
    E.W = reinterpret_cast<int2*>(set + L.W);
    E.I = reinterpret_cast<EnvSmem::Info*>(set + L.info);
    return E;
}

// The interior of a chunk whose reciprocals the end relations left in c[1 .. len] (the chain is
// 17 cycles a row forward and 9 back; a row a turn with its loads and tests took 180, four rows a
// turn take 110), in chunk_interior_knots' arrays: c receives the spline values, d the factors meanwhile.
__device__ __forceinline__ void interior_known(const double* s, double* c, double* d, int len,
                                               double xl, double xr) {
    double l = d[0], u = d[1], s0 = s[1];
    double ri = fma(-l, xl, 3.0 * (s0 - s[0]));
    if (len == 1) ri = fma(-u, xr, ri);
    double iw = c[1];
    double gp = ri * iw;
    d[0] = u * iw;
    c[1] = gp;
    int k = 1;
    // four rows at a time, loaded before the first of them is needed
#pragma unroll 1
    for (; k + 4 < len; k += 4) {
        double du[4], ds[4], dw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            du[i] = d[k + 1 + i];
            ds[i] = s[k + 1 + i];
            dw[i] = c[k + 1 + i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            gp = fma(-u, gp, 3.0 * (ds[i] - s0)) * dw[i];
            s0 = ds[i];
            u = du[i];
            d[k + i] = u * dw[i];
            c[k + 1 + i] = gp;
        }
    }
#pragma unroll 1
    for (; k < len; ++k) {
        l = u;
        u = d[k + 1];
        ri = 3.0 * (s[k + 1] - s0);
        s0 = s[k + 1];
        if (k == len - 1) ri = fma(-u, xr, ri);
        iw = c[k + 1];
        gp = fma(-l, gp, ri) * iw;
        d[k] = u * iw;
        c[k + 1] = gp;
    }
    double xv = gp;
    k = len - 2;
#pragma unroll 1
    for (; k >= 3; k -= 4) {
        double f[4], g[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = d[k - i];
            g[i] = c[k + 1 - i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xv = fma(-f[i], xv, g[i]);
            c[k + 1 - i] = xv;
        }
    }
#pragma unroll 1
    for (; k >= 0; --k) {
        xv = fma(-d[k], xv, c[k + 1]);
        c[k + 1] = xv;
    }
}

// Separator p: its tile and index within the tile.
__device__ __forceinline__ void sep_tile(const EnvSmem::Info& I, int ntiles, int p, int& t,
                                         int& k) {
    t = 0;
    while (t + 1 < ntiles && I.soff[t + 1] <= p) ++t;
    k = p - I.soff[t];
}

// Builds envelope e of the row in H from the signs of its neighbour differences (sg: falls, sl:
// rises, word w at [w + 1], the word before the row 0): knots, end rule, spline, segment
// coefficients.  wait: called by the group's last thread while the others are in the first sweep.
template <class Group, class Wait>
__device__ void build_envelope(const Group& grp, const EnvSmem& E, int* warp_tot, const double* H,
                               const unsigned* sg, const unsigned* sl, int n, int e,
                               const SmallArgs& sa, int j, int r, const Wait& wait) {
    const int tid = grp.tid(), lane = tid & 31, warp = tid >> 5, G = grp.size();
    const int nw = (n + 31) >> 5;
    const int ntiles = (n + kTileSamples - 1) / kTileSamples;
    EnvSmem::Info& I = *E.I;
    // knot words, and the tile's knots before each (a tile's words are two warps')
    unsigned f = 0u;
    int own = 0, incl = 0;
    if (warp < kSmallWords / 32) {
        const int w = tid;
        if (w < nw) {
            const unsigned* fst = e == 0 ? sl : sg;
            const unsigned* snd = e == 0 ? sg : sl;
            f = __funnelshift_l(fst[w], fst[w + 1], 1) & snd[w + 1];
            const int last = n - 1 - 32 * w;  // bit of sample n-1, a knot as sample 0 is
            if (last < 32) f = (f & ((1u << last) - 1u)) | 1u << last;
            if (w == 0) f |= 1u;
        }
        own = __popc(f);
        incl = warp_scan(own, lane);
        if (lane == 31) warp_tot[warp] = incl;
    }
    grp.sync();
    if (warp < kSmallWords / 32 && tid < nw)
        E.W[tid] = make_int2((int)f, incl - own + ((warp & 1) ? warp_tot[warp - 1] : 0));
    if (tid < ntiles) {  // tile tables
        int base = 0, seps = 0, K = 0, prev = -1, c = 0;
        for (int t = 0; t <= tid; ++t) {
            c = warp_tot[2 * t] + warp_tot[2 * t + 1];
            K += c;
            if (t == tid) break;
            if (c > 0) prev = base + kq(c - 1);
            seps += tile_seps(c);
            base += padded(c);
        }
        I.cnt[tid] = c;
        I.base[tid] = base;
        I.soff[tid] = seps;
        I.prev[tid] = tid == 0 ? 0 : prev;  // (sample 0 lies in the first segment)
        int nb = base + padded(c), next = -1;
        for (int t = tid + 1; t < ntiles && next < 0; ++t) {
            const int ct = warp_tot[2 * t] + warp_tot[2 * t + 1];
            if (ct > 0) next = nb;
            nb += padded(ct);
        }
        I.next[tid] = next;
        if (tid == ntiles - 1) {
            I.soff[ntiles] = seps + tile_seps(c);
            I.K = K;
        }
    }
    grp.sync();
    for (int w = warp; w < nw; w += G / 32) {
        const int2 wo = E.W[w];
        if ((unsigned)wo.x >> lane & 1u)
            E.X[I.base[w >> 6] + kq(wo.y + __popc((unsigned)wo.x & ((1u << lane) - 1u)))] =
                (short)(32 * w + lane);
    }
    grp.sync();
    const int K = I.K, P = I.soff[ntiles];
    const int tl = ntiles - 1;
    // slope and length of the segment between slots p0 and p1
    auto segment = [&](int p0, int p1, double y0, double y1) {
        const double len = (double)(E.X[p1] - E.X[p0]);
        E.D[p0] = len;
        E.S[p0] = div_int(y1 - y0, len);
    };
    // slots of the last knot and the one before it
    const int pl = I.base[tl] + kq(I.cnt[tl] - 1);
    const int pl1 = I.cnt[tl] > 1 ? I.base[tl] + kq(I.cnt[tl] - 2) : I.prev[tl];
    if (tid == 0 || tid == 32) {
        // end rule (setBoundaryMax/Min) and the first / last segment, which take the end values
        auto tile_of = [&](int p) {
            int t = tl;
            while (I.cnt[t] == 0 || p < I.base[t]) --t;
            return t;
        };
        auto after = [&](int p) {  // the knot slot after p
            const int t = tile_of(p), d = p - I.base[t], m = d - d / 17;
            return m + 1 < I.cnt[t] ? I.base[t] + kq(m + 1) : I.next[t];
        };
        auto before = [&](int p) {
            const int t = tile_of(p), d = p - I.base[t], m = d - d / 17;
            return m > 0 ? I.base[t] + kq(m - 1) : I.prev[t];
        };
        if (tid == 0) {
            double y0 = H[0];
            const bool near = I.cnt[0] > 2;  // the three knots lie in the first tile
            const int p1 = near ? 1 : after(0);
            if (K - 1 > 4) {
                const int p2 = near ? 2 : after(p1);
                y0 = boundary_left(e, E.X[0], E.X[p1], E.X[p2], H[0], H[E.X[p1]], H[E.X[p2]]);
            }
            I.yend[0] = y0;
            if (K > 2) segment(0, p1, y0, H[E.X[p1]]);
            else segment(0, pl, y0, H[n - 1]);  // (two knots: no rule)
        } else {
            double yL = H[n - 1];
            if (K - 1 > 4) {
                const int c = I.cnt[tl], p2 = c > 2 ? I.base[tl] + kq(c - 3) : before(pl1);
                yL = boundary_right(e, E.X[p2], E.X[pl1], E.X[pl], H[E.X[p2]], H[E.X[pl1]],
                                    H[n - 1]);
            }
            I.yend[1] = yL;
            if (K > 2) segment(pl1, pl, H[E.X[pl1]], yL);
        }
    }
    for (int t = 0; t < ntiles; ++t) {
        const int c = I.cnt[t], b = I.base[t];
        for (int m = tid; m < c; m += G) {
            const int p0 = b + kq(m), p1 = m + 1 < c ? b + kq(m + 1) : I.next[t];
            if (p0 == 0 || p0 == pl1 || p0 == pl) continue;  // above, or no segment
            segment(p0, p1, H[E.X[p0]], H[E.X[p1]]);
        }
    }
    grp.sync();
    if (sa.tblocks) {  // taped forward: bitmap, knot count and end-rule flags of this iteration
        const TapeLayout& L = sa.tl;
        unsigned char* slot =
            sa.tblocks[j / kTapeBlockSlots] + (size_t)(j % kTapeBlockSlots) * L.stride;
        const int words = L.ntiles * (kTileSamples / 32);
        unsigned* bits = reinterpret_cast<unsigned*>(slot) + (size_t)(e * L.nr + r) * words;
        for (int w = tid; w < words; w += G) bits[w] = w < nw ? (unsigned)E.W[w].x : 0u;
        if (tid == 0) {
            reinterpret_cast<int*>(slot + L.off_kc)[e * L.nr + r] = K;
            // a replaced end value differs from the sample in its bits (t > y or t < y)
            (slot + L.off_bf)[e * L.nr + r] = (unsigned char)(
                (__double_as_longlong(I.yend[0]) != __double_as_longlong(H[0]) ? 1 : 0) |
                (__double_as_longlong(I.yend[1]) != __double_as_longlong(H[n - 1]) ? 2 : 0));
        }
    }
    // end relations of the chunk left of each separator
    for (int i = tid; i < ends_items(P); i += G) {
        int p, t, k;
        const bool top = ends_item(i, P, p);
        if (p >= P) continue;
        sep_tile(I, ntiles, p, t, k);
        const int jb = (k - 1) * kChunk, js = min(k * kChunk, I.cnt[t] - 1);
        double* en = E.ends + 6 * p;
        if (k > 0 && js - jb > 1) {
            const int b = I.base[t] + kq(jb);
            if (top) chunk_ends_half<true>(E.X + b, E.S + b, js - jb - 1, en, E.C + b + 1);
            else chunk_ends_half<false>(E.X + b, E.S + b, js - jb - 1, en, nullptr);
        } else if (top) {
            en[3] = 0.0;
            en[4] = 1.0;
            en[5] = 0.0;
        } else {
            en[0] = 0.0;
            en[1] = 0.0;
            en[2] = 1.0;
        }
    }
    if (tid == G - 1) {
        double* en = E.ends + 6 * P;  // after the last separator: empty
        en[0] = 0.0;
        en[1] = 0.0;
        en[2] = 1.0;
        wait();
    }
    grp.sync();
    // the separator rows with the neighbouring chunks eliminated, and their system
    for (int p = tid; p < P; p += G) {
        int t, k;
        sep_tile(I, ntiles, p, t, k);
        const int m = min(k * kChunk, I.cnt[t] - 1), i0 = I.base[t] + kq(m);
        Row sr = identity_row();
        if (i0 != 0 && i0 != pl) {
            const int im = m > 0 ? I.base[t] + kq(m - 1) : I.prev[t];
            sr.l = E.D[im];
            sr.u = E.D[i0];
            sr.m = 2.0 * (sr.l + sr.u);
            sr.r = 3.0 * (E.S[i0] - E.S[im]);
        }
        E.R2[kq(p)] = next_row(sep_row(sr), E.ends + 6 * p);
    }
    grp.sync();
    partition_rows(grp, P, E.R2, E.X2, E.ws);
    // spline values: the separators', then the chunk interiors between them
    for (int p = tid; p < P; p += G) {
        int t, k;
        sep_tile(I, ntiles, p, t, k);
        const int jb = (k - 1) * kChunk, js = min(k * kChunk, I.cnt[t] - 1);
        const double xr = E.X2[kq(p)];
        if (k > 0 && js - jb > 1) {
            const int b = I.base[t] + kq(jb);
            interior_known(E.S + b, E.C + b, E.D + b, js - jb - 1, E.X2[kq(p - 1)], xr);
        }
        E.C[I.base[t] + kq(js > 0 ? js : 0)] = xr;
    }
    grp.sync();
    for (int t = 0; t < ntiles; ++t) {
        const int c = I.cnt[t], b = I.base[t];
        for (int m = tid; m < c; m += G) {
            const int p0 = b + kq(m), p1 = m + 1 < c ? b + kq(m + 1) : I.next[t];
            if (p0 == pl) continue;
            double cb, cd;
            seg_coeffs_int((double)(E.X[p1] - E.X[p0]), E.S[p0], E.C[p0], E.C[p1], cb, cd);
            E.S[p0] = cb;
            E.D[p0] = cd;
        }
    }
}

// The envelope at sample s: the segment of the last knot before it (a rank in the knot bitmap).
__device__ __forceinline__ double env_at(const EnvSmem& E, const double* H, int s) {
    const int2 wo = E.W[s >> 5];
    const int t = s >> 11;
    const int r = wo.y + __popc((unsigned)wo.x & ((1u << (s & 31)) - 1u));
    const int p = r > 0 ? E.I->base[t] + kq(r - 1) : E.I->prev[t];
    const int x = E.X[p];
    const double y = p == 0 ? E.I->yend[0] : H[x];
    return seg_eval(y, E.S[p], E.C[p], E.D[p], (double)(s - x));
}

}  // namespace

size_t small_sift_smem(int n, int mode) { return small_layout(n, mode).total; }

template <int kMode>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_sift_small(const __grid_constant__ SiftArgs a, const __grid_constant__ SmallArgs sa) {
    constexpr int kGroup = kMode == kSmallDual ? kSmallThreads / 2 : kSmallThreads;
    constexpr bool kPair = kMode == kSmallPair;
    constexpr int kWarps = kSmallThreads / 32;
    // samples a thread combines: of its half row, or of the whole row
    constexpr int kOwn = (kPair ? kSmallMaxN / 2 : kSmallMaxN) / kSmallThreads;
    extern __shared__ __align__(16) unsigned char small_smem[];
    __shared__ unsigned s_g[kSmallWords + 1], s_l[kSmallWords + 1];  // signs of h[i] - h[i+1]
    __shared__ int s_part[2 * kWarps];  // counts of every warp of the realization
    __shared__ int s_kcnt[2];           // knot counts, upper and lower
    // how the last iteration's lock-step test ended, as each CTA of the realization saw it
    __shared__ int s_end[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int rank = kPair ? (int)(blockIdx.x & 1) : 0;
    const int nreal = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int n = a.n1, nw = (n + 31) >> 5;
    const SmallLayout L = small_layout(n, kMode);
    double* H = reinterpret_cast<double*>(small_smem + L.H);
    unsigned char* set0 = small_smem + L.H + ((sizeof(double) * (size_t)n + 15) & ~(size_t)15);
    const int group = kMode == kSmallDual ? tid / kGroup : 0;
    const SmallGroup<kGroup> grp{group, kMode == kSmallDual ? tid % kGroup : tid};
    const EnvSmem E0 = env_smem(L, set0);
    const EnvSmem E1 = kMode == kSmallDual ? env_smem(L, set0 + L.set) : E0;
    auto warp_tot = [&](int g) {
        return reinterpret_cast<int*>(set0 + (kMode == kSmallDual ? g * L.set : 0) + L.warp);
    };
    // the half of the row this CTA combines
    const int half = kPair ? small_half(n) : n;
    const int own0 = rank == 0 ? 0 : half, own1 = rank == 0 ? half : n;
    const int oth0 = kPair ? (rank == 0 ? half : 0) : 0, oth1 = kPair ? (rank == 0 ? n : half) : 0;
    double* recv = reinterpret_cast<double*>(set0 + L.recv);  // the other CTA's envelope, own half
    double* recv_peer = nullptr;
    int *part_peer = nullptr, *kcnt_peer = nullptr, *end_peer = nullptr;
    if constexpr (kPair) {
        cg::cluster_group cl = cg::this_cluster();
        recv_peer = cl.map_shared_rank(recv, rank ^ 1);
        part_peer = cl.map_shared_rank(s_part, rank ^ 1);
        kcnt_peer = cl.map_shared_rank(s_kcnt, rank ^ 1);
        end_peer = cl.map_shared_rank(s_end, rank ^ 1);
    }
    ChanState& cst = a.cs[0];
    const int cap = cst.cap;
    const size_t base = (size_t)r * row_ld(n);
    double* mode = cst.mode_out + (size_t)r * n;
    double* menv = a.menv + base;
    double* up = sa.up + base;
    const double* hin = a.h[0] + base;  // the stage input
    const double inv_n = 1.0 / (double)n;
    for (int i = tid; i < n; i += kSmallThreads) H[i] = hin[i];
    if (tid == 0) {
        s_g[0] = s_l[0] = 0u;
        s_end[0] = s_end[1] = kGoOn;
    }
    // every thread carries the realization's state (the same values)
    double frac = a.frac[r];
    int mark = -1, fin = 0;
    double mean[kOwn];  // the mean envelope at the thread's own samples
#pragma unroll
    for (int k = 0; k < kOwn; ++k) mean[k] = 0.0;
    __syncthreads();
    if constexpr (kPair) cg::this_cluster().sync();  // the other CTA has started

    // deferred update of the previous iteration (updateRealizations), or the mode of a realization
    // that finished in it
    auto update = [&]() {
        if (mark == 1) {
            // (the other half's mean envelope is on its way while the own half is subtracted)
            double ov[kPair ? kOwn : 1];
            if constexpr (kPair) {
#pragma unroll
                for (int k = 0; k < kOwn; ++k) {
                    const int s = oth0 + k * kSmallThreads + tid;
                    ov[k] = s < oth1 ? __ldcg(menv + s) : 0.0;
                }
            }
#pragma unroll
            for (int k = 0; k < kOwn; ++k) {
                const int s = own0 + k * kSmallThreads + tid;
                if (s < own1) H[s] = H[s] - mean[k];
            }
            if constexpr (kPair) {
#pragma unroll
                for (int k = 0; k < kOwn; ++k) {
                    const int s = oth0 + k * kSmallThreads + tid;
                    if (s < oth1) H[s] = H[s] - ov[k];
                }
            }
        } else if (mark == 0) {
            for (int s = own0 + tid; s < own1; s += kSmallThreads) mode[s] = H[s];
        }
    };

    int j = 0;
    int end = kGoOn;  // else by the lock-step test: iteration j's work is discarded
    for (; j < cap; ++j) {
        update();
        __syncthreads();
        for (int w = warp; w < nw; w += kWarps) {
            const int i = 32 * w + lane;
            const double x = i < n ? H[i] : 0.0, y = i + 1 < n ? H[i + 1] : x;
            const unsigned g = __ballot_sync(0xffffffffu, x > y);
            const unsigned l = __ballot_sync(0xffffffffu, x < y);
            if (lane == 0) {
                s_g[w + 1] = g;
                s_l[w + 1] = l;
            }
        }
        __syncthreads();
        // the lock-step test of the previous iteration, awaited by one thread under the sweeps
        auto wait = [&]() {
            if (j == 0 || a.forced > 0) return;
            const volatile unsigned long long* word = sa.arrive + (j - 1);
            const unsigned target = (unsigned)nreal + (rank == 0 ? sa.extra : 0u);
            int spins = 0;
            unsigned long long v = *word;
            while ((unsigned)v < target) {
                if (++spins > sa.spin_limit) {
                    s_end[rank] = kGaveUp;
                    return;
                }
                __nanosleep(32);
                v = *word;
            }
            if ((int)(v >> 32) == nreal) s_end[rank] = kStop;
        };
        // (one copy of build_envelope's code, for the instruction cache)
        if constexpr (kMode == kSmallSingle) {
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                build_envelope(grp, E0, warp_tot(0), H, s_g, s_l, n, e, sa, j, r, [&]() {
                    if (e == 0) wait();
                });
                // (before the barrier: every thread decides by both counts)
                if (tid == 0) s_kcnt[e] = E0.I->K;
                __syncthreads();
                if (e == 0) {
#pragma unroll 4
                    for (int s = tid; s < n; s += kSmallThreads) up[s] = env_at(E0, H, s);
                    __syncthreads();
                }
            }
        } else if constexpr (kMode == kSmallDual) {
            const EnvSmem E = env_smem(L, set0 + group * L.set);
            build_envelope(grp, E, warp_tot(group), H, s_g, s_l, n, group, sa, j, r, [&]() {
                if (group == 0) wait();
            });
            if (grp.tid() == 0) s_kcnt[group] = E.I->K;
            __syncthreads();
        } else {
            build_envelope(grp, E0, warp_tot(0), H, s_g, s_l, n, rank, sa, j, r, wait);
            // the solve's workspace (recv) is free in both CTAs, coefficients ready
            cg::this_cluster().sync();
            if (tid == 0) {
                s_kcnt[rank] = kcnt_peer[rank] = E0.I->K;
                end_peer[rank] = s_end[rank];
            }
#pragma unroll 4
            for (int s = oth0 + tid; s < oth1; s += kSmallThreads)
                recv_peer[s - oth0] = env_at(E0, H, s);
            cg::this_cluster().barrier_arrive();
        }
        double ev[kPair ? kOwn : 1];
        if constexpr (kPair) {
#pragma unroll
            for (int k = 0; k < kOwn; ++k) {
                const int s = own0 + k * kSmallThreads + tid;
                ev[k] = s < own1 ? env_at(E0, H, s) : 0.0;
            }
            cg::this_cluster().barrier_wait();
        }
        // The previous iteration was the stage's last, or a wait gave up.  Both CTAs of a pair know
        // what either saw, so they leave together: one that went on alone would write to the
        // other's shared memory after its exit.
        end = kPair ? max(s_end[0], s_end[1]) : s_end[0];
        if (end != kGoOn) break;
        const int kmax = s_kcnt[0], kmin = s_kcnt[1];
        const bool write_mean = kmax > 3 && kmin > 3;
        // the envelopes at the thread's sample k
        auto envelopes = [&](int k, int s, double& u, double& v) {
            if constexpr (kPair) {
                const double o = recv[s - own0];
                u = rank == 0 ? ev[k] : o;
                v = rank == 0 ? o : ev[k];
            } else {
                u = kMode == kSmallSingle ? up[s] : env_at(E0, H, s);
                v = env_at(E1, H, s);
            }
        };
        // sx > sd, sx > sd2 by the signs of p - q t for bounds t around the thresholds, as in
        // k_tile_sift; a thread with an undecided sample or a NaN does its samples again
        int cnt = 0, any = 0, und = 0, smax = 0, amax = -1, bmax = -1;
#pragma unroll
        for (int k = 0; k < kOwn; ++k) {
            const int s = own0 + k * kSmallThreads + tid;
            if (s < own1) {
                double u, v;
                envelopes(k, s, u, v);
                const double sum = u + v, p = fabs(sum), w = fabs(u - v);
                if (write_mean) {
                    mean[k] = sum / 2.0;
                    menv[s] = mean[k];
                } else {
                    mean[k] = __ldcg(menv + s);
                }
                const int s1 = __double2hiint(fma(-a.sd_hi, w, p));
                const int s0 = __double2hiint(fma(-a.sd_lo, w, p));
                und |= (s1 - 1) & ~s0;
                cnt += 1 - (int)((unsigned)s0 >> 31);
                smax = max(smax, s1);
                amax = max(amax, __double2hiint(fma(-a.sd2_hi, w, p)));
                bmax = max(bmax, __double2hiint(fma(-a.sd2_lo, w, p)));
            }
        }
        any = amax > 0 ? 1 : 0;
        if (und < 0 || smax > 0x7ff00000 || (amax <= 0 && bmax >= 0)) {
            cnt = any = 0;
#pragma unroll (kPair ? kOwn : 1)
            for (int k = 0; k < kOwn; ++k) {
                const int s = own0 + k * kSmallThreads + tid;
                if (s < own1) {
                    double u, v;
                    envelopes(k, s, u, v);
                    any |= sx_greater(u, v, a.sd2) ? 1 : 0;
                    cnt += sx_greater(u, v, a.sd) ? 1 : 0;
                }
            }
        }
        any = __any_sync(0xffffffffu, any != 0) ? 1 : 0;
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) {
            const int v = cnt | any << 30;
            s_part[rank * kWarps + warp] = v;
            if constexpr (kPair) part_peer[rank * kWarps + warp] = v;
        }
        if constexpr (kPair) {
            cg::this_cluster().sync();
        } else {
            __syncthreads();
        }
        const int v = lane < (kPair ? 2 : 1) * kWarps ? s_part[lane] : 0;
        const int c = __reduce_add_sync(0xffffffffu, v & 0x3fffffff);
        const bool y = __any_sync(0xffffffffu, (v >> 30) != 0);
        // the sifting-fraction carry and siftingCriterion (as row_criterion)
        frac = (frac + (double)c) * inv_n;
        const bool crit = frac > a.tol || (y && kmax + kmin > 6);
        mark = 1;
        if (fin == 0 && (!crit || j == cap - 1)) {
            mark = 0;
            fin = 1;
        }
        if (tid == kSmallThreads - 1 && rank == 0) {
            if (sa.tblocks)
                reinterpret_cast<signed char*>(sa.tblocks[j / kTapeBlockSlots] +
                                               (size_t)(j % kTapeBlockSlots) * sa.tl.stride +
                                               sa.tl.off_mark)[r] = (signed char)mark;
            atomicAdd(&cst.knots, (unsigned long long)(kmax + kmin));
            // the lock-step test: one more realization here, finished or not
            atomicAdd(sa.arrive + j, 1ull | (unsigned long long)fin << 32);
        }
        if (a.forced > 0 && j + 1 >= a.forced) {
            ++j;
            break;
        }
    }
    if (end == kGaveUp) {  // the host reports CEEMDAN_ERR_TIMEOUT
        if (tid == 0) atomicExch(&cst.err, kErrTimeout);
        return;
    }
    if (end == kGoOn && mark == 0) update();  // the modes of the last iteration
    if (tid == 0 && rank == 0) {
        a.frac[r] = frac;
        if (r == 0) {
            cst.iter = j;
            cst.iters += (unsigned long long)j;
            cst.done = 1;
        }
    }
    if constexpr (kPair) cg::this_cluster().sync();  // no CTA leaves while the other may write to it
}

template __global__ void k_sift_small<kSmallPair>(const __grid_constant__ SiftArgs,
                                                  const __grid_constant__ SmallArgs);
template __global__ void k_sift_small<kSmallDual>(const __grid_constant__ SiftArgs,
                                                  const __grid_constant__ SmallArgs);
template __global__ void k_sift_small<kSmallSingle>(const __grid_constant__ SiftArgs,
                                                    const __grid_constant__ SmallArgs);

}  // namespace ceemdan
