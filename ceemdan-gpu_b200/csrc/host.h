// Host-side internals shared by the engine's translation units (engine.cu, batch.cu): error
// text and launch counter, the library's stream-ordered memory pool, workspaces, the tape of
// the reverse pass and the sift engine that launches one iteration of the sift kernels.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ceemdan_b200.h"
#include "canon.cuh"
#include "kernels.h"

namespace ceemdan {

extern thread_local std::string g_last_error;  // last error text of the calling thread
extern std::atomic<uint64_t> g_launches;        // kernels launched by the library

#define CK(call)                                                                       \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            g_last_error = std::string(#call) + ": " + cudaGetErrorString(e_);         \
            return e_ == cudaErrorMemoryAllocation ? CEEMDAN_ERR_NO_MEMORY            \
                                                   : CEEMDAN_ERR_CUDA;                 \
        }                                                                              \
    } while (0)

#define CKS(expr)                              \
    do {                                       \
        ceemdan_status s_ = (expr);            \
        if (s_ != CEEMDAN_OK) return s_;       \
    } while (0)

constexpr int kThreads = 256;

// The tile kernels run as persistent CTAs over the active tiles.  kEnv: the envelopes of one
// iteration to dbg_upper / dbg_lower, no update and no stop test.  kDense: shared memory for
// kSiftDense entries (three CTAs per SM) or kSiftSparse (five).
// kExtrema: the knots alone.
template <bool kExtrema>
__global__ void k_tile_knots(const __grid_constant__ SiftArgs a);
// kSplit: of the rows of its class only.
template <bool kDense, bool kSplit, bool kEnv>
__global__ void k_tile_sift(const __grid_constant__ SiftArgs a);
template <bool kExtrema>
__global__ void k_spline_solve(const __grid_constant__ SiftArgs a);
__global__ void k_gather_knots(const __grid_constant__ SiftArgs a, int32_t* kx_max,
                               double* ky_max, int32_t* kx_min, double* ky_min);

// the on-chip stage kernel, in one of its three forms
template <int kMode>
__global__ void k_sift_small(const __grid_constant__ SiftArgs a,
                             const __grid_constant__ SmallArgs sa);

int sm_count();
cudaMemPool_t engine_pool();
ceemdan_status pool_alloc(void** p, size_t bytes, cudaStream_t st);
int* pinned_state();
void release_pinned_state(int* p);
void sx_bounds(double t, double* hi, double* lo);
int grid_for(size_t count);
ceemdan_status generate_noise(double* w, size_t count, uint64_t seed, cudaStream_t st);

// Device allocations owned by one decomposition (or one stage-level call), stream-ordered on
// the call's stream: freed after the work queued on it.  A counting workspace allocates nothing
// and only adds up what the pool would hand out (its granule is 512 bytes).
struct Workspace {
    cudaStream_t st;
    std::vector<void*> blocks;
    bool counting = false;
    size_t total = 0;
    explicit Workspace(cudaStream_t s, bool count = false) : st(s), counting(count) {}
    Workspace(const Workspace&) = delete;
    Workspace& operator=(const Workspace&) = delete;
    ceemdan_status alloc(void** p, size_t bytes) {
        total += (std::max<size_t>(bytes, 1) + 511) & ~(size_t)511;
        if (counting) {
            *p = nullptr;
            return CEEMDAN_OK;
        }
        const ceemdan_status s = pool_alloc(p, bytes, st);
        if (s == CEEMDAN_OK) blocks.push_back(*p);
        return s;
    }
    template <class T>
    ceemdan_status alloc_n(T** p, size_t count) {
        return alloc(reinterpret_cast<void**>(p), count * sizeof(T));
    }
    ~Workspace() {
        for (void* p : blocks) cudaFreeAsync(p, st);
    }
};

}  // namespace ceemdan

// Frozen structure of one taped forward call (opaque in the C ABI): one tape slot per executed
// iteration of every signal stage (ceemdan::TapeLayout), in device blocks of kBlockSlots
// slots, plus what the reverse pass of the stage statistics needs: the noise modes, each
// stage's input (y for stage 0, the previous ensemble mean after it) and its carried mean and
// variance.  All of it comes from the library's memory pool.
struct ceemdan_tape {
    static constexpr int kBlockSlots = ceemdan::kTapeBlockSlots;
    struct Stage {
        int J = 0;
        std::vector<unsigned char*> blocks;
    };
    int device = 0;
    size_t nr = 0, n = 0, nimf = 0;
    double nstd = 0.0;
    ceemdan::TapeLayout L{};
    std::vector<Stage> stages;
    double* E = nullptr;      // num_imfs*nr*n
    double* fin = nullptr;    // (num_imfs-1)*n
    double* stats = nullptr;  // 2*(num_imfs-1): mean, variance
    size_t bytes = 0;
    // checkpointed form: instead of the iterations, each stage's input h0 [nr*n] and the
    // mean-envelope [nr*n] and sifting-fraction [nr] carries it started from (the whole state
    // its sift depends on); the reverse pass re-runs the stage from them with the forward's
    // options and sift cap
    bool checkpointed = false;
    double* ck = nullptr;     // (num_imfs-1) * (2*nr*n + nr)
    ceemdan_options opts{};
    size_t max_iter = 0;

    size_t ck_stride() const { return 2 * nr * n + nr; }

    const unsigned char* slot(size_t stage, long j) const {
        return stages[stage].blocks[(size_t)j / kBlockSlots] + (size_t)(j % kBlockSlots) * L.stride;
    }
    ceemdan_status alloc(void** p, size_t b, cudaStream_t st) {
        const ceemdan_status s = ceemdan::pool_alloc(p, b, st);
        if (s == CEEMDAN_OK) bytes += b;
        return s;
    }
    // slot j of a stage being recorded (its block allocated on first use, on st); null when
    // out of device memory
    unsigned char* grow(size_t stage, long j, cudaStream_t st) {
        auto& b = stages[stage].blocks;
        while (b.size() <= (size_t)j / kBlockSlots) {
            void* p = nullptr;
            if (alloc(&p, (size_t)kBlockSlots * L.stride, st) != CEEMDAN_OK) return nullptr;
            b.push_back(static_cast<unsigned char*>(p));
        }
        return b[(size_t)j / kBlockSlots] + (size_t)(j % kBlockSlots) * L.stride;
    }
    // free the blocks past the stage's J executed iterations (after the work queued on st)
    void trim(size_t stage, cudaStream_t st) {
        auto& b = stages[stage].blocks;
        const size_t keep = ((size_t)stages[stage].J + kBlockSlots - 1) / kBlockSlots;
        while (b.size() > keep) {
            cudaFreeAsync(b.back(), st);
            b.pop_back();
            bytes -= (size_t)kBlockSlots * L.stride;
        }
    }
    // free every block after the work queued on st (the tape keeps its other buffers)
    void free_blocks(cudaStream_t st) {
        for (size_t i = 0; i < stages.size(); ++i) {
            for (unsigned char* p : stages[i].blocks) cudaFreeAsync(p, st);
            bytes -= stages[i].blocks.size() * (size_t)kBlockSlots * L.stride;
            stages[i].blocks.clear();
        }
    }
    // every call that used the tape has returned (they are synchronous): free on this
    // thread's stream of the tape's device
    ~ceemdan_tape() {
        int cur = -1;
        const bool other = cudaGetDevice(&cur) == cudaSuccess && cur != device;
        if (other) cudaSetDevice(device);
        for (auto& s : stages)
            for (unsigned char* p : s.blocks) cudaFreeAsync(p, cudaStreamPerThread);
        for (void* p : {(void*)E, (void*)fin, (void*)stats, (void*)ck})
            if (p) cudaFreeAsync(p, cudaStreamPerThread);
        if (other) cudaSetDevice(cur);
    }
};

namespace ceemdan {

// One channel of a sift engine: nr realizations of n samples.
struct ChanSpec {
    int n, nr;
};

// Sifting state of one or several channels (shared by all stages of a call).  With one
// channel, run_stage drives the lock-step sift of a stage from the host; the batched engine
// (batch.cu) drives several channels from the device.
struct SiftEngine {
    SiftArgs a{};
    double* h[2] = {nullptr, nullptr};
    ChanState* cs = nullptr;  // device [nchan]
    int* state = nullptr;     // channel 0's (done, iter, err, cap) = the first words of cs[0]
    int* hstate = nullptr;    // pinned host mirror: two slots of (done, iter, err, cap)
    std::vector<Chan> hchan;  // host copy of the channel table
    Chan* dchan = nullptr;
    int nr = 0, n = 0, ntiles = 0;  // channel 0
    size_t samples = 0;             // of one plane (all channels' row blocks)
    cudaEvent_t group_ev[2] = {nullptr, nullptr};
    int group = 4;
    // persistent grids of the tile kernels, one CTA per spline
    int knots_grid = 0, dense_grid = 0, sift_grid = 0, solve_grid = 0;
    double* kernel_ms = nullptr;           // host accumulators (optional)
    std::vector<cudaEvent_t> ev;           // [group][kinds][2] when timing
    ceemdan_tape* tape = nullptr;          // taped forward: the stage being recorded
    size_t tape_stage = 0;
    bool plan_by_caller = false;           // the batched loop computes the plan (k_commit_plan)

    ceemdan_status init(Workspace& ws, int nr_, int n_, const ceemdan_options& o) {
        return init(ws, std::vector<ChanSpec>{{n_, nr_}}, o);
    }

    // Device bytes of an engine for nr rows of n samples (its arrays, without enable_small's).
    static size_t bytes_of(size_t n_, size_t nr_) {
        SiftEngine e;
        Workspace count(nullptr, true);
        if (e.layout({{(int)n_, (int)nr_}}) == CEEMDAN_OK) (void)e.arrays(count);
        return count.total;
    }

    ceemdan_status init(Workspace& ws, const std::vector<ChanSpec>& chans,
                        const ceemdan_options& o) {
        CKS(layout(chans));
        CKS(arrays(ws));
        return start(ws, o);
    }

    // The rows' places in the arrays.
    ceemdan_status layout(const std::vector<ChanSpec>& chans) {
        const int nchan = (int)chans.size();
        hchan.resize(chans.size());
        long long rows = 0, tiles = 0, samp = 0, rec = 0, red = 0;
        for (int c = 0; c < nchan; ++c) {
            Chan& ch = hchan[c];
            std::memset(&ch, 0, sizeof(ch));
            ch.n = chans[c].n;
            ch.nr = chans[c].nr;
            ch.ntiles = (ch.n + kTileSamples - 1) / kTileSamples;
            ch.cap = ch.n / 2 + 2;
            // separators per spline: per tile with c knots (c + 14)/16 + 1, so at most
            // K/16 + 2*ntiles over the spline (K <= cap)
            ch.rec_stride = ((ch.cap + kChunk - 1) / kChunk + 2 * ch.ntiles + 8 + 3) & ~3;
            ch.row0 = (int)rows;
            ch.tile0 = (int)tiles;
            ch.samp0 = samp;
            ch.rec0 = rec;
            ch.red0 = red;
            rows += ch.nr;
            tiles += (long long)ch.nr * ch.ntiles;
            // every channel's block of rows starts 256-byte aligned (16-byte sample pairs)
            samp += ((long long)ch.nr * row_ld(ch.n) + 31) & ~31LL;
            rec += (long long)ch.nr * ch.rec_stride;
            red += (long long)ch.nr * red_stride_of(ch.rec_stride);
        }
        if (rows > 0x3fffffffLL || tiles > 0x3fffffffLL) {
            g_last_error = "too many realizations or tiles for one engine";
            return CEEMDAN_ERR_INVALID_ARG;
        }
        nr = hchan[0].nr;
        n = hchan[0].n;
        ntiles = hchan[0].ntiles;
        a.n1 = n;
        a.ntiles1 = ntiles;
        a.nr1 = nr;
        a.rs1 = hchan[0].rec_stride;
        a.nrows = (int)rows;
        a.nchan = nchan;
        a.ntot = (int)tiles;
        a.rec_total = rec;
        a.red_total = red;
        samples = (size_t)samp;
        return CEEMDAN_OK;
    }

    ceemdan_status arrays(Workspace& ws) {
        const size_t R = (size_t)a.nrows, T = (size_t)a.ntot, S = samples;
        CKS(ws.alloc_n(&h[0], S));
        CKS(ws.alloc_n(&h[1], S));
        a.h[0] = h[0];
        a.h[1] = h[1];
        CKS(ws.alloc_n(&a.menv, S));
        CKS(ws.alloc_n(&a.mark, R));
        CKS(ws.alloc_n(&a.finish, R));
        CKS(ws.alloc_n(&a.frac, R));
        CKS(ws.alloc_n(&a.cnt, R));
        CKS(ws.alloc_n(&a.any, R));
        CKS(ws.alloc_n(&a.kcount, 2 * R));
        CKS(ws.alloc_n(&a.par, R));
        CKS(ws.alloc_n(&a.acc, R));
        CKS(ws.alloc_n(&a.acc_wide, 2 * R));
        CKS(ws.alloc_n(&a.cmax, 2 * R));
        CKS(ws.alloc_n(&a.cls_count, 2));
        CKS(ws.alloc_n(&a.cls_row, 2 * R));
        CKS(ws.alloc_n(&a.cls_wait, R));
        CKS(ws.alloc_n(&a.tile_cnt, 2 * T));
        CKS(ws.alloc_n(&a.plan, 2 * (size_t)a.nchan + 2));
        CKS(ws.alloc_n(&a.bitmap, 2 * T * (kTileSamples / 32)));
        CKS(ws.alloc_n(&a.scan, T));
        CKS(ws.alloc_n(&a.list_x, 2 * T * kListSlots));
        CKS(ws.alloc_n(&a.list_s, 2 * T * kListSlots));
        CKS(ws.alloc_n(&a.hdr, 2 * T));
        CKS(ws.alloc_n(&a.edge, 2 * T));
        CKS(ws.alloc_n(&a.rows, 2 * T * kRowSlots * 4));
        CKS(ws.alloc_n(&a.sep_off, 2 * (T + R)));
        CKS(ws.alloc_n(&a.tile_rank, 2 * (T + R)));
        CKS(ws.alloc_n(&a.tile_list, 2 * (T + R)));
        CKS(ws.alloc_n(&a.yend, 2 * R * 2));
        CKS(ws.alloc_n(&a.end_x, 2 * R * 2 * kEndKnots));
        CKS(ws.alloc_n(&a.end_y, 2 * R * 2 * kEndKnots));
        // (k_tile_sift copies a whole tile's slots from a tile's first separator on)
        CKS(ws.alloc_n(&a.xsep, 2 * (size_t)a.rec_total + kRowSlots));
        CKS(ws.alloc_n(&a.red, 2 * (size_t)a.red_total));
        CKS(ws.alloc_n(&dchan, (size_t)a.nchan));
        a.chan = dchan;
        CKS(ws.alloc_n(&cs, (size_t)a.nchan));
        a.cs = cs;
        return CEEMDAN_OK;
    }

    // The options, the channel table and the launch shapes.
    ceemdan_status start(Workspace& ws, const ceemdan_options& o) {
        const size_t R = (size_t)a.nrows, T = (size_t)a.ntot;
        a.sd = o.sd;
        a.sd2 = o.sd2;
        sx_bounds(o.sd, &a.sd_hi, &a.sd_lo);
        sx_bounds(o.sd2, &a.sd2_hi, &a.sd2_lo);
        a.tol = o.tol;
        // counts of rows of up to 2^17 - 1 tiles fit one word (CEEMDAN_SPLIT_COUNT=1: never)
        a.count_bits = 17;
        if (const char* e = std::getenv("CEEMDAN_SPLIT_COUNT"))
            if (e[0] == '1') a.count_bits = 0;
        CK(cudaMemcpyAsync(dchan, hchan.data(), sizeof(Chan) * a.nchan, cudaMemcpyHostToDevice,
                           ws.st));
        state = reinterpret_cast<int*>(cs);
        hstate = pinned_state();
        if (!hstate) {
            g_last_error = "cudaMallocHost failed";
            return CEEMDAN_ERR_NO_MEMORY;
        }
        CK(cudaEventCreateWithFlags(&group_ev[0], cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&group_ev[1], cudaEventDisableTiming));
        const size_t rn = samples;
        if (o.group > 0) {
            group = o.group;
        } else {
            group = rn >= (size_t)(1 << 22) ? 4 : (rn >= (size_t)(1 << 18) ? 8 : 32);
        }
        a.solve_wcap = (kSolveSmem - kSolveStage) / (int)sizeof(double);
        CK(cudaFuncSetAttribute(k_spline_solve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSolveSmem));
        for (auto k : {k_tile_sift<false, true, false>, k_tile_sift<false, true, true>})
            CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tile_sift_smem(false)));
        for (auto k : {k_tile_sift<true, false, false>, k_tile_sift<true, false, true>,
                       k_tile_sift<true, true, false>, k_tile_sift<true, true, true>})
            CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tile_sift_smem(true)));
        for (auto k : {k_tile_knots<false>, k_tile_knots<true>})
            CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tile_knots_smem()));
        // persistent CTAs, as many as the GPU holds at once
        auto grid = [&](const void* k, size_t smem) {
            int per = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kTileThreads, smem);
            return std::max(1, (int)std::min<size_t>(T, (size_t)std::max(1, per) * sm_count()));
        };
        knots_grid = grid((const void*)k_tile_knots<false>, tile_knots_smem());
        dense_grid = grid((const void*)k_tile_sift<true, true, false>, tile_sift_smem(true));
        sift_grid = grid((const void*)k_tile_sift<false, true, false>, tile_sift_smem(false));
        CK(cudaGetLastError());
        // as many tiles as the dense form holds at once: one launch does for all rows
        a.sift_split = (size_t)dense_grid < T ? 1 : 0;
        solve_grid = (int)std::max<size_t>(1, 2 * R);
        return CEEMDAN_OK;
    }

    ~SiftEngine() {
        if (hstate) release_pinned_state(hstate);
        for (cudaEvent_t e : group_ev)
            if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
    }

    // kernels of one sift iteration
    int sift_kernels() const { return a.sift_split ? 4 : 3; }

    // kinds timed per iteration (the on-chip stage kernel is timed per launch): the three
    // kernels of an iteration report under the kinds of their main steps
    static constexpr int kIterKinds = 3;
    static constexpr int kIterKind[kIterKinds] = {CEEMDAN_K_EXTREMA, CEEMDAN_K_REDUCED_SOLVE,
                                                  CEEMDAN_K_EVAL};

    ceemdan_status enable_timing(double* ms) {
        kernel_ms = ms;
        ev.resize((size_t)2 * group * kIterKinds * 2 + 2);
        for (auto& e : ev) CK(cudaEventCreate(&e));
        return CEEMDAN_OK;
    }

    cudaEvent_t event(int it, int kind, int end) {
        return ev[((size_t)it * kIterKinds + kind) * 2 + end];
    }

    // Add the event-timed durations of iterations [first, first+count) (completed).
    void harvest_timing(long first, long count) {
        if (!kernel_ms) return;
        for (long j = first; j < first + count; ++j) {
            const int it = (int)(j % (2 * group));
            for (int k = 0; k < kIterKinds; ++k) {
                float ms = 0.f;
                if (cudaEventElapsedTime(&ms, event(it, k, 0), event(it, k, 1)) == cudaSuccess)
                    kernel_ms[kIterKind[k]] += ms;
            }
        }
    }

    // Rows of the engine's planes (row_ld(n) apart) from and to contiguous rows of n samples, rows
    // r0 .. r0 + rows - 1 of channel 0.
    ceemdan_status rows_in(double* plane, const double* src, size_t rows, cudaStream_t st) {
        const size_t w = sizeof(double) * (size_t)n;
        if (row_ld(n) == n)
            CK(cudaMemcpyAsync(plane, src, w * rows, cudaMemcpyDeviceToDevice, st));
        else
            CK(cudaMemcpy2DAsync(plane, sizeof(double) * row_ld(n), src, w, w, rows,
                                 cudaMemcpyDeviceToDevice, st));
        return CEEMDAN_OK;
    }
    ceemdan_status rows_out(double* dst, const double* plane, size_t rows, cudaStream_t st) {
        const size_t w = sizeof(double) * (size_t)n;
        if (row_ld(n) == n)
            CK(cudaMemcpyAsync(dst, plane, w * rows, cudaMemcpyDeviceToDevice, st));
        else
            CK(cudaMemcpy2DAsync(dst, w, plane, sizeof(double) * row_ld(n), w, rows,
                                 cudaMemcpyDeviceToDevice, st));
        return CEEMDAN_OK;
    }

    // Zero the whole-call carries: mean envelope and sifting fraction accumulator, and the
    // channels' states.  mean false: without the mean envelope, for the stage-level entries that
    // neither read nor write it.
    ceemdan_status reset_carries(cudaStream_t st, bool mean = true) {
        const Chan& last = hchan.back();
        const size_t S = (size_t)last.samp0 + (size_t)last.nr * row_ld(last.n);
        if (mean) CK(cudaMemsetAsync(a.menv, 0, sizeof(double) * S, st));
        CK(cudaMemsetAsync(a.frac, 0, sizeof(double) * a.nrows, st));
        CK(cudaMemsetAsync(a.cnt, 0, sizeof(unsigned) * a.nrows, st));
        CK(cudaMemsetAsync(a.any, 0, sizeof(int) * a.nrows, st));
        CK(cudaMemsetAsync(a.par, 0, sizeof(int) * a.nrows, st));
        CK(cudaMemsetAsync(a.acc, 0, sizeof(*a.acc) * a.nrows, st));
        CK(cudaMemsetAsync(a.cls_wait, 0, sizeof(unsigned) * a.nrows, st));
        CK(cudaMemsetAsync(a.acc_wide, 0, sizeof(*a.acc_wide) * 2 * a.nrows, st));
        CK(cudaMemsetAsync(cs, 0, sizeof(ChanState) * a.nchan, st));
        return CEEMDAN_OK;
    }

    // Launch one sift iteration of every channel whose stage runs.
    ceemdan_status launch_iteration(long j, cudaStream_t st) {
        unsigned char* slot = nullptr;
        if (tape) {
            slot = tape->grow(tape_stage, j, st);
            if (!slot) {
                g_last_error = "out of device memory for the tape";
                return CEEMDAN_ERR_NO_MEMORY;
            }
        }
        a.tape_mark = slot ? reinterpret_cast<signed char*>(slot + tape->L.off_mark) : nullptr;
        const bool timed = kernel_ms != nullptr;
        const int ti = (int)(j % (2 * group));
        // inside a stream capture an event record becomes a graph node only as an external
        // event (a plain record would only order the capture)
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (timed) cudaStreamIsCapturing(st, &cap);
        const unsigned ev_flags =
            cap == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
        auto mark_ev = [&](int kind, int end) {
            if (timed) cudaEventRecordWithFlags(event(ti, kind, end), st, ev_flags);
        };
        if (a.nchan > 1 && !plan_by_caller) {
            k_plan<<<1, 1024, 0, st>>>(a);
            ++g_launches;
        }
        mark_ev(0, 0);
        k_tile_knots<false><<<knots_grid, kTileThreads, tile_knots_smem(), st>>>(a);
        mark_ev(0, 1);
        mark_ev(1, 0);
        k_spline_solve<false><<<solve_grid, kSolveThreads, kSolveSmem, st>>>(a);
        mark_ev(1, 1);
        if (slot) {
            const size_t pieces = tape->L.off_kc / 16;  // 16-byte pieces of the bitmaps
            const unsigned g = (unsigned)std::min<size_t>((pieces + kThreads - 1) / kThreads,
                                                          (size_t)sm_count() * 8);
            k_tape_record<<<g, kThreads, 0, st>>>(a, tape->L, slot);
            ++g_launches;
        }
        mark_ev(2, 0);
        auto sift = [&](auto one, auto dense, auto sparse) {
            const size_t sd = tile_sift_smem(true), ss = tile_sift_smem(false);
            if (!a.sift_split) {
                one<<<dense_grid, kTileThreads, sd, st>>>(a);
                return;
            }
            dense<<<dense_grid, kTileThreads, sd, st>>>(a);
            sparse<<<sift_grid, kTileThreads, ss, st>>>(a);
        };
        if (a.dbg_upper)
            sift(k_tile_sift<true, false, true>, k_tile_sift<true, true, true>,
                 k_tile_sift<false, true, true>);
        else
            sift(k_tile_sift<true, false, false>, k_tile_sift<true, true, false>,
                 k_tile_sift<false, true, false>);
        mark_ev(2, 1);
        g_launches += sift_kernels();
        CK(cudaGetLastError());
        return CEEMDAN_OK;
    }

    // Lock-step sift of all realizations of channel 0 until every one has finished (or cap).
    // h[0] holds the stage input; modes are written to mode_out.  Iterations are launched in
    // groups; the host reads the stop word of group g while group g+1 is already queued, so
    // the device never waits for the host.  Iterations after the stop word is set return
    // at once.
    // Short rows (one channel, n <= kSmallMaxN, every realization a CTA resident at once):
    // a stage runs as one cooperative launch of k_sift_small instead of groups of iterations.
    bool small = false;
    SmallArgs sa{};
    int small_mode = -1;

    // Launch configuration of the on-chip kernel in form `mode` (attributes in `at`).
    cudaLaunchConfig_t small_config(int mode, cudaLaunchAttribute* at, cudaStream_t st) const {
        cudaLaunchConfig_t c{};
        c.gridDim = dim3((unsigned)(mode == kSmallPair ? 2 * nr : nr));
        c.blockDim = dim3(kSmallThreads);
        // (one CTA to an SM whatever its shared memory: 512 threads of more than 64 registers)
        c.dynamicSmemBytes = small_sift_smem(n, mode);
        c.stream = st;
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = 2;
        at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
        c.attrs = at;
        c.numAttrs = mode == kSmallPair ? 2 : 1;
        return c;
    }
    static const void* small_kernel(int mode) {
        return mode == kSmallPair   ? (const void*)k_sift_small<kSmallPair>
               : mode == kSmallDual ? (const void*)k_sift_small<kSmallDual>
                                    : (const void*)k_sift_small<kSmallSingle>;
    }

    ceemdan_status enable_small(Workspace& ws, int max_cap, int spin_limit) {
        if (a.nchan != 1 || n > kSmallMaxN) return CEEMDAN_OK;
        if (const char* e = std::getenv("CEEMDAN_SMALL"))
            if (e[0] == '0') return CEEMDAN_OK;
        int dev = 0, coop = 0, most = 0, per = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        CK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        if (!coop) return CEEMDAN_OK;
        // The statically declared shared memory counts too; the attribute is the same for every
        // size, so that concurrent calls of other sizes agree on it.
        const size_t room = (size_t)most - 4096;
        for (int m : {kSmallPair, kSmallDual, kSmallSingle})
            CK(cudaFuncSetAttribute(small_kernel(m), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)room));
        // Two CTAs per realization when they fit one per SM as clusters (CEEMDAN_SMALL_PAIR=0:
        // one CTA); else both envelopes side by side in one CTA when the shared memory holds
        // them (rows of up to about 5000 samples), else one after the other.
        small_mode = -1;
        const char* pe = std::getenv("CEEMDAN_SMALL_PAIR");
        cudaLaunchAttribute at[2];
        if (2 * nr <= sm_count() && !(pe && pe[0] == '0') &&
            small_sift_smem(n, kSmallPair) <= room) {
            cudaLaunchConfig_t c = small_config(kSmallPair, at, nullptr);
            c.attrs = at + 1;  // the cluster dimension alone
            c.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, small_kernel(kSmallPair), &c) ==
                    cudaSuccess &&
                clusters >= nr)
                small_mode = kSmallPair;
            cudaGetLastError();
        }
        for (int m : {kSmallDual, kSmallSingle}) {
            if (small_mode >= 0 || small_sift_smem(n, m) > room) continue;
            CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per, small_kernel(m), kSmallThreads,
                small_config(m, at, nullptr).dynamicSmemBytes));
            if (per >= 1 && nr <= per * sm_count()) small_mode = m;
        }
        if (small_mode < 0) return CEEMDAN_OK;
        CKS(ws.alloc_n(&sa.arrive, (size_t)std::max(1, max_cap)));
        if (small_mode == kSmallSingle) CKS(ws.alloc_n(&sa.up, (size_t)nr * row_ld(n)));
        // device copy of a taped stage's block table (blocks of kTapeBlockSlots slots)
        CKS(ws.alloc_n(&tblocks_dev, (size_t)(std::max(1, max_cap) + kTapeBlockSlots - 1) /
                                         kTapeBlockSlots));
        // a negative limit -k: the test of the timeout path (the waits of every realization's
        // first CTA give up after k polls, the other CTA's of a pair do not)
        sa.spin_limit = spin_limit > 0 ? spin_limit : (spin_limit < 0 ? -spin_limit : (1 << 22));
        sa.extra = spin_limit < 0 ? 1u : 0u;
        small_cap = std::max(1, max_cap);
        small = true;
        return CEEMDAN_OK;
    }
    int small_cap = 0;
    unsigned char** tblocks_dev = nullptr;

    // One stage on chip (k_sift_small); the realizations that finish in the last iteration
    // export their modes inside the kernel.
    ceemdan_status run_stage_small(double* mode_out, int cap, cudaStream_t st, int* iters_out) {
        sa.tblocks = nullptr;
        if (tape) {  // every slot the stage may fill (the caller trims past the iterations run)
            if (!tape->grow(tape_stage, (long)cap - 1, st)) {
                g_last_error = "out of device memory for the tape";
                return CEEMDAN_ERR_NO_MEMORY;
            }
            const auto& blocks = tape->stages[tape_stage].blocks;
            CK(cudaMemcpyAsync(tblocks_dev, blocks.data(), blocks.size() * sizeof(unsigned char*),
                               cudaMemcpyHostToDevice, st));
            sa.tblocks = tblocks_dev;
            sa.tl = tape->L;
        }
        k_begin_stage<<<1, kThreads, 0, st>>>(a, 0, cap, mode_out);
        ++g_launches;
        CK(cudaMemsetAsync(sa.arrive, 0, sizeof(*sa.arrive) * (size_t)std::min(cap, small_cap),
                           st));
        void* args[] = {(void*)&a, (void*)&sa};
        cudaEvent_t* sev = kernel_ms ? &ev[ev.size() - 2] : nullptr;
        if (sev) CK(cudaEventRecord(sev[0], st));
        cudaLaunchAttribute at[2];
        const cudaLaunchConfig_t cfg = small_config(small_mode, at, st);
        CK(cudaLaunchKernelExC(&cfg, small_kernel(small_mode), args));
        ++g_launches;
        if (sev) CK(cudaEventRecord(sev[1], st));
        CK(cudaMemcpyAsync(hstate, state, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (sev) {
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, sev[0], sev[1]));
            kernel_ms[CEEMDAN_K_SIFT_SMALL] += ms;
        }
        if (hstate[2] != 0) {
            g_last_error = hstate[2] == CEEMDAN_ERR_TIMEOUT
                               ? "the lock-step stop test of the on-chip sift ran out of polls"
                               : "a sift kernel reported an error in the device error word";
            return (ceemdan_status)hstate[2];
        }
        if (iters_out) *iters_out = hstate[1];
        return CEEMDAN_OK;
    }

    // Realizations split over parts: the stop test of every iteration is the AND over the
    // parts (ceemdan_split::all_finished), so the stage runs iteration by iteration with the
    // flag read back after each one.
    const ceemdan_split* split = nullptr;

    ceemdan_status run_stage_split(double* mode_out, int cap, cudaStream_t st, int* iters_out,
                                   volatile int32_t* cancel) {
        k_begin_stage<<<1, kThreads, 0, st>>>(a, 0, cap, mode_out);
        ++g_launches;
        CK(cudaGetLastError());
        for (long j = 0; j < cap; ++j) {
            CKS(launch_iteration(j, st));
            CK(cudaMemcpyAsync(hstate, state, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            harvest_timing(j, 1);
            if (hstate[2] != 0) {
                g_last_error = "a sift kernel reported an error in the device error word";
                return (ceemdan_status)hstate[2];
            }
            const int local = hstate[0] != 0 ? 1 : 0;  // this part's realizations all finished
            const int all = split->all_finished(split->ctx, local);
            if (all < 0) {
                g_last_error = "the split's all_finished exchange failed";
                return CEEMDAN_ERR_CUDA;
            }
            if (all) break;
            // another part still sifts: so do this part's realizations (lock step)
            if (local) CK(cudaMemsetAsync(state, 0, sizeof(int), st));
            if (cancel && *cancel) {
                cudaStreamSynchronize(st);
                g_last_error = "cancelled by the host cancel word";
                return CEEMDAN_ERR_CANCELLED;
            }
        }
        if (iters_out) *iters_out = hstate[1];
        const int bx = std::max(1, std::min((n + kThreads - 1) / kThreads, 64));
        k_export_final<<<dim3(bx, nr), kThreads, 0, st>>>(a, 0);
        ++g_launches;
        CK(cudaGetLastError());
        return CEEMDAN_OK;
    }

    ceemdan_status run_stage(double* mode_out, int cap, cudaStream_t st, int* iters_out,
                             volatile int32_t* cancel) {
        if (split) return run_stage_split(mode_out, cap, st, iters_out, cancel);
        if (small && cap <= small_cap) {
            if (cancel && *cancel) {
                g_last_error = "cancelled by the host cancel word";
                return CEEMDAN_ERR_CANCELLED;
            }
            return run_stage_small(mode_out, cap, st, iters_out);
        }
        k_begin_stage<<<1, kThreads, 0, st>>>(a, 0, cap, mode_out);
        ++g_launches;
        CK(cudaGetLastError());
        long launched = 0;
        int slot = 0;
        long group_first[2] = {0, 0};
        auto launch_group = [&](int sl) -> ceemdan_status {
            group_first[sl] = launched;
            for (int g = 0; g < group; ++g) CKS(launch_iteration(launched++, st));
            CK(cudaMemcpyAsync(hstate + 4 * sl, state, 4 * sizeof(int), cudaMemcpyDeviceToHost,
                               st));
            CK(cudaEventRecord(group_ev[sl], st));
            return CEEMDAN_OK;
        };
        CKS(launch_group(slot));
        for (;;) {
            CKS(launch_group(slot ^ 1));
            CK(cudaEventSynchronize(group_ev[slot]));
            harvest_timing(group_first[slot], group);
            const int* hs = hstate + 4 * slot;
            if (hs[2] != 0) {
                cudaStreamSynchronize(st);
                g_last_error = "a sift kernel reported an error in the device error word";
                return (ceemdan_status)hs[2];
            }
            if (hs[0]) break;
            if (cancel && *cancel) {
                cudaStreamSynchronize(st);
                g_last_error = "cancelled by the host cancel word";
                return CEEMDAN_ERR_CANCELLED;
            }
            slot ^= 1;
        }
        CK(cudaStreamSynchronize(st));
        harvest_timing(group_first[slot ^ 1], group);
        const int iters = hstate[4 * (slot ^ 1) + 1];  // final value (latest copy)
        if (iters_out) *iters_out = iters;
        const int bx = std::max(1, std::min((n + kThreads - 1) / kThreads, 64));
        k_export_final<<<dim3(bx, nr), kThreads, 0, st>>>(a, 0);
        ++g_launches;
        CK(cudaGetLastError());
        return CEEMDAN_OK;
    }
};

}  // namespace ceemdan
