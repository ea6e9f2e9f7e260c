// Launch-configuration tables of the sweep kernels, shared by the FP64 and mixed translation units.
//
// Every model/precision instantiates the same candidate tile shapes.  The tile shape only changes which
// thread computes which cell, never the arithmetic of a cell, so all candidates produce identical results;
// the autotuner (vg_autotune in vg_api.cu) times them on the caller's grid and keeps the fastest.
#pragma once

#include <algorithm>
#include <atomic>

#include <cuda_runtime.h>

#include "vg_common.cuh"

namespace vg {

using SweepFn = cudaError_t (*)(const SweepArgs&, cudaStream_t);

constexpr int kNumXCfg = 5;
constexpr int kNumYCfg = 6;

// X sweep: P cells per segment (P-2 outputs), LPB segments per block, MINB = minimum resident blocks
// per SM requested from the register allocator (1: no register cap).
template <class K, class M, int P, int LPB, int MINB>
cudaError_t launch_x(const SweepArgs& a, cudaStream_t st) {
    dim3 grid((a.nx + P - 3) / (P - 2), (a.ny + LPB - 1) / LPB);
    K::template x<M, P, LPB, MINB>(grid, P * LPB, st, a);
    return cudaGetLastError();
}

// Rows marched per Y-sweep block when segments are sized for the device: the segment length from 2 to 4 TY that minimises
// the time of the grid in units of one warp's share of its pipes for a row.  A scheduler with w resident warps takes
// max(3, w + 0.4) such units for a row of all of them: one or two warps wait for their own chains, and many still do not fill
// the pipes.  A block starts its march with about two rows, every full wave of resident blocks runs at the full w, and the last
// one at what its blocks give each SM.  The rule was fitted to sweeps of every model family at 130 x 97, 512^2, 1024^2 and
// 2048^2 with 2 to 128 rows; its choices are within 1.07 of the best of them, 1.003 on average.  (w alone, with a latency of 1.4
// for the exact form, let a chip three fifths full pass for a full one: 2048^2 Euler multiphysics, blocks of 128 at 96 registers,
// 1.16 ms with its 76 rows against 0.96 with 45, and 1.09 of the best on average.)  130 x 97 Euler: 43 us a sweep with 32 rows,
// 13.8 us with 2; 2048^2 MHD: 0.289 ms with 64 rows, 0.257 ms with 56.  The results do not depend on the segmentation.  The
// autotuner times every shape both ways.
inline int y_segment_rows(int ny, int xblocks, int tx, long slots, int sms, int ty0) {
    if (slots <= 0 || sms <= 0 || ny <= 0) return ty0;
    const double warps = tx / 32.0 / 4.0;  // of one block on each scheduler
    auto row = [](double w) { return std::max(3.0, w + 0.4); };
    const double full = row((double)(slots / sms) * warps);
    int best = ty0;
    double best_cost = 1e300;
    for (int ty = 2; ty <= 4 * ty0; ty++) {
        const long blocks = (long)xblocks * ((ny + ty - 1) / ty);
        const long waves = blocks / slots, rest = blocks % slots;
        double cost = (double)waves * full;
        if (rest) cost += row((double)((rest + sms - 1) / sms) * warps);
        cost *= ty + 2;
        if (cost < best_cost) {
            best_cost = cost;
            best = ty;
        }
        if (ty >= ny) break;
    }
    return best;
}

// Resident blocks of a Y shape on the device and its SMs, looked up on first use (every thread stores the same).
template <class K, class M, int TX, int TY, int MINB>
long y_slots(int& sms) {
    static std::atomic<long> cached{0};
    static std::atomic<int> cached_sms{0};
    long slots = cached.load(std::memory_order_acquire);
    if (slots == 0) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        slots = (long)K::template y_resident<M, TX, TY, MINB>() * n;
        if (slots <= 0) slots = -1;
        cached_sms.store(n, std::memory_order_relaxed);
        cached.store(slots, std::memory_order_release);
    }
    sms = cached_sms.load(std::memory_order_relaxed);
    return slots;
}

// Y sweep: TX columns per block, rows marched per thread from y_segment_rows (TY its centre), MINB as above.  The segments are
// sized for the form of the model that the launch takes: the plain Euler form has 164 registers where the general one has 190.
template <class K, class M, int TX, int TY, int MINB>
cudaError_t launch_y(const SweepArgs& a0, cudaStream_t st) {
    if constexpr (!M::HAS_Y) {
        return cudaErrorInvalidValue;
    } else {
        if (a0.nx <= 0) {  // a call that only looks the occupancy up (before a graph capture)
            K::template each_form<M>([](auto m) {
                int sms;
                y_slots<K, decltype(m), TX, TY, MINB>(sms);
            });
            return cudaSuccess;
        }
        K::template form<M>(a0, [&](auto m) {
            using F = decltype(m);
            SweepArgs a = a0;
            const int xblocks = (a.nx + TX - 1) / TX;
            int sms;
            const long slots = y_slots<K, F, TX, TY, MINB>(sms);
            a.ty_rows = a.y_waves ? y_segment_rows(a.ny, xblocks, TX, slots, sms, TY) : TY;
            dim3 grid(xblocks, (a.ny + a.ty_rows - 1) / a.ty_rows);
            K::template y<F, TX, TY, MINB>(grid, TX, st, a);
        });
        return cudaGetLastError();
    }
}

// X sweep staged by TMA (persistent, two rows per thread; see slic_tma.cuh) when the solver holds a tensor map over
// a.in, else the plain two-row kernel of the same shape.
template <class K, class M, int P, int MINB>
cudaError_t launch_x_tma(const SweepArgs& a, cudaStream_t st) {
    static_assert(P == kTmaTile, "the solver's tensor maps have a box of kTmaTile + 2 cells");
    if (!a.tmap) return launch_x<K, M, P, 1, MINB>(a, st);
    K::template x_tma<M, P, MINB>(st, a);
    return cudaGetLastError();
}

template <class M, class = void>
struct pair_sweeps {
    static constexpr bool value = false;
};
template <class M>
struct pair_sweeps<M, decltype((void)M::PAIR_X)> {
    static constexpr bool value = M::PAIR_X;
};

// The exact-form models with shared reciprocals (exact_div.cuh) have long independent chains that the compiler would overlap
// with every register it can get; their own tables cap the registers where more resident warps pay more (kinds 5 and 6,
// index 0 the default).  The caps of kinds 7 and 8, kind 6 of longer states, differ in those shapes alone.
template <class M, class = void>
struct shared_sweeps {
    static constexpr bool value = false;
};
template <class M>
struct shared_sweeps<M, decltype((void)M::SHARED_DIV)> {
    static constexpr bool value = M::SHARED_DIV;
};

// Models with more than 9 conserved components (HPR, 17) use shorter X segments so that the three FP64
// shared-memory tiles stay inside the 48 KB static limit (kind 1); models with more than 21 (the HPR multiphysics
// model, 33) shorter still (kind 4).  The PAIR_X models (two rows per thread in the X sweep) add the TMA-staged X
// shapes for the Euler states of up to four planes (kind 2); other PAIR_X models (MHD) keep the plain two-row shapes
// (kind 3).
template <class M>
constexpr int tile_kind() {
    return (M::NU > 21) ? 4 : (M::NU > 9) ? (shared_sweeps<M>::value ? 5 : 1) : pair_sweeps<M>::value ? (M::NW <= 4 ? 2 : 3)
           : shared_sweeps<M>::value ? (M::NU <= 4 ? 6 : M::NU <= 7 ? 7 : 8) : 0;
}

// Revision of the tables below, part of the key of saved tunings: raise it where an index comes to name another shape.
constexpr int kSweepTables = 2;

template <class K, class M, int KIND = tile_kind<M>()>
struct SweepTable;

template <class K, class M>
struct SweepTable<K, M, 1> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 64, 1, 1>, launch_x<K, M, 32, 2, 1>, launch_x<K, M, 96, 1, 1>,
        launch_x<K, M, 64, 1, 2>, launch_x<K, M, 32, 1, 1>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 32, 32, 1>,
        launch_y<K, M, 32, 64, 1>, launch_y<K, M, 128, 32, 1>, launch_y<K, M, 64, 16, 1>,
    };
};

template <class K, class M>
struct SweepTable<K, M, 4> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 32, 1, 1>, launch_x<K, M, 40, 1, 1>, launch_x<K, M, 48, 1, 1>,
        launch_x<K, M, 56, 1, 1>, launch_x<K, M, 32, 1, 2>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 32, 32, 1>,
        launch_y<K, M, 32, 64, 1>, launch_y<K, M, 128, 32, 1>, launch_y<K, M, 64, 16, 1>,
    };
};

template <class K, class M>
struct SweepTable<K, M, 0> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 128, 1, 1>, launch_x<K, M, 64, 2, 1>, launch_x<K, M, 192, 1, 1>,
        launch_x<K, M, 128, 1, 6>, launch_x<K, M, 128, 1, 8>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 64, 64, 12>,
        launch_y<K, M, 64, 64, 16>, launch_y<K, M, 128, 32, 5>, launch_y<K, M, 32, 64, 1>,
    };
};

template <class K, class M>
struct SweepTable<K, M, 2> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 128, 1, 1>, launch_x_tma<K, M, 128, 7>, launch_x_tma<K, M, 128, 8>,
        launch_x<K, M, 128, 1, 6>, launch_x<K, M, 128, 1, 8>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 64, 64, 12>,
        launch_y<K, M, 64, 64, 16>, launch_y<K, M, 128, 32, 5>, launch_y<K, M, 32, 64, 1>,
    };
};

template <class K, class M>
struct SweepTable<K, M, 3> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 128, 1, 1>, launch_x<K, M, 64, 2, 1>, launch_x<K, M, 128, 1, 4>,
        launch_x<K, M, 128, 1, 6>, launch_x<K, M, 128, 1, 8>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 64, 64, 12>,
        launch_y<K, M, 64, 64, 16>, launch_y<K, M, 128, 32, 5>, launch_y<K, M, 32, 64, 1>,
    };
};

// X, measured in ms a sweep (4096^2 Euler | 2048^2 MHD7 | 2048^2 two-material Euler | 2048^2 MHD9): 7 blocks of 128 (72
// registers) 0.648 | 0.266 | 0.335 | -, 5 (96) 0.689 | 0.264 | 0.332 | 0.403, 4 (128) 0.730 | 0.271 | 0.337 | 0.339, no cap 0.73 |
// 0.38 | 0.45 | 0.36.  Y: 8 blocks of 64 (128 registers) 0.606 for Euler against 0.616 without a cap; the longer states lose
// more to spills than the warps give (MHD7 0.291 against 0.253, two-material Euler 0.358 against 0.344).
template <class K, class M, int XB, int YB>
struct SharedSweepTable {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 128, 1, XB>, launch_x<K, M, 64, 1, 9>, launch_x<K, M, 96, 1, 8>,
        launch_x<K, M, 128, 1, 5>, launch_x<K, M, 128, 1, 8>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, YB>, launch_y<K, M, 64, 32, 5>, launch_y<K, M, 64, 64, 12>,
        launch_y<K, M, 64, 64, 10>, launch_y<K, M, 128, 32, 1>, launch_y<K, M, 32, 64, YB>,
    };
};

template <class K, class M>
struct SweepTable<K, M, 6> : SharedSweepTable<K, M, 7, 8> {};
template <class K, class M>
struct SweepTable<K, M, 7> : SharedSweepTable<K, M, 7, 1> {};
template <class K, class M>
struct SweepTable<K, M, 8> : SharedSweepTable<K, M, 4, 1> {};

// X (1001x777 two-material MHD | 1024^2 HPR): 4 blocks of 96 (168 registers) 0.118 | 0.271, 5 of 64 (168) 0.119 | 0.291, no cap
// 0.135 | 0.288.
template <class K, class M>
struct SweepTable<K, M, 5> {
    static constexpr SweepFn x[kNumXCfg] = {
        launch_x<K, M, 96, 1, 4>, launch_x<K, M, 64, 1, 5>, launch_x<K, M, 64, 1, 1>,
        launch_x<K, M, 32, 2, 5>, launch_x<K, M, 32, 1, 1>,
    };
    static constexpr SweepFn y[kNumYCfg] = {
        launch_y<K, M, 64, 64, 1>, launch_y<K, M, 64, 32, 1>, launch_y<K, M, 32, 32, 1>,
        launch_y<K, M, 32, 64, 1>, launch_y<K, M, 128, 32, 1>, launch_y<K, M, 64, 16, 5>,
    };
};

// Names of the shapes of SweepTable<K, M, kind>.
inline const char* x_cfg_name(int i, int kind = 0) {
    static const char* const n[][kNumXCfg] = {
        {"P128xL1", "P64xL2", "P192xL1", "P128xL1/min6", "P128xL1/min8"},
        {"P64xL1", "P32xL2", "P96xL1", "P64xL1/min2", "P32xL1"},
        {"P128x2", "TMA P128x2/min7", "TMA P128x2/min8", "P128x2/min6", "P128x2/min8"},
        {"P128x2", "P64xL2x2", "P128x2/min4", "P128x2/min6", "P128x2/min8"},
        {"P32xL1", "P40xL1", "P48xL1", "P56xL1", "P32xL1/min2"},
        {"P96xL1/min4", "P64xL1/min5", "P64xL1", "P32xL2/min5", "P32xL1"},
        {"P128xL1/min7", "P64xL1/min9", "P96xL1/min8", "P128xL1/min5", "P128xL1/min8"},
        {"P128xL1/min7", "P64xL1/min9", "P96xL1/min8", "P128xL1/min5", "P128xL1/min8"},
        {"P128xL1/min4", "P64xL1/min9", "P96xL1/min8", "P128xL1/min5", "P128xL1/min8"},
    };
    return i >= 0 && i < kNumXCfg && kind >= 0 && kind < 9 ? n[kind][i] : "?";
}
inline const char* y_cfg_name(int i, int kind = 0) {
    static const char* const n[][kNumYCfg] = {
        {"TX64xTY64", "TX64xTY32", "TX64xTY64/min12", "TX64xTY64/min16", "TX128xTY32/min5", "TX32xTY64"},
        {"TX64xTY64", "TX64xTY32", "TX32xTY32", "TX32xTY64", "TX128xTY32", "TX64xTY16"},
        {"TX64xTY64", "TX64xTY32", "TX64xTY64/min12", "TX64xTY64/min16", "TX128xTY32/min5", "TX32xTY64"},
        {"TX64xTY64", "TX64xTY32", "TX64xTY64/min12", "TX64xTY64/min16", "TX128xTY32/min5", "TX32xTY64"},
        {"TX64xTY64", "TX64xTY32", "TX32xTY32", "TX32xTY64", "TX128xTY32", "TX64xTY16"},
        {"TX64xTY64", "TX64xTY32", "TX32xTY32", "TX32xTY64", "TX128xTY32", "TX64xTY16/min5"},
        {"TX64xTY64/min8", "TX64xTY32/min5", "TX64xTY64/min12", "TX64xTY64/min10", "TX128xTY32", "TX32xTY64/min8"},
        {"TX64xTY64", "TX64xTY32/min5", "TX64xTY64/min12", "TX64xTY64/min10", "TX128xTY32", "TX32xTY64"},
        {"TX64xTY64", "TX64xTY32/min5", "TX64xTY64/min12", "TX64xTY64/min10", "TX128xTY32", "TX32xTY64"},
    };
    return i >= 0 && i < kNumYCfg && kind >= 0 && kind < 9 ? n[kind][i] : "?";
}

}  // namespace vg
