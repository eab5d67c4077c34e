// tiles.cu — plans and launches of the multi-step tile kernels (tiles.cuh).
#include <algorithm>
#include <type_traits>

#include "internal.h"
#include "tiles.cuh"

namespace lbm {

// The shapes.  Region rows start on 16-byte words, so the halo is 4 columns for FP32 and FP64 and 8 for
// 16-bit words.  Small: tiles of 16 columns, up to 8 steps; mid: 64 columns, up to 4 steps, one region; pieces,
// stream: mid with two regions and four moving warps.  Bulk copies do not occupy the load/store units while HBM
// answers, but take some 20 issue slots each: they win where the populations stream from HBM (4096^2 FP32 113 us a
// step against 126 in pieces, 2048 x 1024 19.2 against 20.5), pieces where they stay in L2 (1024^2 10.6 against
// 11.2) and for Shan-Chen's two steps a launch (1024^2 15.1 against 17.5).
// Mid: 16 warps, whose pairs a step make three full turns with 113 registers a thread (24 warps with 80: two turns, and
// slower: FP16S 1000 x 300 4.28 -> 4.03, FP32 256^2 1.74 -> 1.61, 1024 x 256 cavity 3.38 -> 3.27).  ptxas spills 116 bytes of
// the FP64 mid shape, 72 of the FP64 stream, 32 of the FP32 streams (80 registers with 24 warps).
template <class S>
constexpr int kMidHalo = sizeof(S) == 2 ? 8 : 4;
template <class S>
using SmallShape = TileShape<S, false, 32, 32, 24, 8, 12, 0, false>;
template <class S>
using MidShape = TileShape<S, false, 64 + 2 * kMidHalo<S>, 72, sizeof(S) == 8 ? 40 : 44, kMidHalo<S>, 16, 0, false>;
template <class S, bool BULK>
using StreamShape =
    TileShape<S, false, 64 + 2 * kMidHalo<S>, 72, sizeof(S) == 8 ? 20 : 42, kMidHalo<S>, sizeof(S) == 8 ? 12 : 20, 4, BULK>;
template <class S>
using ShanChenShape = TileShape<S, true, 64 + 2 * kMidHalo<S>, 72, sizeof(S) == 2 ? 44 : 40, kMidHalo<S>, 20, 4, false>;

template <class S, bool ABS, class Sh, int G>
static cudaError_t launch_one(const StepParams<typename Codec<S>::Real>& p, const TileLaunch& l, const TilePlan& plan, int steps,
                              cudaStream_t s) {
    static_assert(Sh::smem_bytes() <= 227 * 1024, "a tile's regions must fit into shared memory");
    // what the kernel's indices rely on
    const int T = std::min(steps, plan.steps), total = steps;
    const bool fits = T >= 2 && T % 2 == 0 && T <= Sh::kMaxSteps && plan.h >= 2 && plan.h % 2 == 0 &&
                      plan.h + 2 * Sh::D * T <= Sh::MAXR && p.nx >= Sh::PX && p.ny >= plan.h + 2 * Sh::D * T &&
                      ((size_t)p.nx * sizeof(S)) % G == 0 && 9ULL * (unsigned long long)p.N <= (1ULL << 32);
    if (!fits || total % 2) return cudaErrorInvalidValue;
    auto kern = k_step_tiles<S, ABS, Sh, G>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::smem_bytes());
    if (e != cudaSuccess) return e;
    const int tx = (p.nx + Sh::W - 1) / Sh::W, ty = (p.ny + plan.h - 1) / plan.h;
    const bool rounds = total > T;
    // without moving warps a CTA has one tile; in rounds, every CTA waits for others
    if (Sh::MOVERS ? rounds : tx * ty > l.sms) return cudaErrorInvalidValue;
    if (rounds) {
        const int depth = Sh::D * T, side = std::max(0, plan.h - 2 * depth);
        const int ring = std::min(plan.h, 2 * depth) * Sh::W + side * std::min(Sh::W, 2 * depth);
        const size_t bytes = 2 * sizeof(uint4) * (size_t)(tx * ty) * Sh::kRecords * (size_t)l.ex.cap;
        if (!l.ex.records || !l.ex.rounds || ring > l.ex.cap || bytes > l.ex.bytes || ring > Sh::kMostRing ||
            2 * depth * (Sh::W + 2 * depth) + plan.h * 2 * depth > Sh::kMostHalo)
            return cudaErrorInvalidValue;
    }
    ClassMarks marks{};
    for (int k = 0; k < kMaxClasses; ++k) {
        const uint32_t fl = p.cls.flags[k];
        marks.flags |= (fl ? 1u : 0u) << k;
        marks.outlet |= (fl & kZeroGradXp ? 1u : 0u) << k;
        marks.zouhe |= (fl & (kZouHeVelXm | kZouHeRhoXp) ? 1u : 0u) << k;
    }
    if (Sh::SC && marks.outlet) return cudaErrorInvalidValue;  // no zero-gradient cells in Shan-Chen tiles
    // a launch may be scheduled while the one before it drains (the kernel waits for its end itself); one in rounds
    // starts with all its CTAs or not at all
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    if (rounds) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.gridDim = dim3((unsigned)std::min(tx * ty, l.sms));
    cfg.blockDim = dim3(Sh::BLOCK);
    cfg.dynamicSmemBytes = Sh::smem_bytes();
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, p, plan.h, T, total, tx, tx * ty, marks, -0.0f, l.ex, l.err);
}

template <class S, bool ABS>
static cudaError_t launch_kind(const StepParams<typename Codec<S>::Real>& p, const TileLaunch& l, const TilePlan& plan, int steps,
                               cudaStream_t s) {
    constexpr int kWord = (int)sizeof(S);
    const size_t row = (size_t)p.nx * kWord;
    // the largest pieces that every row starts on
    auto by_piece = [&](auto sh) {
        using Sh = decltype(sh);
        if constexpr (kWord == 2 || !ABS) {
            if (row % 16 == 0) return launch_one<S, ABS, Sh, 16>(p, l, plan, steps, s);
        }
        if constexpr (kWord == 2) {
            if (row % 4 == 0) return launch_one<S, ABS, Sh, 4>(p, l, plan, steps, s);
        }
        return launch_one<S, ABS, Sh, kWord>(p, l, plan, steps, s);
    };
    if constexpr (kWord <= 4 && !ABS) {
        if (plan.kind == kTilesShanChen) {
            if constexpr (kWord == 4) return by_piece(ShanChenShape<S>{});
            // (16-bit words: plan_tiles asks for whole 16-byte words)
            return row % 16 == 0 ? launch_one<S, ABS, ShanChenShape<S>, 16>(p, l, plan, steps, s) : cudaErrorInvalidValue;
        }
    }
    if constexpr (kWord >= 4 && !ABS) {
        if (plan.kind == kTilesStream && row % 16 == 0) return launch_one<S, ABS, StreamShape<S, true>, 16>(p, l, plan, steps, s);
    }
    if constexpr (kWord == 4 && !ABS) {
        if (plan.kind == kTilesPieces) return by_piece(StreamShape<S, false>{});
    }
    if (plan.kind == kTilesSmall) return by_piece(SmallShape<S>{});
    if (plan.kind == kTilesMid) return by_piece(MidShape<S>{});
    return cudaErrorInvalidValue;
}

int tile_launch_steps(const TilePlan& plan) {
    return plan.kind == kTilesSmall || plan.kind == kTilesMid ? 4096 : plan.steps;
}

TileExchange tile_exchange(const lbm_desc& d, const TilePlan& plan) {
    TileExchange e;
    if (plan.kind != kTilesSmall && plan.kind != kTilesMid) return e;
    const int word = storage_bytes(d.storage), w = plan.kind == kTilesSmall ? 16 : 64;
    const int depth = plan.steps;
    const int tiles = ((d.nx + w - 1) / w) * ((d.ny + plan.h - 1) / plan.h);
    e.cap = std::min(plan.h, 2 * depth) * w + std::max(0, plan.h - 2 * depth) * std::min(w, 2 * depth);
    e.bytes = 2 * sizeof(uint4) * (size_t)tiles * (size_t)((9 * word + 11) / 12) * (size_t)e.cap;
    return e;
}

cudaError_t launch_tiles(const lbm_desc& d, const TileLaunch& l, const TilePlan& plan, int steps, cudaStream_t s) {
    const bool abs_arith = d.arithmetic == LBM_ARITH_ABSOLUTE;
    switch (d.storage) {
        case LBM_F32:
            return abs_arith ? launch_kind<float, true>(l.pf, l, plan, steps, s) : launch_kind<float, false>(l.pf, l, plan, steps, s);
        case LBM_F16S: return launch_kind<__half, false>(l.pf, l, plan, steps, s);
        case LBM_BF16S: return launch_kind<__nv_bfloat16, false>(l.pf, l, plan, steps, s);
        default:
            return abs_arith ? launch_kind<double, true>(l.pd, l, plan, steps, s) : launch_kind<double, false>(l.pd, l, plan, steps, s);
    }
}

// When tiles are faster than single steps (measured on B200, lid cavities, us per step, single -> tiles).
// - BGK lattices that one wave of CTAs covers, in rounds of T steps: about 2 us a round for the exchange and T short
//   steps.  Small tiles first, for more CTAs: 96^2 FP32 1.4 -> 0.7, 128^2 1.8 -> 0.8, 192^2 (16-row tiles, 4 steps)
//   2.5 -> 1.1; then 64-column tiles: 256^2 2.9 -> 1.3, 512^2 4.6 -> 2.6, 1000 x 300 4.3 -> 2.8; FP16S 192^2 2.7 -> 1.2,
//   512^2 5.2 -> 3.3, 1000 x 300 5.0 -> 3.5; FP64 256^2 3.3 -> 2.2, 384^2 4.0 -> 3.35, 640 x 400 (30 rows) 5.1 -> 4.6.
// - FP32 BGK in L2, several waves: a wave of h-row tiles takes 2.3 (h + 6) / 36 us, a launch 1.4, a single step 1.5
//   and its cells at 107 G/s, which decides (1024 x 512 6.3 -> 5.6, 1024^2 11.2 -> 9.0; 1500 x 451 7.6 -> 7.0).
//   16-bit words gain nothing there (1024 x 512 FP16S 7.4 -> 7.2, 1024^2 11.4 -> 13.3).
// - BGK lattices whose two buffers leave L2: FP32 from about 80 MB (75 MB 11.2 -> 11.9, 86 MB 13.6 -> 11.8, 151 MB
//   26.3 -> 19.2, 433 MB 70 -> 45; rows that start anywhere move in pieces, from 125 MB: 433 MB 78 -> 52), FP64 with
//   rows of whole 16-byte words from 140 MB (151 MB 24.0 -> 22.4, 302 MB 47 -> 39, 865 MB 132 -> 104; in pieces 134 ->
//   137).  16-bit words cross HBM fast enough in single steps (2048^2 FP16S 39.6 -> 46.6).
// - Shan-Chen, FP32 of any width and 16-bit words in rows of whole 16-byte words (in 2-byte pieces 2049 x 1537
//   60.8 -> 73): FP32 256^2 8.3 -> 3.9, 1024^2 21.4 -> 15.1, 2049 x 1537 64 -> 54, 4096^2 298 -> 211; BF16S 8.2 -> 4.0,
//   22.4 -> 15.8, 4096^2 291 -> 230.  A wave takes about h + 4 rows' time, so the height is the one whose waves times
//   that is least (1024^2: 28 rows, 4.0 waves, 15.1; 32 rows, 3.5 waves, 17.0).
TilePlan plan_tiles(const lbm_desc& d, int sms) {
    const bool abs_arith = d.arithmetic == LBM_ARITH_ABSOLUTE;
    const int word = storage_bytes(d.storage);
    const bool whole = d.nx * word % 16 == 0;  // rows of whole 16-byte words
    const int mid_px = 64 + 2 * (word == 2 ? 8 : 4);
    auto tiles = [&](int w, int h) { return ((d.nx + w - 1) / w) * ((d.ny + h - 1) / h); };
    auto waves = [&](int h) { return (tiles(64, h) + sms - 1) / sms; };
    // the smallest even height (at most `most`) at which tiles of w columns are no more than the SMs, or 0
    auto one_wave = [&](int w, int most) {
        for (int h = 2; h <= most; h += 2)
            if (tiles(w, h) <= sms) return h;
        return 0;
    };
    // the height with the shortest waves in all, a wave taking as long as h + over rows
    auto best_height = [&](int most, int over) {
        int best = 2;
        for (int h = 4; h <= most; h += 2)
            if (waves(h) * (h + over) < waves(best) * (best + over)) best = h;
        return best;
    };
    auto plan = [&](TileKind k, int px, int h, int steps, int depth) {
        return d.nx >= px && d.ny >= h + 2 * depth ? TilePlan{k, h, steps} : TilePlan{};
    };
    if (d.collision == LBM_SHANCHEN) {
        bool outlet = false;
        for (int k = 0; k < d.n_classes; ++k) outlet = outlet || (d.classes[k].flags & LBM_CELL_ZEROGRAD_XP);
        if (abs_arith || word == 8 || outlet || (word == 2 && !whole)) return TilePlan{};
        return plan(kTilesShanChen, mid_px, best_height(word == 2 ? 36 : 32, 4), 2, 4);
    }
    if (const int h = one_wave(16, 8)) return plan(kTilesSmall, 32, h, 8, 8);
    if (const int h = one_wave(16, 16)) return plan(kTilesSmall, 32, h, 4, 4);
    if (const int h = one_wave(64, word == 8 ? 32 : 36)) return plan(kTilesMid, mid_px, h, 4, 4);
    if (abs_arith) return TilePlan{};
    const long long bytes = 2LL * 9 * word * d.nx * d.ny;  // both buffers
    if (word == 4 && whole && bytes > 80000000LL) return plan(kTilesStream, mid_px, 34, 4, 4);
    if (word == 4 && !whole && bytes > 125000000LL) return plan(kTilesPieces, mid_px, 34, 4, 4);
    if (word == 4 && whole) {
        const int h = best_height(34, 6);
        const double tiled = 1.4 + 2.3 / 36 * (double)(waves(h) * (h + 6)), single = 1.5 + (double)(d.nx * d.ny) / 107e3;
        if (tiled < 0.97 * single) return plan(kTilesPieces, mid_px, h, 4, 4);
    }
    if (word == 8 && whole && bytes > 140000000LL) return plan(kTilesStream, mid_px, 12, 4, 4);
    return TilePlan{};
}

// Counts the floats of bit patterns [first, first + count), and their negatives, whose packed reciprocal is not 1 / a.
__global__ void k_test_reciprocal(uint32_t first, uint64_t count, float one, unsigned long long* differ) {
    unsigned long long n = 0;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x) {
        const float a = __uint_as_float(first + (uint32_t)k);
        float lo, hi;
        unpack2(reciprocal(pack2(a, -a), pack2(-a, a)), lo, hi);
        n += (__float_as_uint(lo) != __float_as_uint(one / a)) + (__float_as_uint(hi) != __float_as_uint(one / -a));
    }
    if (n) atomicAdd(differ, n);
}

}  // namespace lbm

extern "C" int lbm_test_reciprocal(uint32_t first, int64_t count, int64_t* differ) {
    using namespace lbm;
    if (!differ) return set_error(LBM_ERR_INVALID, "NULL argument");
    if (count < 0 || count > (1LL << 32) - (int64_t)first) return set_error(LBM_ERR_INVALID, "bit patterns beyond 2^32");
    unsigned long long* n = nullptr;
    unsigned long long got = 0;
    LBM_CK(cudaMalloc(&n, sizeof(*n)));
    cudaError_t e = cudaMemset(n, 0, sizeof(*n));
    if (e == cudaSuccess) {
        k_test_reciprocal<<<1184, 256>>>(first, (uint64_t)count, 1.0f, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&got, n, sizeof(got), cudaMemcpyDeviceToHost);
    cudaFree(n);
    LBM_CK(e);
    *differ = (int64_t)got;
    return LBM_OK;
}
