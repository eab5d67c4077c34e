// tiles.cu — plans and launches of the multi-step tile kernels (tiles.cuh).
#include <algorithm>
#include <type_traits>

#include "internal.h"
#include "tiles.cuh"

namespace lbm {

// The shapes.  Region rows start on 16-byte words, so the halo is 4 columns for FP32 and FP64 and 8 for
// 16-bit words.  Small: tiles of 16 columns, up to 8 steps; mid: 64 columns, up to 4 steps, one region;
// stream: mid with two regions and four moving warps.
template <class S>
constexpr int kMidHalo = sizeof(S) == 2 ? 8 : 4;
template <class S>
using SmallShape = TileShape<S, 32, 32, 24, 8, 12, 0>;
template <class S>
using MidShape = TileShape<S, 64 + 2 * kMidHalo<S>, 72, sizeof(S) == 8 ? 40 : 44, kMidHalo<S>, sizeof(S) == 8 ? 16 : 24, 0>;
template <class S>
using StreamShape = TileShape<S, 64 + 2 * kMidHalo<S>, 72, 42, kMidHalo<S>, 20, 4>;

template <class S, bool ABS, class Sh, int G>
static cudaError_t launch_one(const StepParams<typename Codec<S>::Real>& p, const TileLaunch& l, const TilePlan& plan, int T,
                              cudaStream_t s) {
    static_assert(Sh::smem_bytes() <= 227 * 1024, "a tile's regions must fit into shared memory");
    // what the kernel's indices rely on
    const bool fits = T >= 2 && T % 2 == 0 && T <= Sh::kMaxSteps && T <= Sh::HALO && plan.h >= 2 && plan.h % 2 == 0 &&
                      plan.h + 2 * T <= Sh::MAXR && p.nx >= Sh::PX && p.ny >= plan.h + 2 * T &&
                      ((size_t)p.nx * sizeof(S)) % G == 0 && 9ULL * (unsigned long long)p.N <= (1ULL << 32);
    if (!fits) return cudaErrorInvalidValue;
    auto kern = k_step_tiles<S, ABS, Sh, G>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::smem_bytes());
    if (e != cudaSuccess) return e;
    const int tx = (p.nx + Sh::W - 1) / Sh::W, ty = (p.ny + plan.h - 1) / plan.h;
    ClassMarks marks{};
    for (int k = 0; k < kMaxClasses; ++k) {
        const uint32_t fl = p.cls.flags[k];
        marks.flags |= (fl ? 1u : 0u) << k;
        marks.outlet |= (fl & kZeroGradXp ? 1u : 0u) << k;
        marks.zouhe |= (fl & (kZouHeVelXm | kZouHeRhoXp) ? 1u : 0u) << k;
    }
    // a launch may be scheduled while the one before it drains (the kernel waits for its end itself)
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)std::min(tx * ty, l.sms));
    cfg.blockDim = dim3(Sh::BLOCK);
    cfg.dynamicSmemBytes = Sh::smem_bytes();
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, p, plan.h, T, tx, tx * ty, marks, -0.0f, l.err);
}

template <class S, bool ABS>
static cudaError_t launch_kind(const StepParams<typename Codec<S>::Real>& p, const TileLaunch& l, const TilePlan& plan, int T,
                               cudaStream_t s) {
    constexpr int kWord = (int)sizeof(S);
    const size_t row = (size_t)p.nx * kWord;
    // the largest pieces that every row starts on
    auto by_piece = [&](auto sh) {
        using Sh = decltype(sh);
        if constexpr (kWord == 2 || (kWord == 4 && !ABS)) {
            if (row % 16 == 0) return launch_one<S, ABS, Sh, 16>(p, l, plan, T, s);
        }
        if constexpr (kWord == 2) {
            if (row % 4 == 0) return launch_one<S, ABS, Sh, 4>(p, l, plan, T, s);
        }
        return launch_one<S, ABS, Sh, kWord>(p, l, plan, T, s);
    };
    if (plan.kind == kTilesSmall) return by_piece(SmallShape<S>{});
    if constexpr (kWord == 4 && !ABS) {
        if (plan.kind == kTilesStream && row % 16 == 0) return launch_one<S, ABS, StreamShape<S>, 16>(p, l, plan, T, s);
    }
    return by_piece(MidShape<S>{});
}

cudaError_t launch_tiles(const lbm_desc& d, const TileLaunch& l, const TilePlan& plan, int T, cudaStream_t s) {
    const bool abs_arith = d.arithmetic == LBM_ARITH_ABSOLUTE;
    switch (d.storage) {
        case LBM_F32:
            return abs_arith ? launch_kind<float, true>(l.pf, l, plan, T, s) : launch_kind<float, false>(l.pf, l, plan, T, s);
        case LBM_F16S: return launch_kind<__half, false>(l.pf, l, plan, T, s);
        case LBM_BF16S: return launch_kind<__nv_bfloat16, false>(l.pf, l, plan, T, s);
        default:
            return abs_arith ? launch_kind<double, true>(l.pd, l, plan, T, s) : launch_kind<double, false>(l.pd, l, plan, T, s);
    }
}

// When tiles are faster than single steps (measured on B200, lid cavities, us per step, single -> tiles).
// - Lattices that one wave of CTAs covers: a launch of T steps then costs about 2 us of launch and drain, 2 us of
//   moves and T short steps.  Small tiles first, for more CTAs: 96^2 FP32 1.4 -> 0.9, 128^2 1.8 -> 1.0, 192^2
//   (16-row tiles, 4 steps) 3.5 -> 1.5; then 64-column tiles: 256^2 4.7 -> 1.8, 512^2 4.6 -> 3.5, 1000 x 300 5.0 ->
//   3.7 (FP16S 512^2 6.2 -> 4.0, 1000 x 300 5.0 -> 4.3).  FP64 collisions take twice as long, so only up to
//   14 rows: 256^2 4.1 -> 2.7, 384^2 (16 rows) 4.3 -> 4.2, 512^2 5.3 -> 6.3.
// - Two or three waves: nothing to gain (1024 x 512 FP32 6.6 -> 6.4, FP16S 7.4 -> 7.2; 1024^2 11.2 -> 11.9).
// - FP32 lattices whose two buffers leave L2: streamed tiles, from about 80 MB (75 MB 11.2 -> 11.9, 86 MB 13.6 ->
//   11.8, 118 MB 18.8 -> 16.7, 302 MB 49 -> 35); rows that do not start on 16-byte words cannot be moved in bulk
//   and take the mid shape, from 125 MB (118 MB 18.8 -> 19.6, 122 MB 22.7 -> 20.0, 3001 x 2003 75.6 -> 68.6).
//   16-bit words cross HBM fast enough in single steps (2048^2 FP16S 39.6 -> 46.6), FP64 gains 4 % at most.
TilePlan plan_tiles(const lbm_desc& d, int sms) {
    const bool abs_arith = d.arithmetic == LBM_ARITH_ABSOLUTE;
    const int word = storage_bytes(d.storage);
    // the smallest even height (at most `most`) at which tiles of w columns are no more than the SMs, or 0
    auto one_wave = [&](int w, int most) {
        const long long tx = (d.nx + w - 1) / w;
        for (int h = 2; h <= most; h += 2)
            if (tx * ((d.ny + h - 1) / h) <= sms) return h;
        return 0;
    };
    auto plan = [&](TileKind k, int px, int h, int steps) {
        TilePlan t{};
        if (h > 0 && d.nx >= px && d.ny >= h + 2 * steps) t = TilePlan{k, h, steps};
        return t;
    };
    const int mid_px = 64 + 2 * (word == 2 ? 8 : 4);
    if (const int h = one_wave(16, 8)) return plan(kTilesSmall, 32, h, 8);
    if (const int h = one_wave(16, 16)) return plan(kTilesSmall, 32, h, 4);
    if (const int h = one_wave(64, word == 8 ? 14 : 36)) return plan(kTilesMid, mid_px, h, 4);
    const long long bytes = 2LL * 9 * word * d.nx * d.ny;  // both buffers
    if (word == 4 && !abs_arith) {
        if (d.nx % 4 == 0 && bytes > 80000000LL) return plan(kTilesStream, mid_px, 34, 4);
        if (bytes > 125000000LL) return plan(kTilesMid, mid_px, 34, 4);
    }
    return TilePlan{};
}

}  // namespace lbm
