// tiles.cuh — several time steps of a D2Q9 BGK lattice per launch, on overlapped tiles in shared memory.
//
// A step of the one-step kernels reads and writes every population in HBM (or L2) and ends in a launch
// boundary: large FP32 lattices are bound by HBM, small ones by the launch and its drain.  Here a CTA
// advances a tile of W x h cells by T steps: it brings the tile and a halo of T cells into shared memory
// once, collides T times on a region that shrinks by one cell per side and step, and stores the tile.
// Populations cross HBM once per T steps instead of T times, for the redundant collisions in the halo
// (1.2 per cell with 64 x 34 tiles and 4 steps).
//
// One copy of the populations is enough (the A-A pattern, Bailey et al. 2009).  A cell's populations lie at
// its own index or, after every other step, at its neighbours': a step reads and writes the same nine words,
// which no other cell touches in that step, so it needs no second buffer and one barrier.
//   odd steps   read (x - c_i, i) = f_i's source,              write (x + c_i, opp(i)) <- f_i
//   even steps  read (x, opp(i)) = what an odd step left,      write (x, i)            <- f_i
//
// Cells of the region are indexed flat, k = ly PX + lx, and a step walks whole rows: the outermost valid
// cells give way to invalid ones by one cell per side and step, whatever those hold, so no column bounds are
// tested in the loop.  A direction's words are contiguous and its place is a compile-time constant, so every
// access is one register plus an immediate.
//
// The collision of two cells at a time in packed FP32 (add/mul/fma.f32x2) is what bounds the kernel: a packed
// instruction does two cells' work in one issue slot and two cycles of the FP32 pipe.  A pair takes 109
// packed instructions, 24-36 shared-memory accesses and some 20 others; a step of a 64 x 34 tile takes 3000 to
// 3700 cycles where the FP32 pipe alone needs 2350 (scalar arithmetic: 209 instructions per cell, 110 GLUPS at
// 4096^2 without walls against 146).  The moves: 16-byte cp.async (.cg: past the small L1 that 227 KB of shared memory leave;
// .ca took 710 us per 4 steps at 4096^2 against 540) while the lattice has one tile per SM; where SMs take
// many tiles, four warps of their own move whole rows by bulk copies beside the computing ones (one warp
// issues a bulk copy every 58 cycles, four keep up).
//
// Rounds.  Where one wave of CTAs covers the lattice, tiles stay in their CTAs for a whole run (a cooperative launch:
// all CTAs are resident).  After T steps a CTA gives the cells within T of its tile's edges to its neighbours and
// takes its own halo from them, instead of ending the launch (2 us of drain and launch) and moving the
// whole tile (2 us).  The words travel in 16-byte records that carry the number of their round, so the reader
// polls the data itself, without a fence and a flag: 1.6 us a round for 16-column tiles, 2.1 us for 64-column ones
// (flags: 2.2 and 3.2 us; records sent from the last step's registers, in divergent stores, 2.7 us; all of a thread's
// records requested at once, of which most are not there yet, 2.3 us).
// Two slots of records by turns are enough: a CTA writes a slot again only after it has its neighbours' next records,
// which they sent after reading the last ones.  Waits are bounded (two seconds, then an error).
//
// Measured on B200 (us per step, one-step kernels -> one launch per T steps -> rounds, lid cavities): 128^2 FP32 1.74 ->
// 0.90 -> 0.78 and FP16S 2.07 -> 1.03 -> 0.91 (8 steps of 16 x 8 tiles); 512^2 FP32 4.2 -> 3.3 -> 2.5; 1024 x 256 channel
// FP32 3.9 -> 3.6 -> 2.9; 1000 x 300 channel FP16S 5.1 -> 4.4 -> 3.3; many tiles a CTA: 4096^2 FP32 189 -> 120.5 (139
// GLUPS; without walls 115, 146 GLUPS; at one crossing per step HBM allows 91).
//
// The cell update is the other kernels' (bgk_collide, codecs and random words, with the step counter advanced
// by T), so the results are bit-identical to single steps.  A launch leaves the state after T steps in
// the other buffer and the state T steps earlier where it was, so the host ends every run with a single step
// (lbm_get_macros and lbm_residual_fp64 read the state before the last one).
#pragma once

#include "internal.h"
#include "rowpipe.cuh"

namespace lbm {

// ---- two cells at a time in packed FP32 arithmetic ------------------------------------------
struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 a, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f32x2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ f32x2 operator+(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 operator-(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 operator*(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 mad(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 neg(f32x2 a) { return f32x2{a.v ^ 0x8000000080000000ull}; }
__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// 1 / a: the hardware's approximation and one Newton step in the form that rounds correctly (Markstein
// 1990).  Equal to the division for every float with 2^-24 <= |a| < 2^126 (lbm_test_reciprocal, over all of them): a
// density 1 + drho is zero or no less than 2^-24, and above 2^126 the equilibrium's 4.5 rho overflows in either form.  NaN for
// zero and infinite a, where a velocity j / rho is NaN either way.
__device__ __forceinline__ f32x2 reciprocal(f32x2 a, f32x2 neg_a) {
    float lo, hi;
    unpack2(a, lo, hi);
    const f32x2 r = pack2(rcp_approx(lo), rcp_approx(hi));
    return mad(mad(neg_a, r, both(1.0f)), r, r);
}

// What a class overwrites, as the packed collision takes it (a table in shared memory).
struct __align__(16) PairClass {
    uint32_t fl;
    float rho, ux, uy;
};

// moments() and apply_class() of two cells.
template <bool EXACTW, bool SPECIAL>
__device__ __forceinline__ void pair_moments(const PairClass& A, const PairClass& B, const f32x2 (&v)[9], float isc, f32x2& rho,
                                             f32x2& drho, f32x2& ux, f32x2& uy) {
    const f32x2 isc2 = both(isc);
    f32x2 r = v[0];
    static_for<8>([&](auto I) { r = r + v[I + 1]; });
    const f32x2 jx = ((((v[1] - v[3]) + v[5]) - v[6]) - v[7]) + v[8];
    const f32x2 jy = ((((v[2] - v[4]) + v[5]) + v[6]) - v[7]) - v[8];
    drho = EXACTW ? r : r * isc2;
    rho = both(1.0f) + drho;
    const f32x2 nrho = neg(rho);
    const f32x2 rinv = reciprocal(rho, nrho);
    const f32x2 inv = EXACTW ? rinv : rinv * isc2;  // a power of two: exact
    auto quot = [&](f32x2 j) {
        const f32x2 q = j * inv;
        return mad(mad(q, nrho, EXACTW ? j : j * isc2), rinv, q);
    };
    ux = quot(jx);
    uy = quot(jy);
    if constexpr (SPECIAL) {
        float a, b, c, d;
        unpack2(rho, a, b);
        unpack2(drho, c, d);
        if (A.fl & kSetRho) a = A.rho, c = A.rho - 1.0f;
        if (B.fl & kSetRho) b = B.rho, d = B.rho - 1.0f;
        rho = pack2(a, b);
        drho = pack2(c, d);
        unpack2(ux, a, b);
        if (A.fl & kSetUx) a = A.ux;
        if (B.fl & kSetUx) b = B.ux;
        ux = pack2(a, b);
        unpack2(uy, a, b);
        if (A.fl & kSetUy) a = A.uy;
        if (B.fl & kSetUy) b = B.uy;
        uy = pack2(a, b);
    }
}

// equilibrium_dev() of two cells: put(i, fe_i).
template <bool EXACTW, class Put>
__device__ __forceinline__ void pair_equilibrium(f32x2 rho, f32x2 drho, f32x2 ux, f32x2 uy, float sc, f32x2 minus_zero, Put&& put) {
    using L = D2Q9;
    const f32x2 nusq15 = both(-1.5f) * mad(uy, uy, ux * ux);
    const f32x2 rho3 = both(3.0f) * rho, rho45 = both(4.5f) * rho;
    const f32x2 base = mad(rho, nusq15, drho);
    auto wmul = [&](auto I, f32x2 x) {
        constexpr int i = decltype(I)::value;
        if constexpr (EXACTW) {
            constexpr float hi = float(L::w(i)), lo = float(L::w(i) - double(hi));
            return mad(both(hi), x, both(lo) * x);
        } else {
            return mad(both(float(L::w(i)) * sc), x, minus_zero);
        }
    };
    auto dirs = [&](auto I, f32x2 eu) {
        const f32x2 sym = wmul(I, mad(rho45, eu * eu, base));
        const f32x2 anti = wmul(I, rho3 * eu);
        put(I, sym + anti);
        put(std::integral_constant<int, L::opp(decltype(I)::value)>{}, sym - anti);
    };
    put(std::integral_constant<int, 0>{}, wmul(std::integral_constant<int, 0>{}, base));
    dirs(std::integral_constant<int, 1>{}, ux);
    dirs(std::integral_constant<int, 2>{}, uy);
    dirs(std::integral_constant<int, 5>{}, ux + uy);
    dirs(std::integral_constant<int, 6>{}, uy - ux);
}

// Direction i of two cells after the collision gave o: equilibrium cells take fe, solid ones what came from
// the other side.
template <int i, bool SPECIAL>
__device__ __forceinline__ f32x2 pair_boundary(const PairClass& A, const PairClass& B, f32x2 o, f32x2 fe, const f32x2 (&v)[9]) {
    if constexpr (SPECIAL) {
        float a, b, c, d;
        unpack2(o, a, b);
        unpack2(fe, c, d);
        if (A.fl & kEquilibrium) a = c;
        if (B.fl & kEquilibrium) b = d;
        if constexpr (i > 0) {
            unpack2(v[D2Q9::opp(i)], c, d);
            if (A.fl & kBounce) a = c;
            if (B.fl & kBounce) b = d;
        }
        return pack2(a, b);
    }
    return o;
}

// bgk_collide of two D2Q9 cells at once (FP32 arithmetic on deviations v, in storage units): its operations
// in its order, each on both lanes, so every lane's result is bgk_collide's.  A, B: the cells' classes
// (SPECIAL; without it both are plain fluid).  No Zou-He cells.
// minus_zero: a packed -0 the compiler cannot see through; with it a product that feeds an addition is a
// multiply-add of the same value, which cannot be contracted into the addition.
template <bool EXACTW, bool SPECIAL>
__device__ __forceinline__ void bgk_pair(const StepParams<float>& p, const PairClass& A, const PairClass& B, f32x2 (&v)[9],
                                         float sc, float isc, f32x2 minus_zero, f32x2 (&out)[9]) {
    f32x2 rho, drho, ux, uy;
    pair_moments<EXACTW, SPECIAL>(A, B, v, isc, rho, drho, ux, uy);
    const f32x2 om = both(p.omega), om1 = both(p.one_m_omega);
    pair_equilibrium<EXACTW>(rho, drho, ux, uy, sc, minus_zero, [&](auto I, f32x2 fe) {
        constexpr int i = decltype(I)::value;
        out[i] = pair_boundary<i, SPECIAL>(A, B, mad(om, fe, om1 * v[i]), fe, v);
    });
}

// psi = 1 - exp(-rho) of two cells' streamed density: sc_psi_from on both lanes.
template <bool SPECIAL>
__device__ __forceinline__ f32x2 sc_psi_pair(const PairClass& A, const PairClass& B, const f32x2 (&v)[9], float isc) {
    f32x2 r = v[0];
    static_for<8>([&](auto I) { r = r + v[I + 1]; });
    float a, b;
    unpack2(both(1.0f) + r * both(isc), a, b);  // a power of two: the product is exact
    if constexpr (SPECIAL) {
        if (A.fl & kSetRho) a = A.rho;
        if (B.fl & kSetRho) b = B.rho;
    }
    return pack2(1.0f - expf(-a), 1.0f - expf(-b));
}

// The Shan-Chen force (sc_force_from) and collision (sc_collide_store) of two cells: psi_at(dx, dy) gives both
// cells' neighbours.  Every product that feeds an addition goes through minus_zero (see bgk_pair).
template <bool EXACTW, bool SPECIAL, class PsiAt>
__device__ __forceinline__ void sc_pair(const StepParams<float>& p, const PairClass& A, const PairClass& B, f32x2 (&v)[9],
                                        float sc, float isc, f32x2 minus_zero, PsiAt&& psi_at, f32x2 (&out)[9]) {
    using L = D2Q9;
    f32x2 rho, drho, ux, uy;
    pair_moments<EXACTW, SPECIAL>(A, B, v, isc, rho, drho, ux, uy);
    f32x2 sx, sy;
    static_for<8>([&](auto I) {
        constexpr int i = I + 1, cx = L::cx(i), cy = L::cy(i);
        const f32x2 w = mad(both(float(L::w(i))), psi_at(std::integral_constant<int, cx>{}, std::integral_constant<int, cy>{}),
                            minus_zero);
        if constexpr (i == 1) sx = w;
        else if constexpr (cx == 1) sx = sx + w;
        else if constexpr (cx == -1) sx = sx - w;
        if constexpr (i == 2) sy = w;
        else if constexpr (cy == 1) sy = sy + w;
        else if constexpr (cy == -1) sy = sy - w;
    });
    const f32x2 g = both(-p.G) * psi_at(std::integral_constant<int, 0>{}, std::integral_constant<int, 0>{});
    const f32x2 orho = both(p.omega) * rho;
    const f32x2 k = reciprocal(orho, neg(orho));
    const f32x2 wx = ux + mad(g * sx, k, minus_zero), wy = uy + mad(g * sy, k, minus_zero);
    float a, b, c, d, ra, rb;
    unpack2(rho, ra, rb);  // no shift where rho <= 0
    unpack2(ux, a, b);
    unpack2(wx, c, d);
    const f32x2 vx = pack2(ra > 0.0f ? c : a, rb > 0.0f ? d : b);
    unpack2(uy, a, b);
    unpack2(wy, c, d);
    const f32x2 vy = pack2(ra > 0.0f ? c : a, rb > 0.0f ? d : b);
    const f32x2 om = both(p.omega), om1 = both(p.one_m_omega);
    pair_equilibrium<EXACTW>(rho, drho, vx, vy, sc, minus_zero, [&](auto I, f32x2 fe) {
        constexpr int i = decltype(I)::value;
        out[i] = pair_boundary<i, SPECIAL>(A, B, mad(om, fe, minus_zero) + mad(om1, v[i], minus_zero), fe, v);
    });
}

// Shape of the tile kernel: source regions of up to MAXR rows of PX cells in shared memory, direction by
// direction, HALO columns on either side of the tile's W.  MOVERS: warps that do nothing but bring the
// next tile's region in and store the last one's tile (two buffers), 0: the computing warps do.  BULK: they move
// whole rows by bulk copies where rows start on 16-byte words, else pieces.
// The steps compute the PW middle columns: D T <= (PW - W) / 2.  SC: Shan-Chen, whose step reaches D = 2 cells far
// and keeps psi of the region besides.
template <class S, bool SC_, int PX_, int PW_, int MAXR_, int HALO_, int WARPS_, int MOVERS_, bool BULK_>
struct TileShape {
    static constexpr bool SC = SC_, BULK = BULK_;
    static constexpr int D = SC ? 2 : 1;
    static constexpr int PX = PX_, PW = PW_, MAXR = MAXR_, HALO = HALO_, WARPS = WARPS_, MOVERS = MOVERS_;
    static constexpr int kMaxSteps = (PW - (PX - 2 * HALO)) / (2 * D);
    static constexpr int NBUF = MOVERS > 0 ? 2 : 1;
    static constexpr int W = PX - 2 * HALO, THREADS = 32 * WARPS, BLOCK = THREADS + 32 * MOVERS;
    static constexpr int GUARD = 16 / (int)sizeof(S);  // words before and after a direction's region
    static constexpr int PLANE = MAXR * PX + 2 * GUARD;
    static constexpr int BUF = 9 * PLANE;
    static_assert((PX * sizeof(S)) % 16 == 0 && (HALO * sizeof(S)) % 16 == 0, "rows of whole 16-byte words");
    static constexpr size_t kPop = 64 + sizeof(PairClass) * kMaxClasses;
    static constexpr size_t kPsi = kPop + (size_t)NBUF * BUF * sizeof(S);
    static constexpr size_t kCls = kPsi + (SC ? (size_t)(MAXR * PX + 8) * sizeof(typename Codec<S>::Real) : 0);
    static constexpr size_t kClsBytes = (size_t)(MAXR * PX + 15) / 16 * 16;
    // rounds (no MOVERS): the cells that a tile gives to others, and its halo
    static constexpr int kRecords = (9 * (int)sizeof(S) + 11) / 12;
    static constexpr int kReach = 2 * D * kMaxSteps;
    static constexpr int kMostHalo = (W + kReach) * kReach + (MAXR - kReach) * kReach;
    static constexpr int kMostRing = kReach * W + (MAXR - kReach) * kReach < W * MAXR ? kReach * W + (MAXR - kReach) * kReach : W * MAXR;
    static constexpr int kHaloTurns = (kMostHalo + THREADS - 1) / THREADS;
    static constexpr size_t kOutlets = kCls + NBUF * kClsBytes;  // words of class bytes with zero-gradient cells
    static constexpr size_t kEx = kOutlets + (SC ? 0 : ((size_t)(MAXR * PX / 4) * 2 + 15) / 16 * 16);
    static constexpr size_t kRingBytes = MOVERS ? 0 : ((size_t)kMostRing * 2 + 15) / 16 * 16;
    static constexpr size_t smem_bytes() { return kEx + kRingBytes + (MOVERS ? 0 : (size_t)kMostHalo * 8); }
};

// bgk_collide out of line, for the rare cells that the packed collision leaves (Zou-He), in the shapes without moving
// warps: keeps their loop short (512^2 3.38 -> 3.32 us a step; the others are faster without the call, 4096^2 124.7 -> 122.9).
template <bool EXACTW>
__device__ __noinline__ void tile_collide(const StepParams<float>& p, int cls, float* v, float sc, float isc) {
    float w[9], out[9];
    static_for<9>([&](auto I) { w[I] = v[I]; });
    bgk_collide<D2Q9, false, EXACTW>(p, cls, p.cls.flags[cls], w, sc, isc, out);
    static_for<9>([&](auto I) { v[I] = out[I]; });
}

// How a lattice's multi-step launches are cut.
enum TileKind { kTilesNone = 0, kTilesSmall, kTilesMid, kTilesPieces, kTilesStream, kTilesShanChen };
struct TilePlan {
    int kind = kTilesNone;
    int h = 0;      // rows of a tile (even)
    int steps = 0;  // steps per launch (even)
};
// What tiles that stay in their CTAs exchange between rounds (zeroed when allocated; one lattice's own).
// records: for each tile and cell of its border the nine words, three to a 16-byte record whose fourth word is
// the number of the round that wrote it; two slots, by rounds.
struct TileExchange {
    uint4* records = nullptr;    // [2][tiles][records of a cell][cap]
    unsigned* rounds = nullptr;  // [tiles] exchanges behind each tile
    int cap = 0;                 // cells of a tile's border, at most
    size_t bytes = 0;            // of the records
};
struct TileLaunch {
    StepParams<float> pf;
    StepParams<double> pd;
    int* err;
    TileExchange ex;
    int sms;
};
// Error word of a tile launch that gave up a wait.
constexpr int kTilesTimeout = 2;
// The plan of a D2Q9 BGK or Shan-Chen lattice on a device of `sms` SMs (kTilesNone: single steps are faster).
TilePlan plan_tiles(const lbm_desc& d, int sms);
// Most steps of one launch (where plan.steps is less: in rounds).
int tile_launch_steps(const TilePlan& plan);
// The exchange that launches in rounds of this plan need (cap and bytes; 0: none).
TileExchange tile_exchange(const lbm_desc& d, const TilePlan& plan);
cudaError_t launch_tiles(const lbm_desc& d, const TileLaunch& l, const TilePlan& plan, int steps, cudaStream_t s);

// Two adjacent words.
template <class S>
struct __align__(2 * sizeof(S)) Two {
    S a, b;
};

// A cell's byte in shared memory: class, and marks for a class with flags, a zero-gradient one, a Zou-He one.
constexpr uint32_t kMarkFlags = 0x80u, kMarkOutlet = 0x40u, kMarkZouHe = 0x20u, kMarkClass = 0x0fu;
// The same marks by class, one bit a class.
struct ClassMarks {
    uint32_t flags, outlet, zouhe;
};

__device__ __forceinline__ void bulk_store(void* dst_gmem, const void* src_smem, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem), "r"(smem_addr(src_smem)),
                 "r"(bytes)
                 : "memory");
}

// Place of cell (lx, ly) of a w x h tile in the order of its border (the cells within `depth` of its edges): the rows
// at both ends, then the rest of the columns; -1: an inner cell.
__host__ __device__ inline int ring_index(int lx, int ly, int w, int h, int depth) {
    const int rows = h < 2 * depth ? h : 2 * depth, cols = w < 2 * depth ? w : 2 * depth;
    const int top = h < depth ? h : depth, left = w < depth ? w : depth;
    if (ly < top) return ly * w + lx;
    if (ly >= h - (rows - top)) return (ly - (h - rows)) * w + lx;
    if (lx >= left && lx < w - (cols - left)) return -1;
    return rows * w + (ly - top) * cols + (lx < left ? lx : lx - (w - cols));
}

// Records are read and written whole (128-bit accesses are single-copy atomic): one with the right number is there.
__device__ __forceinline__ void store_record(uint4* to, const uint4& r) {
    asm volatile(
        "{\n\t.reg .b128 r;\n\t.reg .b64 lo, hi;\n\tmov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 r, {lo, hi};\n\t"
        "st.relaxed.gpu.global.b128 [%0], r;\n\t}" ::"l"(to),
        "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w)
        : "memory");
}
__device__ __forceinline__ uint4 load_record(const uint4* from) {
    uint4 r;
    asm volatile(
        "{\n\t.reg .b128 r;\n\t.reg .b64 lo, hi;\n\tld.relaxed.gpu.global.b128 r, [%4];\n\tmov.b128 {lo, hi}, r;\n\t"
        "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(from)
        : "memory");
    return r;
}

// One tile launch: tiles of W x h cells, `total` steps: T (even, D T <= HALO), or (no MOVERS, a tile a CTA) rounds of T.  nx >= PX and ny >= h + 2 D T
// (host-checked): every region cell wraps at most once.  CTAs walk the tiles with a stride.  A thread takes
// two cells at a time (PX and h are even).
// G: bytes of the pieces that regions and tiles move in, 16, 8, 4 or (16-bit words) 2: every row of the
// lattice starts on a multiple of it.
template <class S, bool ABS, class Sh, int G>
__global__ void __launch_bounds__(Sh::BLOCK, 1)
    k_step_tiles(const __grid_constant__ StepParams<typename Codec<S>::Real> p, int h, int T, int total, int tiles_x, int tiles,
                 const ClassMarks marks, float minus_zero, const TileExchange ex, int* __restrict__ err) {
    using L = D2Q9;
    using R = typename Codec<S>::Real;
    constexpr int Q = 9, PX = Sh::PX, PLANE = Sh::PLANE, THREADS = Sh::THREADS, HALO = Sh::HALO, W = Sh::W, NBUF = Sh::NBUF;
    constexpr bool k16 = Codec<S>::kScaled, kMove = Sh::MOVERS > 0;
    constexpr bool kPacked = std::is_same_v<R, float> && !ABS;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem);  // movers: [NBUF] the region is there
    uint64_t* const done = full + 2;                           // movers: [NBUF] the tile is computed
    PairClass* const table = reinterpret_cast<PairClass*>(smem + 64);
    S* const pops = reinterpret_cast<S*>(smem + Sh::kPop) + Sh::GUARD;
    const int tid = (int)threadIdx.x;
    const int nx = p.nx, ny = p.ny;
    const int depth = Sh::D * T, rows = h + 2 * depth;  // rows of the source region
    const uint32_t N = (uint32_t)p.N;  // 9 N <= 2^32 (host-checked)
    const int stride = (int)gridDim.x;
    constexpr int GW = G / (int)sizeof(S);  // cells of a piece
    static_assert(GW >= 1 && GW * (int)sizeof(S) == G, "pieces of whole words");
    constexpr bool SC = Sh::SC, kBulk = kMove && Sh::BULK && G == 16;
    static_assert(!SC || kPacked, "Shan-Chen tiles: packed FP32 arithmetic");
    using Piece = std::conditional_t<G == 16, uint4, std::conditional_t<G == 8, uint2, std::conditional_t<G == 4, uint32_t, uint16_t>>>;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid < kMaxClasses) table[tid] = PairClass{p.cls.flags[tid], (float)p.cls.rho[tid], (float)p.cls.ux[tid], (float)p.cls.uy[tid]};
    if constexpr (kMove) {
        if (tid == 0) {
            for (int b = 0; b < NBUF; ++b) {
                mbar_init(&full[b], kBulk ? 1 : 32 * Sh::MOVERS);
                mbar_init(&done[b], 1);
            }
            mbar_init_fence();
        }
        __syncthreads();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the launch before this one is complete

    const bool has_mask = p.mask != nullptr, words = has_mask && nx % 4 == 0;
    auto mark = [&](uint32_t c) {
        return c | ((marks.flags >> c) & 1u) << 7 | ((marks.outlet >> c) & 1u) << 6 | ((marks.zouhe >> c) & 1u) << 5;
    };
    auto cell_of = [&](int x0, int y0, int k) {  // lattice index of cell k of the region at (x0, y0)
        const int ly = k / PX;
        int x = x0 + (k - ly * PX), y = y0 + ly;
        x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
        y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
        return (uint32_t)y * (uint32_t)nx + (uint32_t)x;
    };
    // The region's class bytes, in words of four cells (x0 and PX are multiples of 4): a thread's words
    // from global memory, and with their marks to shared memory (returns the marks among them).
    constexpr int kClsWords = (Sh::MAXR * (PX / 4) + THREADS - 1) / THREADS;
    auto get_classes = [&](int n, uint32_t (&c)[kClsWords]) {
        const int ty = n / tiles_x, x0 = (n - ty * tiles_x) * W - HALO, y0 = ty * h - depth;
        static_for<kClsWords>([&](auto J) {
            const int j = tid + decltype(J)::value * THREADS;
            c[J] = 0;
            if (!has_mask || j >= rows * (PX / 4)) return;
            if (words)
                c[J] = __ldg(reinterpret_cast<const uint32_t*>(p.mask + cell_of(x0, y0, 4 * j)));
            else
                for (int u = 0; u < 4; ++u) c[J] |= (uint32_t)__ldg(p.mask + cell_of(x0, y0, 4 * j + u)) << (8 * u);
        });
    };
    auto put_classes = [&](const uint32_t (&c)[kClsWords], int b) {
        uint32_t* const dst = reinterpret_cast<uint32_t*>(smem + Sh::kCls + b * Sh::kClsBytes);
        uint32_t seen = 0;
        static_for<kClsWords>([&](auto J) {
            const int j = tid + decltype(J)::value * THREADS;
            if (j >= rows * (PX / 4)) return;
            uint32_t w = mark(0u) * 0x01010101u;
            if (!kMove || c[J] != 0u) {  // (many tiles: most words are class 0 throughout)
                w = 0;
                for (int u = 0; u < 4; ++u) w |= mark((c[J] >> (8 * u)) & 0xffu) << (8 * u);
            }
            dst[j] = w;
            seen |= w;
        });
        seen |= seen >> 16;
        return (seen | seen >> 8) & (kMarkFlags | kMarkOutlet | kMarkZouHe);
    };
    const bool classes = has_mask || mark(0u) != 0;  // some cell of the lattice may not be plain fluid

    // The source region of tile n into buffer b, f_i of cell (x0 + lx, y0 + ly) to [i][ly PX + lx], and tile n
    // out of buffer b, in pieces, by `count` threads.
    auto pieces_in = [&](int n, int b, int who, int count) {
        const int ty = n / tiles_x, x0 = (n - ty * tiles_x) * W - HALO, y0 = ty * h - depth;
        const char* const fin = static_cast<const char*>(p.fin);
        for (int j = who; j < rows * (PX / GW); j += count) {
            const int ly = j / (PX / GW), lx = (j - ly * (PX / GW)) * GW;
            int x = x0 + lx, y = y0 + ly;
            x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
            y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
            const uint32_t off = ((uint32_t)y * (uint32_t)nx + (uint32_t)x) * (uint32_t)sizeof(S);
            S* const dst = pops + b * Sh::BUF + ly * PX + lx;
            static_for<Q>([&](auto I) {
                constexpr int i = I;
                const char* const base = fin + (size_t)i * N * sizeof(S);
                if constexpr (G == 16)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst + i * PLANE)), "l"(base + off)
                                 : "memory");
                else if constexpr (G >= 4)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst + i * PLANE)), "l"(base + off),
                                 "n"(G)
                                 : "memory");
                else
                    dst[i * PLANE] = __ldcg(reinterpret_cast<const S*>(base + off));
            });
        }
    };
    auto pieces_out = [&](int n, int b, int who, int count) {
        const int ty = n / tiles_x, x0 = (n - ty * tiles_x) * W, y0 = ty * h;
        char* const fout = static_cast<char*>(p.fout);
        const S* const buf = pops + b * Sh::BUF + depth * PX + HALO;
        for (int j = who; j < h * (W / GW); j += count) {
            const int ly = j / (W / GW), lx = (j - ly * (W / GW)) * GW;
            const int x = x0 + lx, y = y0 + ly;
            if (x >= nx || y >= ny) continue;
            const uint32_t off = ((uint32_t)y * (uint32_t)nx + (uint32_t)x) * (uint32_t)sizeof(S);
            const S* const src = buf + ly * PX + lx;
            static_for<Q>([&](auto I) {
                constexpr int i = I;
                char* const base = fout + (size_t)i * N * sizeof(S);
                *reinterpret_cast<Piece*>(base + off) = *reinterpret_cast<const Piece*>(src + i * PLANE);
            });
        }
    };
    // barrier of one group of warps (1: computing, 2: moving) and its vote
    auto vote = [](int id, int count, bool v) {
        int r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(r)
            : "r"((unsigned)v), "r"(id), "r"(count)
            : "memory");
        return r != 0;
    };

    if constexpr (kMove) {
        if (tid >= THREADS) {
            constexpr int MT = 32 * Sh::MOVERS;
            const int m = tid - THREADS;
            auto move_in = [&](int n, int b) {
                if constexpr (!kBulk) {
                    pieces_in(n, b, m, MT);
                    if constexpr (G >= 4)  // arrives when this thread's copies have landed
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(&full[b])) : "memory");
                    else
                        mbar_arrive(&full[b]);
                } else {
                    const int ty = n / tiles_x, x0 = (n - ty * tiles_x) * W - HALO, y0 = ty * h - depth;
                    const S* __restrict__ const fin = static_cast<const S*>(p.fin);
                    const int a = x0 < 0 ? x0 + nx : x0, len = nx - a < PX ? nx - a : PX;  // before the wrap in x
                    if (m == 0) mbar_arrive_expect_tx(&full[b], (uint32_t)(Q * rows * PX * (int)sizeof(S)));
                    for (int j = m; j < Q * rows; j += MT) {
                        const int ly = j / Q, i = j - ly * Q;
                        int y = y0 + ly;
                        y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
                        const S* const row = fin + ((size_t)i * N + (size_t)((uint32_t)y * (uint32_t)nx));
                        S* const dst = pops + b * Sh::BUF + i * PLANE + ly * PX;
                        bulk_load(dst, row + a, (uint32_t)(len * (int)sizeof(S)), &full[b]);
                        if (len < PX) bulk_load(dst + len, row, (uint32_t)((PX - len) * (int)sizeof(S)), &full[b]);
                    }
                }
            };
            auto move_out = [&](int n, int b) {
                if constexpr (!kBulk) {
                    pieces_out(n, b, m, MT);
                } else {
                    const int ty = n / tiles_x, x0 = (n - ty * tiles_x) * W, y0 = ty * h;
                    const int w = nx - x0 < W ? nx - x0 : W, hh = ny - y0 < h ? ny - y0 : h;
                    S* const fout = static_cast<S*>(p.fout);
                    for (int j = m; j < Q * hh; j += MT) {
                        const int r = j / Q, i = j - r * Q;
                        bulk_store(fout + ((size_t)i * N + (size_t)((uint32_t)(y0 + r) * (uint32_t)nx + (uint32_t)x0)),
                                   pops + b * Sh::BUF + i * PLANE + (r + depth) * PX + HALO, (uint32_t)(w * (int)sizeof(S)));
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            };
            // Pieces of lattices beyond L2: the lines of the tile after the next one are asked into L2 meanwhile.  Pieces
            // in flight are few (the small L1 holds them), so it is their latency that counts: Shan-Chen FP32
            // 2049 x 1537 53.8 -> 50.3 us a step, 4096 x 1024 56.1 -> 54.9, BGK FP32 3001 x 2003 63.6 -> 57.0.  In L2 it
            // costs more than it gives (Shan-Chen 1023^2, 75 MB, 16.4 -> 16.8; BGK 1501 x 1201, 130 MB, 21.1 -> 20.4), and
            // bulk copies need no help (4096^2 FP32 125.8 -> 130.2).
            const bool far = !kBulk && 18ULL * sizeof(S) * N > 110000000ULL;
            auto prefetch = [&](int n2) {
                if (n2 >= tiles) return;
                constexpr int LINES = (PX * (int)sizeof(S) + 124) / 128 + 1, LW = 128 / (int)sizeof(S);
                const int ty = n2 / tiles_x, x0 = (n2 - ty * tiles_x) * W - HALO, y0 = ty * h - depth;
                for (int j = m; j < rows * Q * LINES; j += MT) {
                    const int ly = j / (Q * LINES), rest = j - ly * (Q * LINES), i = rest / LINES, part = rest - i * LINES;
                    const uint32_t c = cell_of(x0, y0, ly * PX + (part * LW < PX - 1 ? part * LW : PX - 1));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const S*>(p.fin) + ((size_t)i * N + c)));
                }
            };
            int n = (int)blockIdx.x;
            for (int b = 0; b < NBUF; ++b)
                if (n + b * stride < tiles) move_in(n + b * stride, b);
            if (far) prefetch(n + NBUF * stride);
            for (int turn = 0; n < tiles; ++turn, n += stride) {
                const int b = turn & 1;
                const bool ok = mbar_wait_bounded(&done[b], (uint32_t)((turn >> 1) & 1));
                if (vote(2, MT, !ok)) {
                    if (!ok) atomicExch(err, kTilesTimeout);
                    if constexpr (kBulk) {  // wait, briefly and bounded, for copies that may still land in this CTA's regions
                        mbar_wait_bounded(&full[b], (uint32_t)((turn >> 1) & 1), 1LL << 28);
                        if (n + stride < tiles) mbar_wait_bounded(&full[b ^ 1], (uint32_t)(((turn + 1) >> 1) & 1), 1LL << 28);
                    }
                    break;
                }
                move_out(n, b);
                if (n + NBUF * stride < tiles) {
                    if constexpr (kBulk) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    vote(2, MT, false);  // every mover has read its part of the buffer
                    move_in(n + NBUF * stride, b);
                    if (far) prefetch(n + (NBUF + 1) * stride);
                }
            }
            if constexpr (kBulk) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
            return;
        }
    }
    auto barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); };
    auto any = [&](bool v) { return vote(1, THREADS, v); };

    R sc, isc;
    storage_scale<S>(p, sc, isc);
    unsigned t0 = 0;
    if constexpr (k16) {
        if (p.sr) {
            t0 = p.tick[p.parity];
            if ((blockIdx.x | (unsigned)tid) == 0) p.tick[p.parity ^ 1] = t0 + (unsigned)total;
        }
    }
    uint32_t next_cls[kClsWords], seen = 0;
    if (kMove && classes && (int)blockIdx.x < tiles) {
        get_classes((int)blockIdx.x, next_cls);
        seen = put_classes(next_cls, 0);
    }
#pragma unroll 1
    for (int turn = 0, n = (int)blockIdx.x; n < tiles; ++turn, n += stride) {
        const int b = NBUF == 2 ? turn & 1 : 0;
        const int ty = n / tiles_x, tx = n - ty * tiles_x;
        const int x0 = tx * W - HALO, y0 = ty * h - depth;
        S* const pop = pops + b * Sh::BUF;
        if constexpr (!kMove) pieces_in(n, 0, tid, THREADS);
        const uint8_t* const cls_s = smem + Sh::kCls + b * Sh::kClsBytes;
        uint32_t kind = 0;  // marks among the region's cells
        if constexpr (kMove) {
            const bool ok = mbar_wait_bounded(&full[b], (uint32_t)((turn >> 1) & 1));
            if (!ok) atomicExch(err, kTilesTimeout);
            if (any(!ok)) return;
        } else {
            if (classes) {
                get_classes(n, next_cls);
                seen = put_classes(next_cls, 0);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        if (classes) {
            kind = any(seen != 0) ? kMarkFlags : 0u;
            if (kind) kind |= (any((seen & kMarkOutlet) != 0) ? kMarkOutlet : 0u) | (any((seen & kMarkZouHe) != 0) ? kMarkZouHe : 0u);
        } else if (!kMove) {
            barrier();
        }
        // the words of class bytes with zero-gradient cells, last first
        uint16_t* const outlet = reinterpret_cast<uint16_t*>(smem + Sh::kOutlets);
        int outlets = 0;
        if (!SC && (kind & kMarkOutlet)) {
            int* const found = reinterpret_cast<int*>(smem + 32);
            if (tid < 32) {
                const int words_ = rows * (PX / 4);
                int sum = 0;
#pragma unroll 4
                for (int from = 0; from < words_; from += 32) {
                    const int m = words_ - 1 - from - tid;
                    const uint32_t c = m >= 0 ? reinterpret_cast<const uint32_t*>(cls_s)[m] : 0u;
                    const bool has = (c & (kMarkOutlet * 0x01010101u)) != 0;
                    const unsigned all = __ballot_sync(0xffffffffu, has);
                    if (has) outlet[sum + __popc(all & ((1u << tid) - 1u))] = (uint16_t)m;
                    sum += __popc(all);
                }
                if (tid == 0) *found = sum;
            }
            barrier();
            outlets = *found;
        }
        unsigned base = 0;
        int ring = 0, halo = 0;
        uint16_t* const ring_k = reinterpret_cast<uint16_t*>(smem + Sh::kEx);
        uint2* const halo_k = reinterpret_cast<uint2*>(smem + Sh::kEx + Sh::kRingBytes);
        if (!kMove && total > T) {
            // Rounds.  ring_k: the region's index of each cell that others need, in the order of its records;
            // halo_k: for each cell of the halo its first record and its index.
            base = ex.rounds[n];
            auto width = [&](int t) { return nx - t * W < W ? nx - t * W : W; };
            auto height = [&](int t) { return ny - t * h < h ? ny - t * h : h; };
            const int w = width(tx), hh = height(ty);
            auto ends = [&](int size) { return size < 2 * depth ? size : 2 * depth; };
            ring = ends(hh) * w + (hh - ends(hh)) * ends(w);
            for (int q = tid; q < hh * w; q += THREADS) {
                const int ly = q / w, lx = q - ly * w;
                const int at = ring_index(lx, ly, w, hh, depth);
                if (at >= 0) ring_k[at] = (uint16_t)((ly + depth) * PX + lx + HALO);
            }
            const int full = w + 2 * depth, caps = 2 * depth * full;
            halo = caps + hh * 2 * depth;
            for (int m = tid; m < halo; m += THREADS) {
                int ly, lx;
                if (m < caps) {
                    ly = m / full;
                    lx = m - ly * full;
                    if (ly >= depth) ly += hh;
                } else {
                    ly = (m - caps) / (2 * depth);
                    lx = m - caps - ly * 2 * depth;
                    ly += depth;
                    if (lx >= depth) lx += w;
                }
                lx += HALO - depth;
                const uint32_t c = cell_of(x0, y0, ly * PX + lx);
                const int y = (int)(c / (uint32_t)nx), x = (int)(c - (uint32_t)y * (uint32_t)nx);
                const int sx = x / W, sy = y / h;
                const int at = ring_index(x - sx * W, y - sy * h, width(sx), height(sy), depth);
                halo_k[m] = uint2{(uint32_t)((sy * tiles_x + sx) * Sh::kRecords) * (uint32_t)ex.cap + (uint32_t)at,
                                  (uint32_t)(ly * PX + lx)};
            }
            barrier();
        }
        // the next tile's classes travel while this one is computed
        if (kMove && classes && n + stride < tiles) get_classes(n + stride, next_cls);

        int before = 0;  // steps behind
        // One step.  AROUND (odd t): reads and writes the neighbours' words; else the cell's own.
        auto step = [&](auto Around, auto Special, int t) {
            constexpr bool around = decltype(Around)::value, SPECIAL = decltype(Special)::value;
            Rounding rnd{0u, false};
            if constexpr (k16) {
                if (p.sr) rnd = Rounding{seed_of_step(t0 + (unsigned)((kMove ? 0 : before) + t - 1)), true};
            }
            // the two cells of a thread: adjacent, or (FP32 and FP64 words around, where adjacent cells would
            // meet in a bank) half the rows apart
            constexpr bool adj = !around || k16;
            constexpr int PW = Sh::PW;
            const int edge = Sh::D * t;  // the outermost rows that are not computed
            const int half = (rows / 2 - edge) * PX;
            const int count = (rows / 2 - edge) * PW, second = adj ? 1 : half;  // pairs of cells
            const int first = edge * PX;
            if constexpr (SPECIAL && !SC) {
                // A zero-gradient cell's c_x = -1 populations are f_i(x, y - c_iy) of its own column, which
                // the cell to its left reads and overwrites.  They are copied to where the cell itself
                // reads, which no other cell touches in this step.
                // Cell k's copies go where those of cell k + 1 come from, so the last cells are first.
                for (int from = 0; from < outlets; from += THREADS) {
                    const int m = from + tid < outlets ? (int)outlet[from + tid] : -1;
                    const bool mine = m >= first / 4 && m < (rows * PX - first) / 4;
                    const uint32_t word = mine ? reinterpret_cast<const uint32_t*>(cls_s)[m] : 0u;
                    S zg[4][3];
                    static_for<4>([&](auto U) {
                        constexpr int u = U;
                        if ((word >> (8 * u)) & kMarkOutlet)
                            static_for<3>([&](auto J) {
                                constexpr int i = J == 0 ? 3 : (J == 1 ? 6 : 7);
                                const int k = 4 * m + u;
                                zg[u][J] = around ? pop[i * PLANE + k - L::cy(i) * PX] : pop[L::opp(i) * PLANE + k - 1];
                            });
                    });
                    barrier();
                    static_for<4>([&](auto U) {
                        constexpr int u = U;
                        if ((word >> (8 * u)) & kMarkOutlet)
                            static_for<3>([&](auto J) {
                                constexpr int i = J == 0 ? 3 : (J == 1 ? 6 : 7);
                                const int k = 4 * m + u;
                                (around ? pop[i * PLANE + k - L::cy(i) * PX + 1] : pop[L::opp(i) * PLANE + k]) = zg[u][J];
                            });
                    });
                    barrier();
                }
            }
            auto value = [&](S w, auto I) -> R {
                if constexpr (ABS)
                    return R(w);
                else
                    return Codec<S>::raw(w, R(L::w(decltype(I)::value)));
            };
            auto pair_of = [&](int j, int from) {  // first cell of pair j of the rows from `from` on
                int k = from + (adj ? 2 * j : j);
                if constexpr (PW < PX) {
                    constexpr int PR = adj ? PW / 2 : PW;  // pairs of a row
                    k += (j / PR) * (PX - PW) + (PX - PW) / 2;
                }
                return k;
            };
            auto load_pair = [&](const S* c, const S* d, S(&wA)[Q], S(&wB)[Q]) {
                static_for<Q>([&](auto I) {
                    constexpr int i = I, o = around ? i * PLANE - (L::cy(i) * PX + L::cx(i)) : L::opp(i) * PLANE;
                    if constexpr (adj && (!around || L::cx(i) == 0)) {
                        const Two<S> w = *reinterpret_cast<const Two<S>*>(c + o);
                        wA[i] = w.a;
                        wB[i] = w.b;
                    } else {
                        wA[i] = c[o];
                        wB[i] = d[o];
                    }
                });
            };
            auto pack_pair = [&](const S(&wA)[Q], const S(&wB)[Q], f32x2(&v)[Q]) {
                static_for<Q>([&](auto I) {
                    constexpr int i = I;
                    if constexpr (k16)
                        v[i] = pack2(value(wA[i], I), value(wB[i], I));
                    else if constexpr (kPacked)
                        v[i] = pack2(wA[i], wB[i]) - both(float(L::w(i)));
                });
            };
            [[maybe_unused]] R* const psi = reinterpret_cast<R*>(smem + Sh::kPsi) + 4;
            if constexpr (SC) {
                // psi of the streamed densities, one cell further out than what is collided
                const int rim = edge - 1, apart = (rows / 2 - rim) * PX, away = adj ? 1 : apart;
#pragma unroll 1
                for (int j = tid; j < (rows / 2 - rim) * PW; j += THREADS) {
                    const int k = pair_of(j, rim * PX);
                    S wA[Q], wB[Q];
                    f32x2 v[Q];
                    load_pair(pop + k, pop + k + away, wA, wB);
                    pack_pair(wA, wB, v);
                    PairClass A{}, B{};
                    if constexpr (SPECIAL) {
                        A = table[cls_s[k] & kMarkClass];
                        B = table[cls_s[k + away] & kMarkClass];
                    }
                    float a, b2;
                    unpack2(sc_psi_pair<SPECIAL>(A, B, v, isc), a, b2);
                    if constexpr (adj) {
                        *reinterpret_cast<float2*>(psi + k) = float2{a, b2};
                    } else {
                        psi[k] = a;
                        psi[k + away] = b2;
                    }
                }
                barrier();
            }
#pragma unroll 1
            for (int j = tid; j < count; j += THREADS) {
                const int k = pair_of(j, first);
                S* const c = pop + k;
                S* const d = c + second;
                S wA[Q], wB[Q];
                load_pair(c, d, wA, wB);
                uint32_t mA = 0, mB = 0;
                if constexpr (SPECIAL) {
                    mA = cls_s[k];
                    mB = cls_s[k + second];
                }
                R oA[Q], oB[Q];  // stored values: collided deviations for the 16-bit codecs, populations else
                auto scalar = [&](const S(&w)[Q], uint32_t m, R(&o)[Q]) {
                    R v[Q], out[Q];
                    const int cls = (int)(m & kMarkClass);
                    static_for<Q>([&](auto I) { v[I] = value(w[I], I); });
                    if constexpr (kPacked && !kMove) {
                        tile_collide<kExactWeights<S>>(p, cls, v, sc, isc);
                        static_for<Q>([&](auto I) { out[I] = v[I]; });
                    } else {
                        bgk_collide<L, ABS, kExactWeights<S>>(p, cls, SPECIAL ? p.cls.flags[cls] : 0u, v, sc, isc, out);
                    }
                    static_for<Q>([&](auto I) {
                        constexpr int i = I;
                        if constexpr (k16 || ABS)
                            o[i] = out[i];
                        else
                            o[i] = Codec<S>::enc(out[i], R(L::w(i)));
                    });
                };
                if constexpr (kPacked) {
                    auto packed = [&](auto Sp) {
                        f32x2 v[Q], out[Q];
                        pack_pair(wA, wB, v);
                        PairClass A{}, B{};
                        if constexpr (decltype(Sp)::value) {
                            A = table[mA & kMarkClass];
                            B = table[mB & kMarkClass];
                        }
                        if constexpr (SC) {
                            auto psi_at = [&](auto DX, auto DY) {
                                constexpr int dx = decltype(DX)::value, o = decltype(DY)::value * PX + dx;
                                if constexpr (adj && dx == 0) {
                                    const float2 q = *reinterpret_cast<const float2*>(psi + k + o);
                                    return pack2(q.x, q.y);
                                } else {
                                    return pack2(psi[k + o], psi[k + second + o]);
                                }
                            };
                            sc_pair<kExactWeights<S>, decltype(Sp)::value>(p, A, B, v, sc, isc, both(minus_zero), psi_at, out);
                        } else {
                            bgk_pair<kExactWeights<S>, decltype(Sp)::value>(p, A, B, v, sc, isc, both(minus_zero), out);
                        }
                        static_for<Q>([&](auto I) {
                            constexpr int i = I;
                            // F32: the stored word w + d
                            unpack2(k16 ? out[i] : both(float(L::w(i))) + out[i], oA[i], oB[i]);
                        });
                    };
                    if constexpr (!SPECIAL) {
                        packed(std::false_type{});
                    } else if (!__any_sync(__activemask(), ((mA | mB) & kMarkFlags) != 0u)) {
                        packed(std::false_type{});
                    } else if (SC || !(kind & kMarkZouHe)) {
                        packed(std::true_type{});
                    } else {
                        scalar(wA, mA, oA);
                        scalar(wB, mB, oB);
                    }
                } else {
                    scalar(wA, mA, oA);
                    scalar(wB, mB, oB);
                }
                // stored words
                if constexpr (k16) {
                    // the same random bits as encode16 gives each cell, both cells of a direction in one conversion
                    const uint32_t cA = cell_of(x0, y0, k) + p.cell_base, cB = cell_of(x0, y0, k + 1) + p.cell_base;
                    const PairBits pb{(cell_hash16(cB, rnd.seed) << 16) | cell_hash16(cA, rnd.seed)};
                    static_for<Q>([&](auto I) {
                        constexpr int i = I, o = around ? L::opp(i) * PLANE + (L::cy(i) * PX + L::cx(i)) : i * PLANE;
                        const uint32_t w = rnd.sr ? Pair16<S>::rs(oB[i], oA[i], pb.template word<i, i>()) : Pair16<S>::rn(oB[i], oA[i]);
                        if constexpr (!around || L::cx(i) == 0) {
                            *reinterpret_cast<uint32_t*>(c + o) = w;
                        } else {
                            c[o] = Pair16<S>::lo(w);
                            d[o] = Pair16<S>::hi(w);
                        }
                    });
                } else {
                    static_for<Q>([&](auto I) {
                        constexpr int i = I, o = around ? L::opp(i) * PLANE + (L::cy(i) * PX + L::cx(i)) : i * PLANE;
                        if constexpr (adj) {
                            *reinterpret_cast<Two<S>*>(c + o) = Two<S>{S(oA[i]), S(oB[i])};
                        } else {
                            c[o] = S(oA[i]);
                            d[o] = S(oB[i]);
                        }
                    });
                }
            }
            if (kBulk && !around && t == T) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            barrier();
        };
        auto steps = [&](auto Special) {
#pragma unroll 1
            for (int t = 1; t < (kMove ? T : min(T, total - before)); t += 2) {
                step(std::true_type{}, Special, t);
                step(std::false_type{}, Special, t + 1);
            }
        };
        int r = 0;  // rounds behind
#pragma unroll 1
        while (true) {
            if (kind)
                steps(std::true_type{});
            else
                steps(std::false_type{});
            if constexpr (kMove) break;
            before += T;
            if (before >= total) break;
            ++r;
            const unsigned tag = base + (unsigned)r;
            const uint32_t slot = (tag & 1u) * (uint32_t)(tiles * Sh::kRecords) * (uint32_t)ex.cap;
            for (int q = tid; q < ring; q += THREADS) {
                const S* const at = pop + ring_k[q];
                uint32_t wd[3 * Sh::kRecords] = {};
                static_for<Q>([&](auto I) {
                    constexpr int i = I;
                    const S v = at[i * PLANE];
                    if constexpr (sizeof(S) == 2)
                        wd[i / 2] |= (uint32_t)*reinterpret_cast<const uint16_t*>(&v) << (16 * (i & 1));
                    else if constexpr (sizeof(S) == 4)
                        wd[i] = __float_as_uint((float)v);
                    else {
                        wd[2 * i] = (uint32_t)__double2loint((double)v);
                        wd[2 * i + 1] = (uint32_t)__double2hiint((double)v);
                    }
                });
                uint4* const to = ex.records + slot + (uint32_t)(n * Sh::kRecords) * (uint32_t)ex.cap + q;
                static_for<Sh::kRecords>([&](auto J) {
                    constexpr int j = J;
                    store_record(to + j * ex.cap, uint4{wd[3 * j], wd[3 * j + 1], wd[3 * j + 2], tag});
                });
            }
            bool late = false;
            static_for<Sh::kHaloTurns>([&](auto U) {
                const int m = tid + (int)U * THREADS;
                if (m >= halo) return;
                const uint2 cell = halo_k[m];
                const uint4* const from = ex.records + slot + cell.x;
                uint4 rec[Sh::kRecords];
                static_for<Sh::kRecords>([&](auto J) { rec[J] = load_record(from + J * ex.cap); });
                while (true) {
                    int missing = -1;
                    static_for<Sh::kRecords>([&](auto J) { missing = rec[J].w != tag ? (int)J : missing; });
                    if (missing < 0 || late) break;
                    const long long c0 = clock64();
                    while (!late && load_record(from + missing * ex.cap).w != tag) late = clock64() - c0 > (1LL << 32);
                    static_for<Sh::kRecords>([&](auto J) { rec[J] = load_record(from + J * ex.cap); });
                }
                S* const at = pop + cell.y;
                uint32_t wd[3 * Sh::kRecords];
                static_for<Sh::kRecords>([&](auto J) {
                    wd[3 * J] = rec[J].x;
                    wd[3 * J + 1] = rec[J].y;
                    wd[3 * J + 2] = rec[J].z;
                });
                static_for<Q>([&](auto I) {
                    constexpr int i = I;
                    if constexpr (sizeof(S) == 2)
                        reinterpret_cast<uint16_t*>(at)[i * PLANE] = (uint16_t)(wd[i / 2] >> (16 * (i & 1)));
                    else if constexpr (sizeof(S) == 4)
                        at[i * PLANE] = S(__uint_as_float(wd[i]));
                    else
                        at[i * PLANE] = S(__hiloint2double((int)wd[2 * i + 1], (int)wd[2 * i]));
                });
            });
            if (late) atomicExch(err, kTilesTimeout);
            if (any(late)) return;
        }
        if (!kMove && total > T && tid == 0) ex.rounds[n] = base + (unsigned)r;
        if constexpr (kMove) {
            if (tid == 0) mbar_arrive(&done[b]);
            if (classes && n + stride < tiles) seen = put_classes(next_cls, b ^ 1);
        } else {
            pieces_out(n, 0, tid, THREADS);  // (one tile a CTA)
        }
    }
}

}  // namespace lbm
