// The pressure solve as ONE persistent cooperative kernel per solve on sm_103a.
//
// Multigrid-preconditioned conjugate gradients on the two potentials (pressure * dt and
// the density-correction potential) side by side, each with its own step lengths and
// convergence flag (reduce_tail.glsl:61-116), preconditioned by an aggregation V-cycle:
// Galerkin 2 x 2 coarse matrices (mg_build.comp:147-197, mg_tail.comp:44-70), red-black
// Gauss-Seidel from zero on the way down with restriction of the residual (mg_down.comp),
// coarse correction with omega = 1.8 and the mirrored sweep on the way up (mg_up.comp),
// and the small levels (<= 1500 cells) in one thread block (mg_tail.comp:159-225).
//
// What the reference spreads over ~15 dispatches and barriers per iteration, with a
// host-recorded iteration count, runs here inside one kernel with a device-decided exit:
// the phases are separated by a grid-wide barrier (bounded spin; on timeout every block
// sets the error word and leaves), every block computes the solve's scalars itself from the
// per-tile partial sums (the same work-group trees and strided totals as
// reduce.glsl / reduce_tail.glsl, so every block gets identical values), and the residual
// update of conjugate gradients is fused into the first restriction of the next V-cycle by
// double-buffering the level-0 residual.
//
// Two precisions, one kernel template:
//   Plain  the reference's arithmetic: every value FP32, the dot products summed in FP32 in
//          the reference's order (bit-exact with the oracle).
//   Mixed  the V-cycle's matrices (every level's couplings) stored in BF16 and computed in
//          FP32; the CG operator (level 0's matrix), every vector, iterate, residual and
//          direction stay FP32; the dot products summed in FP32 as the plain solve sums
//          them, their totals widened to FP64 for the step lengths and the convergence
//          test; the refinement's checks and the closing true residual b - A x evaluated
//          as float pairs (products exact, sums compensated). The BF16 couplings come with
//          an FP32 diagonal that keeps each row's exact excess over them (see Mixed::setA).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "dev_common.cuh"
#include "kernels.h"
#include "solve_common.cuh"

namespace sprout {

namespace {

using namespace solve;

__constant__ int NBX[4] = {-1, 1, 0, 0};
__constant__ int NBY[4] = {0, 0, -1, 1};


// ---- the two precisions ---------------------------------------------------------------

struct Plain {
    static constexpr bool kMixed = false;
    static constexpr uint32_t kHier = HIER_PLAIN;
    using acc = float;
    using acc4 = float4;
    DEV static float4 A(const DevScene& d, int i) { return d.mga[i]; }
    DEV static float Dg(const DevScene& d, int i) { return d.mgd[i]; }
    DEV static void setA(const DevScene& d, int i, float4 a, float dg) {
        d.mga[i] = a;
        d.mgd[i] = dg;
        d.mgy[i] = make_float2(dg, recip_row(dg, a));
    }
    DEV static acc4* part(const DevScene& d) { return d.partials; }
    DEV static acc4 zero4() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
    // the four products a_k b_k of a cell's partial sums, and a total as the scalars use it
    DEV static acc4 prod4(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
        return make_float4(a0 * b0, a1 * b1, a2 * b2, a3 * b3);
    }
    DEV static float4 fin(acc4 a) { return a; }
    // what the smoothers read of a row: its couplings, and the diagonal with its reciprocal (zero
    // where the cell is no unknown)
    using Row = float4;
    using Diag = float2;
    DEV static const Row* rows(const DevScene& d) { return d.mga; }
    DEV static const Diag* diags(const DevScene& d) { return d.mgy; }
    DEV static float4 wide(const Row& a) { return a; }
    DEV static Diag no_diag() { return make_float2(0.0f, 0.0f); }
    DEV static bool unk(const Diag& y) { return y.x > 0.0f; }
    DEV static float4 pack_red(float2 r, const Diag& y) { return make_float4(r.x, r.y, y.x, y.y); }
    DEV static void unpack_red(const float4& v, float2& r, Diag& y) {
        r = make_float2(v.x, v.y);
        y = make_float2(v.z, v.w);
    }
    // a / D the fast way, whether it may be taken that way (an unknown's), the IEEE division, and y
    // with a reciprocal that says it may not
    DEV static float2 quot(float2 a, const Diag& y) { return quot2(a, y); }
    DEV static bool ok(float2 a, const Diag& y) { return quot_ok<60>(a, y.y); }
    DEV static float2 quot_ieee(float2 a, const Diag& y) { return quot2_ieee(a, y); }
    DEV static Diag spoilt(const Diag& y) { return make_float2(y.x, __int_as_float(0x7fffffff)); }
};

// a pair of BF16 values in 32 bits (x in the low half), rounded to nearest even
DEV uint32_t pack(float2 v) {
    __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
DEV float2 unpack(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u)); }

struct Mixed {
    static constexpr bool kMixed = true;
    static constexpr uint32_t kHier = HIER_MIXED;
    using acc = double;
    // the dot products' partial sums and totals in FP32 as the plain solve takes them (the
    // reference's trees), widened to FP64 for the step lengths and the convergence test
    using acc4 = float4;
    // the hierarchy in BF16: a row's four couplings as two bfloat162 in a uint2
    DEV static float4 A(const DevScene& d, int i) {
        const uint2 u = d.hga[i];
        const float2 a = unpack(u.x), b = unpack(u.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    DEV static float Dg(const DevScene& d, int i) { return d.hgd[i]; }
    // A row whose couplings m (a mask of the unknown neighbours) link it to other unknowns:
    // the couplings rounded to BF16, the diagonal rebuilt as its excess over the FP32
    // couplings plus the rounded ones, so that every row sum (the air, solid and vent terms
    // that keep a sealed region's matrix definite) is kept exactly and the stored matrix
    // stays a weighted graph Laplacian plus the same non-negative diagonal.
    DEV static void setA(const DevScene& d, int i, float4 a, float dg, int m = 15) {
        const uint2 u = make_uint2(pack(make_float2(a.x, a.y)), pack(make_float2(a.z, a.w)));
        d.hga[i] = u;
        if (dg <= 0.0f) {
            d.hgd[i] = 0.0f;
            d.hgi[i] = 0.0f;
            return;
        }
        const float2 lo = unpack(u.x), hi = unpack(u.y);
        const float c32 = ((m & 1) ? a.x : 0.0f) + ((m & 2) ? a.y : 0.0f) + ((m & 4) ? a.z : 0.0f) + ((m & 8) ? a.w : 0.0f);
        const float c16 = ((m & 1) ? lo.x : 0.0f) + ((m & 2) ? lo.y : 0.0f) + ((m & 4) ? hi.x : 0.0f) + ((m & 8) ? hi.y : 0.0f);
        const float D = (dg - c32) + c16;
        d.hgd[i] = D;
        d.hgi[i] = D > 0.0f ? 1.0f / D : 0.0f;
    }
    // the vectors stay FP32 on every level: rounding them would make the V-cycle a
    // nonlinear operator, which conjugate gradients does not tolerate (it stagnates near the
    // rounding level); the matrices are fixed during a solve, so the V-cycle built on their
    // BF16 copies stays a linear, symmetric positive definite preconditioner
    DEV static acc4* part(const DevScene& d) { return d.partials; }
    DEV static acc4 zero4() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
    DEV static acc4 prod4(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
        return make_float4(a0 * b0, a1 * b1, a2 * b2, a3 * b3);
    }
    DEV static Dbl4 fin(acc4 a) { return Dbl4{(double)a.x, (double)a.y, (double)a.z, (double)a.w}; }
    using Row = uint2;
    // the smoothers read the inverse diagonal (positive exactly where the diagonal is) and
    // multiply by it instead of dividing: a V-cycle is a preconditioner here, not the
    // reference's arithmetic
    using Diag = float;
    DEV static const Row* rows(const DevScene& d) { return d.hga; }
    DEV static const Diag* diags(const DevScene& d) { return d.hgi; }
    DEV static float4 wide(const Row& u) {
        const float2 a = unpack(u.x), b = unpack(u.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    DEV static Diag no_diag() { return 0.0f; }
    DEV static bool unk(const Diag& y) { return y > 0.0f; }
    DEV static float4 pack_red(float2 r, const Diag& y) { return make_float4(r.x, r.y, y, 0.0f); }
    DEV static void unpack_red(const float4& v, float2& r, Diag& y) {
        r = make_float2(v.x, v.y);
        y = v.z;
    }
    DEV static float2 quot(float2 a, const Diag& y) { return make_float2(a.x * y, a.y * y); }
    DEV static bool ok(float2, const Diag&) { return true; }
    DEV static float2 quot_ieee(float2 a, const Diag&) { return a; }   // (never taken)
    DEV static Diag spoilt(const Diag& y) { return y; }
};

template <class T>
struct Solve {
    T rz[2], alpha[2], beta[2], bb[2], rr[2];
    T rmark;   // mixed precision: the pressure column's r.r at the last residual check
    uint32_t done[2], iters[2];
    uint32_t bad;   // a total was not finite: the solve stopped (SolveState ERR_DIVERGED)
    uint32_t replaced;   // residual replacements in this solve
    uint32_t floor_hit;  // a check found the carried residual near the FP32 rounding floor
    uint32_t adopt;      // a batch: this iteration's check adopts the true residual
};

template <class A4>
DEV bool finite4(const A4& a) { return isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && isfinite(a.w); }

// ---- setup phases ---------------------------------------------------------------------

// Unknowns of the CG operator.
DEV bool unknown_op(const DevScene& d, const Lv& L, int x, int y) { return l_inside(L, x, y) && d.mgd[l_at(L, x, y)] > 0.0f; }

// cg_scale.comp on level-0 tile t: warm start from last substep's potential rescaled to
// this substep. Also level 0's diagonal with its reciprocal, or (mixed) its matrix in BF16, for
// the V-cycle (every cell: rhs.comp rewrote them all).
template <class M>
DEV void cg_scale_tile(const DevScene& d, int t, int mode) {
    const Lv F = lev(d.lv, 0);
    const float ratio = d.S->dt / d.S->dt_prev;
    const int cx = (t % tiles_x(F)) * 16 + (threadIdx.x & 15), cy = (t / tiles_x(F)) * 16 + (threadIdx.x >> 4);
    if (!l_inside(F, cx, cy)) return;
    const int i = l_at(F, cx, cy);
    const uint32_t active = d.ptile[F.toff + t];
    const float2 pres = d.pres[i];   // (with the rest, before any is used)
    if (M::kMixed) {
        int m = 0;
        for (int q = 0; q < 4; q++) m |= unknown_op(d, F, cx + NBX[q], cy + NBY[q]) ? (1 << q) : 0;
        Mixed::setA(d, i, d.mga[i], d.mgd[i], m);
    } else {
        d.mgy[i] = make_float2(d.mgd[i], recip_row(d.mgd[i], d.mga[i]));
    }
    if (active == 0u) return;
    if (d.mgd[i] > 0.0f) {
        float p = pres.x;
        if (mode == 1) p -= d.p2keep[i];
        else d.p2keep[i] = 0.0f;
        d.pres[i].x = p * ratio;
    } else {
        d.pres[i] = make_float2(0.0f, 0.0f);
    }
}

// mg_build.comp's aggregation: a coarse cell's diagonal D and couplings A from its four fine cells
// and their neighbours. dg(x, y), x and y from -1 to 2: the fine cell's diagonal, 0 where there is
// no unknown; row(x, y): its couplings. Everything is loaded before any of it is used: a load at a
// time behind its neighbour's test was 24 latencies in a row.
template <class Dg, class Row>
DEV void galerkin(Dg&& dg, Row&& row, float& D, float4& A) {
    float c[2][2], l[2], r[2], b[2], t[2];
    float4 w[2][2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        l[k] = dg(-1, k);
        r[k] = dg(2, k);
        b[k] = dg(k, -1);
        t[k] = dg(k, 2);
#pragma unroll
        for (int x = 0; x < 2; x++) {
            c[k][x] = dg(x, k);
            w[k][x] = row(x, k);
        }
    }
    D = 0.0f;
    A = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int y = 0; y < 2; y++)
#pragma unroll
        for (int x = 0; x < 2; x++) {
            if (!(c[y][x] > 0.0f)) continue;
            const float4 v = w[y][x];
            D += c[y][x];
            if (x == 1) { if (c[y][0] > 0.0f) D -= v.x; }
            else if (l[y] > 0.0f) A.x += v.x;
            if (x == 0) { if (c[y][1] > 0.0f) D -= v.y; }
            else if (r[y] > 0.0f) A.y += v.y;
            if (y == 1) { if (c[0][x] > 0.0f) D -= v.z; }
            else if (b[x] > 0.0f) A.z += v.z;
            if (y == 0) { if (c[1][x] > 0.0f) D -= v.w; }
            else if (t[x] > 0.0f) A.w += v.w;
        }
    if (!(D > 1e-7f)) {
        D = 0.0f;
        A = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// mg_build.comp on tile t of coarse level l + 1, from level l. One tile is two latencies, its flags'
// and its cells' (galerkin); the three levels of a 384 x 216 tank took 6, 6 and 5 us, 2.9, 2.3 and 2.1 now.
// A tile without unknowns is cleared when its flag falls, or when the flags are the other precision's:
// that one's builds did not clear this hierarchy.
template <class M>
DEV void mg_build_tile(const DevScene& d, int l, int t) {
    const Lv F = lev(d.lv, l), C = lev(d.lv, l + 1);
    const int tfx = tiles_x(F), tfy = tiles_y(F), tcx = tiles_x(C);
    const int ty = qdiv(t, C.tm), tx = t - ty * tcx;
    const uint32_t slot = (uint32_t)C.toff + (uint32_t)t;
    const uint32_t was = d.ptile[slot] | (d.K->hier != M::kHier ? 1u : 0u);
    uint32_t on = 0u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int fx = 2 * tx + (k & 1), fy = 2 * ty + (k >> 1);
        if (fx < tfx && fy < tfy) on |= d.ptile[F.toff + fy * tfx + fx];
    }
    __syncthreads();   // every thread has read what the first one writes
    if (threadIdx.x == 0) d.ptile[slot] = on != 0u ? 1u : 0u;
    const int Cx = tx * 16 + (threadIdx.x & 15), Cy = ty * 16 + (threadIdx.x >> 4);
    if ((on | was) == 0u || Cx >= C.w || Cy >= C.h) return;
    const int o = l_at(C, Cx, Cy);
    float D = 0.0f;
    float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (on != 0u)
        galerkin(
            [&](int x, int y) {
                x += 2 * Cx;
                y += 2 * Cy;
                return l_inside(F, x, y) ? M::Dg(d, l_at(F, x, y)) : 0.0f;
            },
            [&](int x, int y) {
                x += 2 * Cx;
                y += 2 * Cy;
                return l_inside(F, x, y) ? M::A(d, l_at(F, x, y)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            },
            D, A);
    M::setA(d, o, A, D);
}

// cg_init.comp over this block's `count` active level-0 tiles (at(k, t): the k-th's scene, its tile
// in t): r = b - A x (the FP32 operator) and the tile's sum of b.b in the partials' second half. A
// cell's loads are all issued before the first is used, and one warp adds up a tile's products
// while the others go on to the next, in the other of two buffers at sums. A load at a time behind
// its neighbour's test, and a tree of the whole block, the phase (beside it a few blocks set up
// their tails) took 29 us at 1600 x 900, 20 now.
template <class M, class At>
DEV void residual_pass(int count, float4* sums, At&& at) {
    static_assert(std::is_same<typename M::acc4, float4>::value, "the products are float4");
    for (int k = 0; k < count; k++) {
        int t;
        const DevScene& d = at(k, t);
        const Lv F = lev(d.lv, 0);
        const int2 og = tile_origin(F, t);
        const int cx = og.x + (threadIdx.x & 15), cy = og.y + (threadIdx.x >> 4);
        float4 a4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (l_inside(F, cx, cy)) {
            const int i = l_at(F, cx, cy);
            const float D = d.mgd[i];
            const float4 w = d.mga[i], b = d.prhs[i];
            const float2 x = d.pres[i];
            float nd[4];
            float2 np[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int nx = cx + NBX[q], ny = cy + NBY[q];
                const bool in = l_inside(F, nx, ny);
                const int j = in ? l_at(F, nx, ny) : i;
                nd[q] = in ? d.mgd[j] : 0.0f;
                np[q] = d.pres[j];
            }
            float2 r = make_float2(0.0f, 0.0f);
            if (D > 0.0f) {
                float axx = D * x.x, axy = D * x.y;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (nd[q] > 0.0f) {
                        const float wd = wcomp(w, q);
                        axx -= wd * np[q].x;
                        axy -= wd * np[q].y;
                    }
                r = make_float2(b.x - axx, b.y - axy);
                a4 = M::prod4(b.x, b.x, b.y, b.y, 0.0f, 0.0f, 0.0f, 0.0f);
            }
            d.mgr[i] = r;
        }
        float4* const buf = sums + (k & 1) * NT;
        buf[threadIdx.x] = a4;
        __syncthreads();
        if (threadIdx.x >= 7 * 32) {
            const float4 v = warp_tree(buf);
            if (threadIdx.x == 7 * 32) M::part(d)[d.nwg + t] = v;
        }
    }
    __syncthreads();
}

// Tiles of level l of one scene.
DEV int level_tiles(const DevScene& d, int l) {
    const Lv L = lev(d.lv, l);
    return tiles_x(L) * tiles_y(L);
}

// ---- the V-cycle --------------------------------------------------------------------------

// The tail levels' state in each block's shared memory (dynamic, FP32 in both precisions). A
// level's unknowns are listed by colour, the even cells first: entry p of the list holds the
// cell's row (couplings, zero towards cells that are no unknowns; diagonal and reciprocal), its
// slot, its right-hand side and the entries of its four cells of the level above, so that a
// thread finds all of these from its own number alone; the iterates lie by slot (the cells'
// offsets from the first tail level, the slots of mg_tail.comp), where neighbours are at fixed
// distances. Slots that are no unknown hold zero.
struct TailLevel {
    int o, n, w, h;     // its cells are slots o .. o + n - 1
    uint32_t wm;        // division constant of the width
    int n0, n1, pad;    // unknowns with (x + y) even (entries o ..) and odd (entries o + n0 ..)
};
constexpr int kTailLevels = 16;
constexpr uint32_t kNoEntry = 0xffffu;
struct Tail {
    float4* a;
    float2* dy;
    float2* x;       // (of the first level: read by the way up above the tail)
    float2* r;
    TailLevel* lv;
    uint16_t* slot;  // an entry's slot
    uint16_t* kid;   // of a coarser level's entry p: the four entries at 4 (p - nf) (kNoEntry: no unknown)
    int base, T, nf, nl;
};

// A tail of T cells, the first nf of them its first level's, in nl levels, laid out in shared
// memory at smem; its right-hand sides, live only inside the tail phase, at r.
DEV Tail tail_at(unsigned char* smem, float2* r, int base, int T, int nf, int nl) {
    Tail tl;
    tl.base = base;
    tl.T = T;
    tl.nf = nf;
    tl.nl = nl;
    tl.a = reinterpret_cast<float4*>(smem);
    tl.lv = reinterpret_cast<TailLevel*>(tl.a + T);
    tl.dy = reinterpret_cast<float2*>(tl.lv + kTailLevels);
    tl.x = tl.dy + T;
    tl.r = r;
    tl.slot = reinterpret_cast<uint16_t*>(tl.x + T);
    tl.kid = tl.slot + T;
    return tl;
}

// The persistent kernels' dynamic shared memory: the level passes' exchange of cell values
// (TileSmem), and one scene's tail. While no tile is being computed its bytes hold the tail's
// right-hand sides (the tail phase) or the block's tree buffer (the totals, the refinement's checks
// and the closing residual).
//
// With every array of its own a block took 119.5 KB at 1600 x 900 (a tail of 50 x 29 and coarser
// cells), of which an SM holds one, and 304 blocks became 152; sharing the stages' bytes it is 112 KB
// there and at most 115 with any tail of up to 2050 cells, two an SM. (A tail has more only on a grid
// several times as long as it is wide.) A substep of the 1600 x 900 dam 1.303 -> 1.249 ms, of the mixed
// pour on 701 x 397 2.69 -> 2.58; 8 tanks of 400 x 225 in a mixed batch 1.324 -> 1.225 (plain 1.177 ->
// 1.102). A tank with few active tiles does not need the second block: a quarter-full dam of 800 x 450
// takes 0.695 ms with it and 0.685 without, a full pour there 3.0 and 3.1.
constexpr size_t kStageBytes = 17200;
struct TileSmem {
    unsigned char stage[2][kStageBytes];   // two tiles' fields, staged asynchronously (LevelStage, ApplyStage)
    float4 red[200];         // per red slot of a way down: its right-hand side, diagonal and reciprocal
    float2 black[200];       // per black slot: its new value
};
constexpr size_t kTileBytes = sizeof(TileSmem);
static_assert(kTileBytes % 16 == 0, "the tail follows");
static_assert(kTileBytes >= 3000 * sizeof(float2), "the tail's right-hand sides fit (a tail has fewer than 3000 cells)");
extern __shared__ __align__(16) unsigned char dyn_smem[];
DEV Tail make_tail(const DevScene& d) {
    const Lv F = lev(d.lv, d.lv.tail), E = lev(d.lv, d.lv.n - 1);
    return tail_at(dyn_smem + kTileBytes, reinterpret_cast<float2*>(dyn_smem), F.off, E.off + E.w * E.h - F.off, F.w * F.h,
                   d.lv.n - d.lv.tail);
}

// Cells of the tail levels, and the tail's bytes without its right-hand sides.
__host__ __device__ inline int tail_cells(const Levels& lv) { return lv.off[lv.n - 1] + lv.w[lv.n - 1] * lv.h[lv.n - 1] - lv.off[lv.tail]; }
__host__ __device__ inline size_t tail_bytes(int T, int nf) {
    return (kTailLevels * sizeof(TailLevel) + (size_t)T * (sizeof(float4) + 2 * sizeof(float2) + sizeof(uint16_t)) +
            (size_t)(T - nf) * 4 * sizeof(uint16_t) + 15) / 16 * 16;
}

// The lists of the tail's unknowns by colour, of its first level or of all the others at once (a
// pass has the latency of a chain of shared accesses, a level at a time that was paid per level).
// An entry's place among its colour does not matter to a half-sweep: the first level's warps
// count their cells and add once for each colour (an add a cell waited for its turn). The
// couplings and diagonals so far lie by slot, so they move through registers.
template <bool FIRST>
DEV void tail_lists(const Tail& tl, uint16_t* ent) {
    constexpr int PER = 6;   // the first level has at most 1500 cells, the others together fewer than that
    const int s0 = FIRST ? 0 : tl.nf, s1 = FIRST ? tl.nf : tl.T;
    // a cell's place among its colour, from the list's end if odd, under its level and the mask of
    // its neighbours that are unknowns; none: no unknown
    constexpr uint32_t kNone = 0xffffffffu, kOdd = 0x8000u;
    uint32_t p[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int s = s0 + (int)threadIdx.x + j * NT;
        p[j] = kNone;
        int l = 0;
        bool odd = false;
        if (s < s1) {
            if (!FIRST) {
                l = 1;
                while (l + 1 < tl.nl && s >= tl.lv[l + 1].o) l++;
            }
            const TailLevel& Q = tl.lv[l];
            const int t = s - Q.o, y = qdiv(t, Q.wm), x = t - y * Q.w;
            odd = (x + y) & 1;
            const uint32_t m = (x > 0 && tl.dy[s - 1].x > 0.0f ? 1u : 0u) | (x + 1 < Q.w && tl.dy[s + 1].x > 0.0f ? 2u : 0u) |
                               (y > 0 && tl.dy[s - Q.w].x > 0.0f ? 4u : 0u) | (y + 1 < Q.h && tl.dy[s + Q.w].x > 0.0f ? 8u : 0u);
            if (tl.dy[s].x > 0.0f) p[j] = (uint32_t)l << 20 | m << 16;
            tl.x[s] = make_float2(0.0f, 0.0f);
        }
        const bool on = p[j] != kNone;
        TailLevel& Q = tl.lv[l];
        if (FIRST) {
            const uint32_t even_m = __ballot_sync(0xffffffffu, on && !odd), odd_m = __ballot_sync(0xffffffffu, on && odd);
            const int lane = threadIdx.x & 31;
            int e = 0, o = 0;
            if (lane == 0) {
                if (even_m) e = atomicAdd(&Q.n0, __popc(even_m));
                if (odd_m) o = atomicAdd(&Q.n1, __popc(odd_m));
            }
            e = __shfl_sync(0xffffffffu, e, 0);
            o = __shfl_sync(0xffffffffu, o, 0);
            const uint32_t before = (1u << lane) - 1u;
            if (on) p[j] |= odd ? kOdd | (uint32_t)(o + __popc(odd_m & before)) : (uint32_t)(e + __popc(even_m & before));
        } else if (on) {
            p[j] |= odd ? kOdd | (uint32_t)atomicAdd(&Q.n1, 1) : (uint32_t)atomicAdd(&Q.n0, 1);
        }
    }
    float4 a[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (p[j] == kNone) continue;
        a[j] = tl.a[s0 + (int)threadIdx.x + j * NT];
        if (!(p[j] & 1u << 16)) a[j].x = 0.0f;
        if (!(p[j] & 2u << 16)) a[j].y = 0.0f;
        if (!(p[j] & 4u << 16)) a[j].z = 0.0f;
        if (!(p[j] & 8u << 16)) a[j].w = 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; j++) {   // the entry: the odd cells follow the even ones
        const int s = s0 + (int)threadIdx.x + j * NT;
        if (p[j] == kNone) {
            if (s < s1) ent[s] = (uint16_t)kNoEntry;
            continue;
        }
        const TailLevel& Q = tl.lv[p[j] >> 20];
        const uint32_t k = p[j] & (kOdd - 1u);
        const uint32_t e = (uint32_t)Q.o + ((p[j] & kOdd) ? (uint32_t)(Q.n0 + Q.n1) - 1u - k : k);
        p[j] = e;
        tl.a[e] = a[j];
        tl.slot[e] = (uint16_t)s;
        ent[s] = (uint16_t)e;
    }
    float2 dy[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (p[j] == kNone) continue;
        const float D = tl.dy[s0 + (int)threadIdx.x + j * NT].x;
        dy[j] = make_float2(D, recip(D));
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; j++)
        if (p[j] != kNone) tl.dy[p[j]] = dy[j];
}

// mg_tail.comp mode 1 in every block's shared memory, once per solve: the first tail
// level's matrix from global memory, then the Galerkin matrices of the coarser tail levels
// (the arithmetic of mg_build.comp). Block 0 also stores them for inspection.
template <class M>
DEV void tail_setup(const DevScene& d, const Tail& tl, bool writer) {
    if (threadIdx.x < (uint32_t)tl.nl) {
        const Lv L = lev(d.lv, d.lv.tail + threadIdx.x);
        tl.lv[threadIdx.x] = TailLevel{L.off - tl.base, L.w * L.h, L.w, L.h, L.wm, 0, 0, 0};
    }
    for (int s = threadIdx.x; s < tl.nf; s += NT) {
        tl.a[s] = M::A(d, tl.base + s);
        tl.dy[s].x = M::Dg(d, tl.base + s);
    }
    __syncthreads();
    for (int l = d.lv.tail; l < d.lv.n - 1; l++) {
        Lv F = lev(d.lv, l), C = lev(d.lv, l + 1);
        const int o = F.off - tl.base, oc = C.off - tl.base;
        for (int t = threadIdx.x; t < C.w * C.h; t += NT) {
            const int ccy = qdiv(t, C.wm), ccx = t - ccy * C.w;
            float D;
            float4 A;
            galerkin(
                [&](int x, int y) {
                    x += 2 * ccx;
                    y += 2 * ccy;
                    return l_inside(F, x, y) ? tl.dy[o + y * F.w + x].x : 0.0f;
                },
                [&](int x, int y) {
                    x += 2 * ccx;
                    y += 2 * ccy;
                    return l_inside(F, x, y) ? tl.a[o + y * F.w + x] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                },
                D, A);
            tl.dy[oc + t].x = D;
            tl.a[oc + t] = A;
            if (writer) M::setA(d, C.off + t, A, D);
        }
        __syncthreads();
    }
    // the lists; ent: a slot's entry, kept where the right-hand sides will be
    uint16_t* const ent = reinterpret_cast<uint16_t*>(tl.r);
    tail_lists<true>(tl, ent);
    tail_lists<false>(tl, ent);
    __syncthreads();
    for (int l = 1; l < tl.nl; l++) {
        const TailLevel F = tl.lv[l - 1], C = tl.lv[l];
        for (int t = threadIdx.x; t < 4 * (C.n0 + C.n1); t += NT) {
            const int p = C.o + (t >> 2), c = tl.slot[p] - C.o, cy = qdiv(c, C.wm), cx = c - cy * C.w;
            const int x = 2 * cx + (t & 1), y = 2 * cy + ((t >> 1) & 1);
            tl.kid[4 * (p - tl.nf) + (t & 3)] = x < F.w && y < F.h ? ent[F.o + y * F.w + x] : (uint16_t)kNoEntry;
        }
    }
    __syncthreads();
}
// ... of a batch's scene, called: inlined at both of the batch's places it took the registers of the
// passes around them
template <class M>
__device__ __noinline__ void tail_setup_of(const DevScene* d) { tail_setup<M>(*d, make_tail(*d), false); }

// ---- the level passes ---------------------------------------------------------------------------
//
// A block takes a 16 x 16 tile at a time, a thread per cell: warps 0-3 its black cells, warps
// 4-7 its red ones, so that no warp mixes the two colours' formulas. What a smoothing pass
// needs around the tile comes with it: the 32 black cells just outside it that its red border
// cells touch are computed here too (warp 4), and the 66 red cells around those are read by
// warps 5-7. A thread stages its own cell's fields one tile ahead by asynchronous copies into
// slots only it reads (cp.async: waiting for a register load would also wait for the later ones
// that share one of a warp's few scoreboards); what neighbours need goes through shared memory
// by colour, each colour's slots contiguous (slot row ly + 2 of ten, column (lx + 2) / 2), so
// that a warp's accesses do not conflict. Two block barriers a tile.
//
// A pass is bound by the latency of its steps, not by bytes (L2 carries 16 % of its peak): what
// counts is how few instructions stand between a tile's arrival and its results, and that none
// of them waits for memory. Against the pass this replaced (every thread staging and
// reading up to 400 slots, ten IEEE divisions inlined per black cell, 250 KB of code in the
// loop), per iteration of the 1024 x 576 full-physics pour, 7.6 tiles a block: way down on
// level 0 18.5 -> 12.8 us, way up 15.4 -> 10.1, apply 11.4 -> 8.2, a coarse level with one tile a
// block 2.3-3.0 -> 1.7-2.0. Tried and slower: ten lanes of a warp marching up a tile without
// block barriers (too few warps to hide its ~1000 instructions a row pair: 19 / 12 / 13 us).
//
// A quotient whose operands left the fast form's range is taken again by its thread with the IEEE
// division, where it stands: few threads do, but in a tank with spray some do in most phases (small
// drops converge to residuals below the range long before the rest). With the block's whole pass
// taken again instead, a batch of 64 uneven dam breaks took 24 to 26.6 ms a substep once 0.3 % of its
// tiles held such a drop, 18.8 to 19.8 now (18 to 18.8 without one); a 384 x 216 dam 0.68 and 0.48.
//
// The values are those of the shaders' work groups, term by term in their order. A neighbour
// that is no unknown is a term less there; here its value is -0 (or, where the term is
// subtracted, +0), which adds nothing to any sum.
constexpr int SP = 10;   // slots of a row
DEV int slot_of(int lx, int ly) { return (ly + 2) * SP + ((lx + 2) >> 1); }
// The 32 black cells just outside a tile that its red border cells touch: (-1, 2j), (16, 2j + 1),
// (2j, -1), (2j + 1, 16).
DEV int2 ring_black(int r) {
    const int j = r & 7;
    switch (r >> 3) {
        case 0: return make_int2(-1, 2 * j);
        case 1: return make_int2(16, 2 * j + 1);
        case 2: return make_int2(2 * j, -1);
        default: return make_int2(2 * j + 1, 16);
    }
}
// The 66 red cells around the tile that those and the tile's black cells touch: 32 beside it,
// 32 one further out, two corners.
DEV int2 ring_red(int r) {
    const int j = r & 7;
    switch (r >> 3) {
        case 0: return make_int2(-1, 2 * j + 1);
        case 1: return make_int2(16, 2 * j);
        case 2: return make_int2(2 * j + 1, -1);
        case 3: return make_int2(2 * j, 16);
        case 4: return make_int2(-2, 2 * j);
        case 5: return make_int2(17, 2 * j + 1);
        case 6: return make_int2(2 * j, -2);
        case 7: return make_int2(2 * j + 1, 17);
        default: return j == 0 ? make_int2(-1, -1) : make_int2(16, 16);
    }
}
// A thread's cell of the tile and its slot (left neighbour's slot: s - e, right: s - e + 1,
// below: s - SP, above: s + SP), and its cell of the ring: kind 1 black, 2 red, 0 none.
struct Geo {
    int lx, ly, s, e;
    int ex, ey, es, ee, kind;
    bool red;
};
DEV Geo geo() {   // (once per kernel: the passes take it)
    Geo g;
    const int t = threadIdx.x, u = t & 127;
    g.red = t >= 128;
    g.ly = u >> 3;
    g.lx = 2 * (u & 7) + ((g.ly & 1) ^ (g.red ? 0 : 1));
    g.s = slot_of(g.lx, g.ly);
    g.e = 1 - (g.lx & 1);
    g.kind = t < 128 ? 0 : t < 160 ? 1 : t < 226 ? 2 : 0;
    const int2 c = g.kind == 1 ? ring_black(t - 128) : g.kind == 2 ? ring_red(t - 160) : make_int2(0, 0);
    g.ex = c.x;
    g.ey = c.y;
    g.es = slot_of(c.x, c.y);
    g.ee = 1 - (c.x & 1);
    return g;
}

DEV float2 f2sel(bool c, float2 a, float z) { return make_float2(c ? a.x : z, c ? a.y : z); }
DEV float2 mul2(float w, float2 v) { return make_float2(w * v.x, w * v.y); }
// r + t0 + t1 + t2 + t3 (left, right, below, above)
DEV float2 sum4(float2 r, float2 t0, float2 t1, float2 t2, float2 t3) {
    float2 s = r;
    s.x += t0.x; s.y += t0.y;
    s.x += t1.x; s.y += t1.y;
    s.x += t2.x; s.y += t2.y;
    s.x += t3.x; s.y += t3.y;
    return s;
}

// The tree of reduce.glsl:5-14 over a tile's 256 products (a cell's at the number of the thread that
// has it in the smoothing passes: product_of), by one warp: the tree's row steps of a column by its
// two lanes, then the column steps by shuffles; the sum comes out in lane 0.
DEV int product_of(int lx, int ly) { return ((lx + ly) & 1 ? 0 : 128) + ly * 8 + (lx >> 1); }
DEV float2 tile_tree(const float2* prod) {
    const int x = threadIdx.x & 15, h = (threadIdx.x >> 4) & 1;
    const float2* const v = prod + product_of(x, h) - h * 8;   // (rows of one parity: one colour a lane)
    auto b = [&](int j) {
        const float2 v0 = v[j * 8], v1 = v[(j + 4) * 8], v2 = v[(j + 8) * 8], v3 = v[(j + 12) * 8];
        return make_float2((v0.x + v2.x) + (v1.x + v3.x), (v0.y + v2.y) + (v1.y + v3.y));
    };
    const float2 b0 = b(h), b1 = b(h + 2);
    float2 s = make_float2(b0.x + b1.x, b0.y + b1.y);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
        s.x += __shfl_down_sync(0xffffffffu, s.x, k);
        s.y += __shfl_down_sync(0xffffffffu, s.y, k);
    }
    return s;
}
constexpr int kTreeWarp = 7;

// A tile's fields as they are staged: thread t's own cell in entry t, its cell of the ring in
// entry t - 128 of the e arrays. On level 0 p's entries take the products of the tile's sums once
// the way down has read its direction there (the way up stages nothing in them).
template <class M>
struct LevelStage {
    typename M::Row a[NT], ea[32];
    float2 r[NT], er[98], q[NT], eq[98], p[NT], x[NT];
    typename M::Diag y[NT], ey[98];
};
static_assert(sizeof(LevelStage<Plain>) == kStageBytes && sizeof(LevelStage<Mixed>) <= kStageBytes, "two tiles' fields");
struct ApplyStage {
    float4 a[NT];
    float2 z[NT], o[NT], ez[64], eo[64];
    float D[NT], eD[64];
};

// A tile of a level of a scene as a pass works on it.
struct DownArgs {
    const float2 *r, *q;   // the right-hand side; on level 0 fused with cg_update.comp, A p (else null)
    float ax, ay;          // ... and its step lengths,
    const float2* p;       // the directions,
    float2* r_out;         // and where the updated residual goes
};
struct DownTile {
    int scene;
    Lv F, C;
    int t;
    DownArgs a;
};

// mg_down.comp on this block's tiles of a level (at(k): its k-th, first and next(k): the indices it
// takes): red-black Gauss-Seidel from zero, the residual summed over 2 x 2 cells into the next
// level. On level 0 (top) also the tile's sums of r.r into part[tile].zw (the way up adds those
// of r.z) and, where q is set, x += alpha p, r -= alpha q (a cell that is no unknown has p = 0,
// and what its r holds is never used).
template <class M, class Of, class At, class Next>
DEV void down_pass(const Geo& g, int count, bool top, Of&& of, At&& at, Next&& next) {
    TileSmem& S = *reinterpret_cast<TileSmem*>(dyn_smem);
    const int t = threadIdx.x;
    using Stage = LevelStage<M>;
    auto fetch = [&](const DownTile& T, Stage& n) {
        const DevScene& d = of(T.scene);
        const int2 og = tile_origin(T.F, T.t);
        const int x = og.x + g.lx, y = og.y + g.ly;
        const bool in = x < T.F.w && y < T.F.h;
        const int i = in ? l_at(T.F, x, y) : 0;
        cp_async<sizeof(typename M::Row)>(&n.a[t], M::rows(d) + i, in);
        cp_async<sizeof(typename M::Diag)>(&n.y[t], M::diags(d) + i, in);
        cp_async<8>(&n.r[t], T.a.r + i, in);
        if (T.a.q) {
            cp_async<8>(&n.q[t], T.a.q + i, in);
            cp_async<8>(&n.p[t], T.a.p + i, in);
            cp_async<8>(&n.x[t], d.pres + i, in);
        }
        if (g.kind != 0) {
            const int ex = og.x + g.ex, ey = og.y + g.ey;
            const bool ein = l_inside(T.F, ex, ey);
            const int e = ein ? l_at(T.F, ex, ey) : 0;
            cp_async<sizeof(typename M::Diag)>(&n.ey[t - 128], M::diags(d) + e, ein);
            cp_async<8>(&n.er[t - 128], T.a.r + e, ein);
            if (T.a.q) cp_async<8>(&n.eq[t - 128], T.a.q + e, ein);
            if (g.kind == 1) cp_async<sizeof(typename M::Row)>(&n.ea[t - 128], M::rows(d) + e, ein);
        }
    };
    auto stage = [](int turn) -> Stage& { return *reinterpret_cast<Stage*>(dyn_smem + (turn & 1) * sizeof(TileSmem::stage) / 2); };
    int k = next(0);
    if (k >= count) return;
    DownTile T = at(k);
    fetch(T, stage(0));
    cp_commit();
    for (int turn = 0;; turn++) {
        const DownTile cur = T;
        k = next(k + 1);
        const bool more = k < count;
        if (more) {
            T = at(k);
            fetch(T, stage(turn + 1));
        }
        cp_commit();
        cp_wait<1>();
        Stage& n = stage(turn);
        const int2 og = tile_origin(cur.F, cur.t);
        const bool fused = cur.a.q != nullptr, in = og.x + g.lx < cur.F.w && og.y + g.ly < cur.F.h;
        const int i = l_at(cur.F, og.x + g.lx, og.y + g.ly);
        const typename M::Diag y = n.y[t];
        typename M::Diag ey = M::no_diag();
        float2 r = n.r[t], er = make_float2(0.0f, 0.0f);
        if (fused) {
            const float2 q = n.q[t], p = n.p[t], x = n.x[t];
            r.x = r.x - cur.a.ax * q.x;
            r.y = r.y - cur.a.ay * q.y;
            if (in) {
                of(cur.scene).pres[i] = make_float2(x.x + cur.a.ax * p.x, x.y + cur.a.ay * p.y);
                cur.a.r_out[i] = r;
            }
        }
        if (g.kind != 0) {
            ey = n.ey[t - 128];
            er = n.er[t - 128];
            if (fused) {
                const float2 eq = n.eq[t - 128];
                er.x = er.x - cur.a.ax * eq.x;
                er.y = er.y - cur.a.ay * eq.y;
            }
        }
        const bool unk = M::unk(y), eunk = M::unk(ey);
        if (top) n.p[t] = f2sel(unk, make_float2(r.x * r.x, r.y * r.y), 0.0f);
        r = f2sel(unk, r, -0.0f);
        er = f2sel(eunk, er, -0.0f);
        if (g.red) {
            const bool out = unk && !M::ok(r, y);
            float2 z = M::quot(r, y);
            if (__builtin_expect(out, 0)) z = M::quot_ieee(r, y);
            S.red[g.s] = M::pack_red(r, out ? M::spoilt(y) : y);
            if (in) of(cur.scene).mgx[i] = f2sel(unk, z, 0.0f);
            if (g.kind == 2) S.red[g.es] = M::pack_red(er, eunk && !M::ok(er, ey) ? M::spoilt(ey) : ey);
        }
        __syncthreads();
        if (t < 160) {   // the black cells, and warp 4 those of the ring
            const bool own = t < 128;
            const int s = own ? g.s : g.es, e = own ? g.e : g.ee;
            const float4 w = M::wide(own ? n.a[t] : n.ea[t - 128]);
            const typename M::Diag yo = own ? y : ey;
            auto term = [&](float wq, int j) {
                float2 v;
                typename M::Diag yn;
                M::unpack_red(S.red[j], v, yn);
                return M::quot(mul2(wq, v), yn);
            };
            const float2 sum = sum4(own ? r : er, term(w.x, s - e), term(w.y, s - e + 1), term(w.z, s - SP), term(w.w, s + SP));
            const bool u = own ? unk : eunk;
            float2 z = M::quot(sum, yo);
            if (__builtin_expect(u && !M::ok(sum, yo), 0)) {   // (a spoilt neighbour's term is not a number)
                float2 a = own ? r : er;
#pragma unroll 1
                for (int q = 0; q < 4; q++) {
                    float2 v;
                    typename M::Diag yn;
                    M::unpack_red(S.red[q < 2 ? s - e + q : s + (2 * q - 5) * SP], v, yn);
                    v = M::quot_ieee(mul2(wcomp(w, q), v), yn);
                    a.x += v.x;
                    a.y += v.y;
                }
                z = M::quot_ieee(a, yo);
            }
            z = f2sel(u, z, 0.0f);
            S.black[s] = z;
            if (own && in) of(cur.scene).mgx[i] = z;
        } else if (top && t >= 32 * kTreeWarp) {
            const float2 rr = tile_tree(n.p);
            if ((t & 31) == 0) reinterpret_cast<float2*>(M::part(of(cur.scene)) + cur.t)[1] = rr;
        }
        __syncthreads();
        if (g.red) {   // the restriction: a coarse cell's red cells are in lanes l (even row) and l + 8
            const float4 w = M::wide(n.a[t]);
            const float2 t0 = mul2(w.x, S.black[g.s - g.e]), t1 = mul2(w.y, S.black[g.s - g.e + 1]);
            const float2 t2 = mul2(w.z, S.black[g.s - SP]), t3 = mul2(w.w, S.black[g.s + SP]);
            float2 s = f2sel(unk, sum4(make_float2(0.0f, 0.0f), t0, t1, t2, t3), 0.0f);
            s.x = __shfl_up_sync(0xffffffffu, s.x, 8);
            s.y = __shfl_up_sync(0xffffffffu, s.y, 8);
            if (g.ly & 1) {
                const float2 v = sum4(s, t0, t1, t2, t3);
                s = unk ? v : s;
                const int X = (og.x + g.lx) >> 1, Y = (og.y + g.ly) >> 1;
                if (X < cur.C.w && Y < cur.C.h) of(cur.scene).mgr[l_at(cur.C, X, Y)] = s;
            }
        }
        if (!more) break;
    }
}

struct UpTile {
    int scene;
    Lv F, C;
    int t;
    const float2* r;    // the right-hand side
    const float2* zc;   // the coarse level's values in global memory,
    const float2* zs;   // or (else null) this block's copy of the tail in shared memory
};

// mg_up.comp on this block's tiles of a level: the coarse correction with omega and the
// mirrored sweep. On level 0 (top) the tile's sums of r.z into part[tile].xy.
template <class M, class Of, class At, class Next>
DEV void up_pass(const Geo& g, int count, bool top, Of&& of, At&& at, Next&& next) {
    TileSmem& S = *reinterpret_cast<TileSmem*>(dyn_smem);
    float2* const sred = reinterpret_cast<float2*>(S.red);
    const int t = threadIdx.x;
    using Stage = LevelStage<M>;   // (q: the red cells' pre-smoothed values, then their coarse ones; x: the ring's coarse ones)
    auto fetch = [&](const UpTile& T, Stage& n) {
        const DevScene& d = of(T.scene);
        const int2 og = tile_origin(T.F, T.t);
        const int x = og.x + g.lx, y = og.y + g.ly;
        const bool in = x < T.F.w && y < T.F.h;
        const int i = in ? l_at(T.F, x, y) : 0;
        cp_async<sizeof(typename M::Row)>(&n.a[t], M::rows(d) + i, in);
        cp_async<sizeof(typename M::Diag)>(&n.y[t], M::diags(d) + i, in);
        cp_async<8>(&n.r[t], T.r + i, in);
        if (g.red) {
            cp_async<8>(&n.q[t - 128], d.mgx + i, in);
            if (!T.zs) cp_async<8>(&n.q[t], T.zc + (in ? (y >> 1) * T.C.w + (x >> 1) : 0), in);
        }
        if (g.kind != 0) {
            const int ex = og.x + g.ex, ey = og.y + g.ey;
            const bool ein = l_inside(T.F, ex, ey);
            const int e = ein ? l_at(T.F, ex, ey) : 0;
            cp_async<sizeof(typename M::Diag)>(&n.ey[t - 128], M::diags(d) + e, ein);
            if (g.kind == 1) {
                cp_async<sizeof(typename M::Row)>(&n.ea[t - 128], M::rows(d) + e, ein);
                cp_async<8>(&n.er[t - 128], T.r + e, ein);
            } else {
                cp_async<8>(&n.eq[t - 128], d.mgx + e, ein);
                if (!T.zs) cp_async<8>(&n.x[t - 128], T.zc + (ein ? (ey >> 1) * T.C.w + (ex >> 1) : 0), ein);
            }
        }
    };
    // s / D where the cell is an unknown
    auto value = [&](float2 s, const typename M::Diag& y) {
        float2 z = M::quot(s, y);
        if (__builtin_expect(M::unk(y) && !M::ok(s, y), 0)) z = M::quot_ieee(s, y);
        return z;
    };
    auto corrected = [](float2 v, float2 zc) { return make_float2(v.x + MG_OMEGA * zc.x, v.y + MG_OMEGA * zc.y); };
    auto tree = [&](const UpTile& T, const float2* prod) {
        if (t < 32 * kTreeWarp) return;
        const float2 rz = tile_tree(prod);
        if ((t & 31) == 0) reinterpret_cast<float2*>(M::part(of(T.scene)) + T.t)[0] = rz;
    };
    auto stage = [](int turn) -> Stage& { return *reinterpret_cast<Stage*>(dyn_smem + (turn & 1) * sizeof(TileSmem::stage) / 2); };
    int k = next(0);
    if (k >= count) return;
    UpTile T = at(k);
    fetch(T, stage(0));
    cp_commit();
    for (int turn = 0;; turn++) {
        const UpTile cur = T;
        k = next(k + 1);
        const bool more = k < count;
        if (more) {
            T = at(k);
            fetch(T, stage(turn + 1));
        }
        cp_commit();
        cp_wait<1>();
        Stage& n = stage(turn);
        const int2 og = tile_origin(cur.F, cur.t);
        const int X = og.x + g.lx, Y = og.y + g.ly, i = l_at(cur.F, X, Y);
        const bool in = X < cur.F.w && Y < cur.F.h;
        const typename M::Diag y = n.y[t];
        typename M::Diag ey = M::no_diag();
        if (g.kind != 0) ey = n.ey[t - 128];
        const bool unk = M::unk(y), eunk = M::unk(ey);
        const float2 r = n.r[t];
        if (g.red) {
            // (the tail's values are this block's own, in shared memory)
            float2 zc = make_float2(0.0f, 0.0f);
            if (unk) zc = cur.zs ? cur.zs[(Y >> 1) * cur.C.w + (X >> 1)] : n.q[t];
            sred[g.s] = f2sel(unk, corrected(n.q[t - 128], zc), -0.0f);
            if (g.kind == 2) {
                const int EX = og.x + g.ex, EY = og.y + g.ey;
                float2 ez = make_float2(0.0f, 0.0f);
                if (eunk) ez = cur.zs ? cur.zs[(EY >> 1) * cur.C.w + (EX >> 1)] : n.x[t - 128];
                sred[g.es] = f2sel(eunk, corrected(n.eq[t - 128], ez), -0.0f);
            }
        }
        __syncthreads();
        if (t < 160) {   // the black cells, and warp 4 those of the ring
            const bool own = t < 128;
            const int s = own ? g.s : g.es, e = own ? g.e : g.ee;
            const float4 w = M::wide(own ? n.a[t] : n.ea[t - 128]);
            const typename M::Diag yo = own ? y : ey;
            const float2 z = value(sum4(own ? r : n.er[t - 128], mul2(w.x, sred[s - e]), mul2(w.y, sred[s - e + 1]), mul2(w.z, sred[s - SP]),
                                        mul2(w.w, sred[s + SP])), yo);
            const bool u = own ? unk : eunk;
            S.black[s] = f2sel(u, z, -0.0f);
            if (own) {
                if (in) of(cur.scene).mgz[i] = f2sel(u, z, 0.0f);
                if (top) n.p[t] = f2sel(u, make_float2(r.x * z.x, r.y * z.y), 0.0f);
            }
        }
        __syncthreads();
        if (g.red) {
            const float4 w = M::wide(n.a[t]);
            const float2 z = value(sum4(r, mul2(w.x, S.black[g.s - g.e]), mul2(w.y, S.black[g.s - g.e + 1]), mul2(w.z, S.black[g.s - SP]),
                                        mul2(w.w, S.black[g.s + SP])), y);
            if (in) of(cur.scene).mgz[i] = f2sel(unk, z, 0.0f);
            if (top) n.p[t] = f2sel(unk, make_float2(r.x * z.x, r.y * z.y), 0.0f);
        }
        if (top) {
            __syncthreads();
            tree(cur, n.p);
        }
        if (!more) break;
    }
}

// cg_apply.comp on this block's level-0 tiles: p = z + beta p_old, q = A p (the FP32 operator),
// the tile's sum of p.q into part[n + tile].zw. A thread per cell in row order, the 64 cells
// beside the tile read by warps 4 and 5; the directions go through shared memory, two tiles in
// flight, one block barrier a tile.
struct ApplyTile {
    int scene;
    Lv F;
    int t;
    float b0, b1;
    const float2* p_old;
    float2* p_new;
};
template <class M, class Of, class At, class Next>
DEV void apply_pass(int count, Of&& of, At&& at, Next&& next) {
    if (count == 0) return;
    TileSmem& S = *reinterpret_cast<TileSmem*>(dyn_smem);
    constexpr int PW = 18;
    static_assert(PW * PW * sizeof(float2) <= sizeof(S.red), "the directions in the red slots' bytes");
    float2* const P = reinterpret_cast<float2*>(S.red);
    const int t = threadIdx.x, lx = t & 15, ly = t >> 4;
    const int hr = t - 128, hj = t & 15;   // the halo cell of threads 128 .. 191
    const bool halo = t >= 128 && t < 192;
    const int hx = hr < 16 ? -1 : hr < 32 ? 16 : hj, hy = hr < 32 ? hj : hr < 48 ? -1 : 16;
    const int s0 = (ly + 1) * PW + lx + 1, sh = (hy + 1) * PW + hx + 1, sp = product_of(lx, ly);
    using Stage = ApplyStage;
    auto nob = [](const ApplyTile& T) { return T.b0 == 0.0f && T.b1 == 0.0f; };
    auto fetch = [&](const ApplyTile& T, Stage& n) {
        const DevScene& d = of(T.scene);
        const int2 og = tile_origin(T.F, T.t);
        const int x = og.x + lx, y = og.y + ly;
        const bool in = x < T.F.w && y < T.F.h;
        const int i = in ? l_at(T.F, x, y) : 0;
        cp_async<16>(&n.a[t], d.mga + i, in);
        cp_async<4>(&n.D[t], d.mgd + i, in);
        cp_async<8>(&n.z[t], d.mgz + i, in);
        if (!nob(T)) cp_async<8>(&n.o[t], T.p_old + i, in);
        if (halo) {
            const int ex = og.x + hx, ey = og.y + hy;
            const bool ein = l_inside(T.F, ex, ey);
            const int e = ein ? l_at(T.F, ex, ey) : 0;
            cp_async<4>(&n.eD[hr], d.mgd + e, ein);
            cp_async<8>(&n.ez[hr], d.mgz + e, ein);
            if (!nob(T)) cp_async<8>(&n.eo[hr], T.p_old + e, ein);
        }
    };
    auto dir = [&](const ApplyTile& T, float2 z, float2 po, float D) {   // +0 where no unknown
        float2 v = z;
        if (!nob(T)) v = make_float2(T.b0 != 0.0f ? z.x + T.b0 * po.x : z.x, T.b1 != 0.0f ? z.y + T.b1 * po.y : z.y);
        return f2sel(D > 0.0f, v, 0.0f);
    };
    auto stage = [](int slot) -> Stage& { return *reinterpret_cast<Stage*>(dyn_smem + slot * sizeof(Stage)); };
    int slot = 0;   // this tile's stage
    static_assert(3 * sizeof(Stage) + NT * sizeof(float2) <= sizeof(S.stage), "three tiles in flight, and the products");
    float2* const prod = reinterpret_cast<float2*>(dyn_smem + 3 * sizeof(Stage));
    int k = next(0);
    if (k >= count) return;
    ApplyTile T = at(k), T1 = T;
    fetch(T, stage(0));
    cp_commit();
    k = next(k + 1);
    if (k < count) {
        T1 = at(k);
        fetch(T1, stage(1));
    }
    cp_commit();
    for (;;) {
        const ApplyTile cur = T;
        const bool more = k < count;   // (tile T1 is there)
        T = T1;
        if (more) k = next(k + 1);
        if (more && k < count) {
            T1 = at(k);
            fetch(T1, stage(slot == 0 ? 2 : slot - 1));
        }
        cp_commit();
        cp_wait<2>();
        const Stage& n = stage(slot);
        const int2 og = tile_origin(cur.F, cur.t);
        const bool in = og.x + lx < cur.F.w && og.y + ly < cur.F.h;
        const int i = l_at(cur.F, og.x + lx, og.y + ly);
        const float D = n.D[t];
        const float2 p = dir(cur, n.z[t], n.o[t], D);
        P[s0] = p;
        if (halo) P[sh] = dir(cur, n.ez[hr], n.eo[hr], n.eD[hr]);
        __syncthreads();
        const float4 a = n.a[t];
        const float2 l = P[s0 - 1], r = P[s0 + 1], b = P[s0 - PW], u = P[s0 + PW];
        float2 q = make_float2(D * p.x, D * p.y);
        q.x -= a.x * l.x; q.y -= a.x * l.y;
        q.x -= a.y * r.x; q.y -= a.y * r.y;
        q.x -= a.z * b.x; q.y -= a.z * b.y;
        q.x -= a.w * u.x; q.y -= a.w * u.y;
        if (in) {
            cur.p_new[i] = p;
            of(cur.scene).cgq[i] = q;
        }
        prod[sp] = f2sel(D > 0.0f, make_float2(p.x * q.x, p.y * q.y), 0.0f);
        __syncthreads();
        if (t >= 32 * kTreeWarp) {
            const float2 pq = tile_tree(prod);
            if ((t & 31) == 0) reinterpret_cast<float2*>(M::part(of(cur.scene)) + of(cur.scene).nwg + cur.t)[1] = pq;
        }
        if (!more) break;
        slot = slot == 2 ? 0 : slot + 1;
    }
}

// The tail's phases, over J cells a thread at once so that their chains overlap (past the end a
// thread repeats the last one, whose value comes out the same).
//
// A quotient out of the fast form's range is taken the IEEE way after the thread has stored its others
// (a branch before the store lengthened every phase's chain: a solve of 128 x 72 took 2 % longer). What
// the fast form makes of it, which need not be a number, is never stored: a slot past the end of a row
// or of a level is read too, and its zero coupling would not hide one.
//
// A half-sweep over entries p0 .. p0 + cnt - 1 of a level of width w: entry p's sum, and the level's cells
// of one colour from the other's.
DEV float2 tail_sum(const Tail& tl, int p, int s, int w) {
    const float4 a = tl.a[p];
    const float2 x0 = tl.x[max(s - 1, 0)], x1 = tl.x[min(s + 1, tl.T - 1)];
    const float2 x2 = tl.x[max(s - w, 0)], x3 = tl.x[min(s + w, tl.T - 1)];
    return sum4(tl.r[p], mul2(a.x, x0), mul2(a.y, x1), mul2(a.z, x2), mul2(a.w, x3));
}
// The half-sweep's form over J cells a thread: value(p, s) is entry p's sum at slot s.
template <int J, class Value>
DEV void tail_cells_of(const Tail& tl, int p0, int cnt, Value&& value) {
    if ((int)(threadIdx.x & ~31u) < cnt) {
        int s[J];
        float2 z[J];
        bool ok[J], all = true;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const int p = p0 + min((int)threadIdx.x + j * NT, cnt - 1);
            s[j] = tl.slot[p];
            const float2 v = value(p, s[j]), dy = tl.dy[p];
            z[j] = quot2(v, dy);
            ok[j] = quot_ok<80>(v, dy.y);
            all &= ok[j];
        }
#pragma unroll
        for (int j = 0; j < J; j++)
            if (ok[j]) tl.x[s[j]] = z[j];
        if (__builtin_expect(!all, 0)) {   // (a cell's unknown neighbours are the other colour's)
#pragma unroll 1
            for (int j = 0; j < J; j++) {
                const int p = p0 + min((int)threadIdx.x + j * NT, cnt - 1), q = tl.slot[p];
                tl.x[q] = quot2_ieee(value(p, q), tl.dy[p]);
            }
        }
    }
    __syncthreads();
}
template <int J>
DEV void tail_sweep(const Tail& tl, int p0, int cnt, int w) {
    tail_cells_of<J>(tl, p0, cnt, [&](int p, int s) { return tail_sum(tl, p, s, w); });
}
// The black half-sweep of a way up: its neighbours are read with their coarse correction.
template <int J>
DEV void tail_correct(const Tail& tl, const TailLevel& L, const TailLevel& C) {
    tail_cells_of<J>(tl, L.o + L.n0, L.n1, [&](int p, int s) {
        const float4 a = tl.a[p];
        const int k = s - L.o, y = qdiv(k, L.wm), x = k - y * L.w;
        const int m = C.o + (y >> 1) * C.w + (x >> 1);
        auto term = [&](float w, int sn, int c) {
            const float2 xn = tl.x[min(max(sn, 0), tl.T - 1)], xc = tl.x[min(max(c, 0), tl.T - 1)];
            return make_float2(w * (xn.x + MG_OMEGA * xc.x), w * (xn.y + MG_OMEGA * xc.y));
        };
        return sum4(tl.r[p], term(a.x, s - 1, m - 1 + (x & 1)), term(a.y, s + 1, m + (x & 1)),
                    term(a.z, s - L.w, (y & 1) ? m : m - C.w), term(a.w, s + L.w, (y & 1) ? m + C.w : m));
    });
}
// The right-hand side of entry p of a tail level, and its first half-sweep, which starts from
// zero: the level's even unknowns (entries below odd) are r / D. The odd ones are written before
// anything reads them.
DEV void tail_rhs(const Tail& tl, int p, int s, int odd, float2 dy, float2 r, bool on) {
    const float2 x = quot2(r, dy);
    const bool ok = quot_ok<80>(r, dy.y), even = on && p < odd;
    if (on) tl.r[p] = r;
    if (even && ok) tl.x[s] = x;
    if (__builtin_expect(even && !ok, 0)) tl.x[s] = quot2_ieee(r, dy);
}
// The residual of the level above summed over the four cells of each entry of level C (w: the
// width above), four lanes to an entry, one per cell: a cell that is no unknown adds nothing (the
// sum is never -0, so leaving it out or adding +0 is the same).
DEV void tail_restrict(const Tail& tl, const TailLevel& C, int w) {
    const int cnt = 4 * (C.n0 + C.n1), b = threadIdx.x & 28;
#pragma unroll 1
    for (int t = threadIdx.x; (t & ~31) < cnt; t += NT) {
        const int u = min(t, cnt - 4 + (t & 3)), p = C.o + (u >> 2);
        const uint32_t q = tl.kid[4 * (C.o - tl.nf) + u];
        const bool on = q != kNoEntry;
        const int e = on ? (int)q : 0, s = tl.slot[e], cs = tl.slot[p];
        const float4 a = tl.a[e];
        const float2 rh = tl.r[e], cdy = tl.dy[p];
        const float D = tl.dy[e].x;
        const float2 xs = tl.x[s], x0 = tl.x[max(s - 1, 0)], x1 = tl.x[min(s + 1, tl.T - 1)];
        const float2 x2 = tl.x[max(s - w, 0)], x3 = tl.x[min(s + w, tl.T - 1)];
        float2 z = make_float2(D * xs.x, D * xs.y);
        z.x -= a.x * x0.x; z.y -= a.x * x0.y;
        z.x -= a.y * x1.x; z.y -= a.y * x1.y;
        z.x -= a.z * x2.x; z.y -= a.z * x2.y;
        z.x -= a.w * x3.x; z.y -= a.w * x3.y;
        const float ex = on ? rh.x - z.x : 0.0f, ey = on ? rh.y - z.y : 0.0f;
        float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v.x += __shfl_sync(0xffffffffu, ex, b + k);
            v.y += __shfl_sync(0xffffffffu, ey, b + k);
        }
        tail_rhs(tl, p, cs, C.o + C.n0, cdy, v, (t & 3) == 0 && t < cnt);
    }
    __syncthreads();
}

// mg_tail.comp mode 0, computed by EVERY block in its own shared memory: the V-cycle on the
// tail levels, right-hand side R (the first tail level's mgr), result left in tl.x (the first
// tail level's slots). Every block gets the same values; the way up of the level above
// reads them from its own copy, so no grid barrier follows the tail.
//
// It is a chain of ~24 block-wide phases of a few cells each, bound by each phase's latency:
// two dependent shared-memory reads, eight dependent adds and multiplies and a fast quotient, about
// 250 cycles. With the way up of the level above: 12.8 -> 6.4 us (32 x 18 cells, 4 levels),
// 17.9 -> 8.0 us (48 x 27, 6 levels).
constexpr int kTailJ = 3;   // a first tail level has at most 1500 cells, 750 of a colour
DEV void tail_cycle(const float2* R, const Tail& tl) {
    const int last = tl.nl - 1;
    TailLevel L = tl.lv[0];
    {   // (every load in flight before the first is used)
        constexpr int PER = 6;
        const int cnt = L.n0 + L.n1;
        int s[PER];
        float2 v[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
            if ((int)(threadIdx.x & ~31u) + j * NT >= cnt) break;
            s[j] = tl.slot[min((int)threadIdx.x + j * NT, cnt - 1)];
            v[j] = R[s[j]];
        }
#pragma unroll
        for (int j = 0; j < PER; j++) {
            if ((int)(threadIdx.x & ~31u) + j * NT >= cnt) break;
            const int p = min((int)threadIdx.x + j * NT, cnt - 1);
            tail_rhs(tl, p, s[j], L.n0, tl.dy[p], v[j], true);
        }
    }
    __syncthreads();
    // a level's cells of one colour are one a thread unless there are more than a block's threads
    auto sweep = [&](bool odd) {
        const int cnt = odd ? L.n1 : L.n0, p0 = odd ? L.o + L.n0 : L.o;
        if (cnt <= NT) tail_sweep<1>(tl, p0, cnt, L.w);
        else tail_sweep<kTailJ>(tl, p0, cnt, L.w);
    };
    sweep(true);
#pragma unroll 1
    for (int l = 0; l < last; l++) {
        const TailLevel C = tl.lv[l + 1];
        tail_restrict(tl, C, L.w);
        L = C;
        sweep(true);
    }
    // the coarsest level's other seven half-sweeps
#pragma unroll 1
    for (int k = 0; k < 7; k++) sweep(k & 1);
#pragma unroll 1
    for (int l = last - 1; l >= 0; l--) {
        const TailLevel C = L;
        L = tl.lv[l];
        if (L.n1 <= NT) tail_correct<1>(tl, L, C);
        else tail_correct<kTailJ>(tl, L, C);
        sweep(false);
    }
}
// (Z: where the first tail level's result goes, for inspection; a batch's way up reads it)
DEV void phase_tail(const float2* R, float2* Z, const Tail& tl) {
    tail_cycle(R, tl);
    if (Z)
        for (int s = threadIdx.x; s < tl.nf; s += NT) Z[s] = tl.x[s];
}

// The active-tile list of level l (below the tail) of scene d, from ptile (one block).
DEV void build_plist(const DevScene& d, int l) {
    const Lv L = lev(d.lv, l);
    compact_flags(d.ptile + L.toff, tiles_x(L) * tiles_y(L), d.plist + L.toff, d.pcount + l);
}

// Level-0 tiles without unknowns keep zero partial sums through the solve (their tile
// bodies are never run): set them once at its start, every half and precision.
template <class M>
DEV void zero_inactive_tile(const DevScene& d, int t) {
    if (d.ptile[t] != 0u) return;
    const int n = d.nwg;
    M::part(d)[t] = M::zero4();
    M::part(d)[n + t] = M::zero4();
    if (M::kMixed) d.partials64[t] = Dbl4{0.0, 0.0, 0.0, 0.0};
}

// This block's share of the active-tile lists, read once per solve into shared memory:
// entry k of level l is work item blockIdx.x + k x gridDim.x (a tile index; in a batch the
// scene in the high 16 bits), so a phase starts on its tiles without first waiting for
// global memory. Items past kCachePer, or on levels past kCacheLevels, are read as before.
constexpr int kCacheLevels = 8, kCachePer = 32;
struct TileCache {
    uint32_t cnt[kCacheLevels];
    uint32_t item[kCacheLevels][kCachePer];
};
template <class I>
DEV void fill_level(TileCache& tc, int l, uint32_t tiles, I&& item) {
    if (threadIdx.x == 0) tc.cnt[l] = tiles;
    for (int k = threadIdx.x; k < kCachePer; k += NT) {
        const uint32_t j = blockIdx.x + (uint32_t)k * gridDim.x;
        if (j < tiles) tc.item[l][k] = item(j);
    }
}
// how many of a level's tiles this block takes, and the k-th of them
DEV int my_count(uint32_t tiles) { return blockIdx.x < tiles ? (int)((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0; }
template <class I>
DEV uint32_t my_item(const TileCache& tc, int l, int k, I&& item) {
    return (l < kCacheLevels && k < kCachePer) ? tc.item[l][k] : item(blockIdx.x + (uint32_t)k * gridDim.x);
}
struct EveryOne {
    DEV int operator()(int k) const { return k; }
};

DEV uint32_t active_tiles(const DevScene& d, int l, const TileCache& tc) {
    return l < kCacheLevels ? tc.cnt[l] : *(volatile uint32_t*)&d.pcount[l];
}
DEV void fill_cache(const DevScene& d, TileCache& tc) {
    for (int l = 0; l < kCacheLevels && l < d.lv.tail; l++) {
        const uint32_t* list = d.plist + d.lv.toff[l];
        fill_level(tc, l, *(volatile uint32_t*)&d.pcount[l], [&](uint32_t k) { return list[k]; });
    }
    __syncthreads();
}
DEV int my_tile(const DevScene& d, const TileCache& tc, int l, int k) {
    return (int)my_item(tc, l, k, [&](uint32_t j) { return d.plist[d.lv.toff[l] + j]; });
}

// For every active tile of level l of scene d, one at a time by the whole block.
template <class F>
DEV void for_active(const DevScene& d, int l, const TileCache& tc, F&& f) {
    const uint32_t cnt = active_tiles(d, l, tc);
    const uint32_t* list = d.plist + d.lv.toff[l];
    for (uint32_t j = blockIdx.x; j < cnt; j += gridDim.x) f((int)list[j]);
}

// Whether this block computes the tail of scene d: it owns a tile of the level above the tail
// (whose way up reads the tail's result from the block's own copy), or it is block 0.
DEV bool tail_reader(const DevScene& d, const TileCache& tc) {
    return blockIdx.x == 0 || blockIdx.x < active_tiles(d, d.lv.tail - 1, tc);
}

// One V-cycle of one scene: level 0's right-hand side through A (fused with the CG update
// when A.q is set), result in mgz of level 0, partials of r.z and r.r; r_new: the residual
// after the update. Returns false on a barrier timeout.
template <class M>
DEV bool vcycle(const DevScene& d, const Geo& g, const Tail& tl, const DownArgs& A, const float2* r_new, const TileCache& tc) {
    const int tail = d.lv.tail;
    auto of = [&d](int) -> const DevScene& { return d; };
#pragma unroll 1
    for (int l = 0; l < tail; l++) {
        const Lv F = lev(d.lv, l), C = lev(d.lv, l + 1);
        DownArgs D = A;
        if (l > 0) D = DownArgs{d.mgr, nullptr, 0.0f, 0.0f, nullptr, nullptr};
        down_pass<M>(g, my_count(active_tiles(d, l, tc)), l == 0, of, [&](int k) { return DownTile{0, F, C, my_tile(d, tc, l, k), D}; }, EveryOne());
        if (!grid_sync(d.K)) return false;
    }
    // only the blocks with a tile of the level above the tail read the tail's result (from
    // their own copy); block 0 also stores it
    if (tail_reader(d, tc)) phase_tail(d.mgr + tl.base, blockIdx.x == 0 ? d.mgz + tl.base : nullptr, tl);
#pragma unroll 1
    for (int l = tail - 1; l >= 0; l--) {
        const Lv F = lev(d.lv, l), C = lev(d.lv, l + 1);
        const float2* zs = l == tail - 1 ? tl.x : nullptr;
        const float2* r = l == 0 ? r_new : d.mgr;
        up_pass<M>(g, my_count(active_tiles(d, l, tc)), l == 0, of, [&](int k) { return UpTile{0, F, C, my_tile(d, tc, l, k), r, d.mgz + C.off, zs}; }, EveryOne());
        if (!grid_sync(d.K)) return false;
    }
    return true;
}

// b - A x of a level-0 cell's pressure column, and of both columns, evaluated as float pairs:
// each product exact (fma), the sum compensated (about 48 significant bits, FP64's job here
// at a small fraction of FP64's cost on this GPU), rounded once to FP32 at the end
DEV float2 pair_prod(float a, float b) {
    const float p = a * b;
    return make_float2(p, fmaf(a, b, -p));
}
DEV float2 pair_acc(float2 s, float2 t) { return ff_add(s.x, s.y, t.x, t.y); }

// The true residual |b - A x| / |b| of the pressure column after a mixed-precision solve:
// the tile's sums of (b - A x)^2 and b^2 as float pairs into part[t].
DEV void true_residual_tile(const DevScene& d, int t, FF4* part, FF4* buf) {
    const Lv F = lev(d.lv, 0);
    if (d.ptile[F.toff + t] == 0u) {
        if (threadIdx.x == 0) part[t] = FF4{make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
        return;
    }
    const int2 og = tile_origin(F, t);
    const int cx = og.x + (threadIdx.x & 15), cy = og.y + (threadIdx.x >> 4);
    FF4 a4{make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
    if (l_inside(F, cx, cy)) {
        const int i = l_at(F, cx, cy);
        const float D = d.mgd[i];
        if (D > 0.0f) {
            const float4 w = d.mga[i];
            const float b = d.prhs[i].x;
            const float2 dx = pair_prod(D, d.pres[i].x);
            float2 r = pair_acc(make_float2(b, 0.0f), make_float2(-dx.x, -dx.y));
            for (int q = 0; q < 4; q++) {
                const int nx = cx + NBX[q], ny = cy + NBY[q];
                if (unknown_op(d, F, nx, ny)) r = pair_acc(r, pair_prod(wcomp(w, q), d.pres[l_at(F, nx, ny)].x));
            }
            const float rf = r.x + r.y;
            a4 = ff_prod4(rf, rf, b, b, 0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    buf[threadIdx.x] = a4;
    block_tree(buf);
    if (threadIdx.x == 0) part[t] = buf[0];
    __syncthreads();
}

// The mixed solve's refinement (residual replacement: van der Vorst and Ye, "Residual
// replacement strategies for Krylov subspace iterative methods", SIAM J. Sci. Comput. 22,
// 2000). The recurrence r -= alpha q drifts from b - A x by rounding; at a few points of the
// convergence the true residual of the current iterate is evaluated (the products and sums of
// the FP32 values as float pairs, rounded once to FP32) and, where the drift is worth removing, it
// replaces the carried one; the iteration continues with its directions unchanged.
//
// check_tile: on level-0 tile t, the true residual b - A x of both columns into rt, and the
// tile's sums of |b - A x|^2 and of (eps |A| |x|)^2 of the pressure column into part[t]: the
// second is the size of the residual that rounding x to FP32 alone leaves (eps = 2^-24), below
// which a replacement would feed that rounding back into the recurrence instead of removing
// drift.
DEV void check_tile(const DevScene& d, int t, float2* rt, FF4* part, FF4* buf) {
    const Lv F = lev(d.lv, 0);
    const FF4 zero{make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
    if (d.ptile[F.toff + t] == 0u) {
        if (threadIdx.x == 0) part[t] = zero;
        return;
    }
    const int2 og = tile_origin(F, t);
    const int cx = og.x + (threadIdx.x & 15), cy = og.y + (threadIdx.x >> 4);
    FF4 a4 = zero;
    if (l_inside(F, cx, cy)) {
        const int i = l_at(F, cx, cy);
        const float D = d.mgd[i];
        if (D > 0.0f) {
            const float4 w = d.mga[i];
            const float2 x = d.pres[i];
            const float4 b = d.prhs[i];
            const float2 dx = pair_prod(D, x.x), dy = pair_prod(D, x.y);
            float2 rx = pair_acc(make_float2(b.x, 0.0f), make_float2(-dx.x, -dx.y));
            float2 ry = pair_acc(make_float2(b.y, 0.0f), make_float2(-dy.x, -dy.y));
            float ax = fabsf(D * x.x);
            for (int q = 0; q < 4; q++) {
                const int nx = cx + NBX[q], ny = cy + NBY[q];
                if (unknown_op(d, F, nx, ny)) {
                    const float2 xn = d.pres[l_at(F, nx, ny)];
                    const float wq = wcomp(w, q);
                    rx = pair_acc(rx, pair_prod(wq, xn.x));
                    ry = pair_acc(ry, pair_prod(wq, xn.y));
                    ax += fabsf(wq * xn.x);
                }
            }
            const float rfx = rx.x + rx.y, rfy = ry.x + ry.y;
            rt[i] = make_float2(rfx, rfy);
            const float fl = ax * 0x1p-24f;
            a4 = ff_prod4(rfx, rfx, fl, fl, 0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            rt[i] = make_float2(0.0f, 0.0f);
        }
    }
    buf[threadIdx.x] = a4;
    block_tree(buf);
    if (threadIdx.x == 0) part[t] = buf[0];
    __syncthreads();
}

// ... and, where it is adopted, the carried residual r of tile t replaced by it.
DEV void adopt_tile(const DevScene& d, int t, const float2* rt, float2* r) {
    const Lv F = lev(d.lv, 0);
    if (d.ptile[F.toff + t] == 0u) return;
    const int2 og = tile_origin(F, t);
    const int cx = og.x + (threadIdx.x & 15), cy = og.y + (threadIdx.x >> 4);
    if (!l_inside(F, cx, cy)) return;
    const int i = l_at(F, cx, cy);
    if (d.mgd[i] > 0.0f) r[i] = rt[i];
}

// When to check: each time the pressure column's carried r.r has fallen by kCheckDrop (its
// norm by 100) since the start or the last check, before the solve has converged, unless a
// check found the carried residual already near the rounding floor.
// Whether to adopt: the true residual is more than twice the carried one (drift worth
// removing) and more than ten times the rounding floor.
constexpr double kCheckDrop = 1e-4;
template <class T>
DEV bool want_check(const Solve<T>& K) {
    return K.done[0] == 0u && K.floor_hit == 0u && K.rr[0] > 0 && K.rr[0] <= (T)kCheckDrop * K.rmark;
}
// Decides from the check's totals (|b - A x|^2, floor^2); updates the marks. Returns adopt.
template <class T>
DEV bool decide_check(Solve<T>& K, const Dbl4& tot) {
    K.rmark = K.rr[0];
    const double carried = (double)K.rr[0];
    if (carried <= 100.0 * tot.y) K.floor_hit = 1u;
    const bool adopt = tot.x > 4.0 * carried && tot.x > 100.0 * tot.y;
    if (adopt) K.replaced += 1u;
    return adopt;
}

template <class T>
DEV T mix_was(T a, T keep, uint32_t was) { return mixf(a, keep, (float)was); }
template <>
DEV double mix_was<double>(double a, double keep, uint32_t was) { return was ? keep : a; }

// The solve's scalar steps (reduce_tail.glsl:61-116), shared by the single-scene and batched
// kernels so that a scene's numbers do not depend on which one solved it.
// mode 0 / 8: the start, from the totals a = (r.z, r.r) and b = (b.b).
template <class T, class A4>
DEV void scal_start(Solve<T>& K, const A4& a, const A4& b, T tx, T ty, int second) {
    K.bb[0] = b.x;
    K.bb[1] = b.y;
    K.rz[0] = a.x;
    K.rz[1] = a.y;
    K.rr[0] = a.z;
    K.rr[1] = a.w;
    K.rmark = a.z;
    K.replaced = 0u;
    K.floor_hit = 0u;
    K.adopt = 0u;
    K.beta[0] = K.beta[1] = 0;
    K.alpha[0] = K.alpha[1] = 0;
    K.iters[0] = K.iters[1] = 0u;
    K.done[0] = a.z <= tx * tx * b.x ? 1u : 0u;
    K.done[1] = a.w <= ty * ty * b.y ? 1u : 0u;
    if (second) K.done[1] = 1u;
    // a non-finite right-hand side or residual: no iteration can converge, stop here
    K.bad = finite4(a) && finite4(b) ? 0u : 1u;
    if (K.bad) K.done[0] = K.done[1] = 1u;
}

// mode 1: the step lengths from p.q.
template <class T, class A4>
DEV void scal_alpha(Solve<T>& K, const A4& b) {
    T ax = 0, ay = 0;
    if (K.done[0] == 0u && b.z > 0) ax = K.rz[0] / b.z;
    if (K.done[1] == 0u && b.w > 0) ay = K.rz[1] / b.w;
    K.alpha[0] = ax;
    K.alpha[1] = ay;
}

// mode 2: convergence and the next direction's beta from the new (r.z, r.r).
template <class T, class A4>
DEV void scal_beta(Solve<T>& K, const A4& a, T tx, T ty) {
    uint32_t was0 = K.done[0], was1 = K.done[1];
    K.iters[0] += 1u - was0;
    K.iters[1] += 1u - was1;
    uint32_t now0 = a.z <= tx * tx * K.bb[0] ? 1u : 0u, now1 = a.w <= ty * ty * K.bb[1] ? 1u : 0u;
    uint32_t d0 = was0 > now0 ? was0 : now0, d1 = was1 > now1 ? was1 : now1;
    T bx = 0, by = 0;
    if (d0 == 0u && K.rz[0] > 0) bx = a.x / K.rz[0];
    if (d1 == 0u && K.rz[1] > 0) by = a.y / K.rz[1];
    K.beta[0] = bx;
    K.beta[1] = by;
    K.rz[0] = a.x;
    K.rz[1] = a.y;
    K.rr[0] = mix_was<T>(a.z, K.rr[0], was0);
    K.rr[1] = mix_was<T>(a.w, K.rr[1], was1);
    K.done[0] = d0;
    K.done[1] = d1;
    if (!finite4(a)) {
        K.bad = 1u;
        K.done[0] = K.done[1] = 1u;
    }
}

// mode 3 / 9: the statistics of the finished solve into the scene's SolveState.
template <class M, class T>
DEV void scal_stats(SolveState* G, const Solve<T>& K, int second, double true_rel) {
    if (true_rel >= 0.0) {
        G->p_true_res = (float)true_rel;
        G->p_true_res_max = maxf(G->p_true_res_max, (float)true_rel);
    }
    G->p_repl += K.replaced;
    for (int c = 0; c < 2; c++) {
        G->p_rz[c] = (float)K.rz[c];
        G->p_alpha[c] = (float)K.alpha[c];
        G->p_beta[c] = (float)K.beta[c];
        G->p_bb[c] = (float)K.bb[c];
        G->p_rr[c] = (float)K.rr[c];
        G->p_done[c] = K.done[c];
        if (!second) G->p_iters[c] = K.iters[c];
    }
    if (second) G->p2_iters = K.iters[0];
    G->solves += 1u;
    if (!second) {
        uint32_t m = K.iters[0] > K.iters[1] ? K.iters[0] : K.iters[1];
        if (m > G->p_it_max) G->p_it_max = m;
        if (K.done[0] == 0u) G->p_unconv += 1u;
        if (m > G->f_it[0]) G->f_it[0] = m;
        if (K.done[0] == 0u) G->f_un[0] += 1u;
    } else {
        if (K.iters[0] > G->p2_it_max) G->p2_it_max = K.iters[0];
        if (K.done[0] == 0u) G->p2_unconv += 1u;
        if (K.iters[0] > G->f_it[1]) G->f_it[1] = K.iters[0];
        if (K.done[0] == 0u) G->f_un[1] += 1u;
    }
    if (K.bad) atomicOr(&G->error, ERR_DIVERGED);
    const float rel = K.bb[0] > 0 ? (float)sqrt((double)K.rr[0] / (double)K.bb[0]) : 0.0f;
    G->p_res_max = maxf(G->p_res_max, M::kMixed ? rel : (K.bb[0] > 0 ? sqrtf((float)K.rr[0] / (float)K.bb[0]) : 0.0f));
}

}  // namespace

// The whole pressure solve. `second`: the solve after the implicit viscosity (cg_reduce
// mode 8/9: same matrix and hierarchy, density correction counted as solved).
template <class M>
__global__ void __launch_bounds__(NT, 2) k_mgpcg(const __grid_constant__ DevScene d, int second, int scale_mode) {
    grid_begin(d.K);
    using acc = typename M::acc;
    using acc4 = typename M::acc4;
    __shared__ TileCache tc;
    // the block's tree buffer, in the stages' bytes: no tile is staged while it is used
    static_assert(NT * sizeof(FF4) <= sizeof(TileSmem::stage), "the refinement's checks sum float pairs");
    acc4* const buf = reinterpret_cast<acc4*>(dyn_smem);
    __shared__ Solve<acc> K;
    const DevParams* P = d.P;
    const int n = d.nwg;
    acc4* part = M::part(d);
    const Tail tl = make_tail(d);
    const Geo g = geo();
    if (!second) {
        for (int t = blockIdx.x; t < n; t += gridDim.x) cg_scale_tile<M>(d, t, scale_mode);
        for (int l = 1; l <= d.lv.tail; l++) {
            if (!grid_sync(d.K)) return;
            const int T = level_tiles(d, l);
            for (int t = blockIdx.x; t < T; t += gridDim.x) mg_build_tile<M>(d, l - 1, t);
        }
        if (!grid_sync(d.K)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) d.K->hier = M::kHier;
    }
    // the active-tile lists (ptile is final now) and the inactive tiles' zero partial sums
    for (int l = blockIdx.x; l < d.lv.tail; l += gridDim.x) build_plist(d, l);   // a level a block
    for (int t = blockIdx.x * NT + threadIdx.x; t < n; t += gridDim.x * NT) zero_inactive_tile<M>(d, t);
    if (!grid_sync(d.K)) return;
    fill_cache(d, tc);
    if (tail_reader(d, tc)) tail_setup<M>(d, tl, blockIdx.x == 0);
    float2* r_cur = d.mgr;    // level 0 of mgr: the residual, double-buffered with mgr2
    float2* r_nxt = d.mgr2;
    residual_pass<M>(my_count(active_tiles(d, 0, tc)), reinterpret_cast<float4*>(dyn_smem), [&](int k, int& t) -> const DevScene& {
        t = my_tile(d, tc, 0, k);
        return d;
    });
    if (!grid_sync(d.K)) return;
    // b.b now, while nothing writes the second half of the partials: the first apply phase
    // after the V-cycle does, and a block can reach it before a slower one has summed them
    const auto b = M::fin(total(part + n, n, buf));
    const acc tx = (acc)P->tol[0], ty = (acc)P->tol[1];
    float2* p_old = d.cgp;
    float2* p_new = d.cgp2;
    const Lv L0 = lev(d.lv, 0);
    const uint32_t cap = d.K->cap[second ? 1 : 0];   // this frame's recorded iterations
    // it = 0: the start (a V-cycle on the residual of x0); it > 0: the iterations
    for (uint32_t it = 0;; it++) {
        DownArgs A{r_cur, nullptr, 0.0f, 0.0f, nullptr, nullptr};
        if (it > 0) {
            if (it > cap || (K.done[0] && K.done[1])) break;
            if constexpr (M::kMixed) {
                // the refinement (the same decisions in every block: the same K); q is free until
                // the apply phase rewrites it, and the partials' second half until it sums p.q
                if (it > 1 && want_check(K)) {
                    FF4* pc = reinterpret_cast<FF4*>(d.partials64) + n;
                    for_active(d, 0, tc, [&](int t) { check_tile(d, t, d.cgq, pc, reinterpret_cast<FF4*>(dyn_smem)); });
                    if (!grid_sync(d.K)) return;
                    const Dbl4 tot = to_dbl(total(pc, n, reinterpret_cast<FF4*>(dyn_smem)));
                    __shared__ int s_adopt;
                    if (threadIdx.x == 0) s_adopt = decide_check(K, tot) ? 1 : 0;
                    __syncthreads();
                    if (s_adopt) {
                        for_active(d, 0, tc, [&](int t) { adopt_tile(d, t, d.cgq, r_cur); });
                        if (!grid_sync(d.K)) return;
                    }
                }
            }
            const float b0 = (float)K.beta[0], b1 = (float)K.beta[1];
            apply_pass<M>(my_count(active_tiles(d, 0, tc)), [&d](int) -> const DevScene& { return d; }, [&](int k) { return ApplyTile{0, L0, my_tile(d, tc, 0, k), b0, b1, p_old, p_new}; }, EveryOne());
            if (!grid_sync(d.K)) return;
            const auto pq = M::fin(total(part + n, n, buf));
            if (threadIdx.x == 0) scal_alpha<acc>(K, pq);
            __syncthreads();
            A = DownArgs{r_cur, d.cgq, (float)K.alpha[0], (float)K.alpha[1], p_new, r_nxt};
        }
        if (!vcycle<M>(d, g, tl, A, it > 0 ? r_nxt : r_cur, tc)) return;
        const auto a = M::fin(total(part, n, buf));
        if (threadIdx.x == 0) {
            if (it == 0) scal_start<acc>(K, a, b, tx, ty, second);
            else scal_beta<acc>(K, a, tx, ty);
        }
        __syncthreads();
        if (it == 0) continue;
        float2* t = p_old;
        p_old = p_new;
        p_new = t;
        t = r_cur;
        r_cur = r_nxt;
        r_nxt = t;
    }
    double true_rel = -1.0;
    if constexpr (M::kMixed) {
        FF4* pt = reinterpret_cast<FF4*>(d.partials64);
        for_active(d, 0, tc, [&](int t) { true_residual_tile(d, t, pt, reinterpret_cast<FF4*>(dyn_smem)); });
        if (!grid_sync(d.K)) return;
        const Dbl4 t4 = to_dbl(total(pt, n, reinterpret_cast<FF4*>(dyn_smem)));
        true_rel = t4.y > 0.0 ? sqrt(t4.x / t4.y) : 0.0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) scal_stats<M, acc>(d.K, K, second, true_rel);
    trace_launch_done(d.K);
}

// ---- many scenes in one persistent solve --------------------------------------------------
//
// The same solve for a batch of scenes of any sizes in one cooperative launch: every phase
// runs over a flattened list of (scene, tile) work items of its level, so the small levels
// of many scenes fill one pass instead of leaving most blocks idle, and one set of grid
// barriers serves them all. Each scene's tiles go through the same tile bodies as above and
// its scalars through the same steps, summed by one block over its own partials in the
// same order; so a scene's result is the same alone and in any batch, to the bit. The
// differences: a scene's tail is computed by one block into global memory (one more
// barrier per V-cycle), each reduction is a phase of its own followed by a barrier (the
// scalars then live in global memory), and a converged scene (or one at its iteration
// limit) simply drops out of the work lists.

namespace {

// The scene, tile and level of work item g of level l: o holds the ns + 1 prefix sums of
// the scenes' tile counts of level l.
DEV int scene_of(const int* o, int ns, int g) {
    int lo = 0, hi = ns;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (o[mid] <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <class F>
DEV void for_tiles(const BatchView& B, int l, F&& f) {
    const int* o = B.off + l * (B.ns + 1);
    const int N = o[B.ns];
    for (int g = blockIdx.x; g < N; g += gridDim.x) {
        const int s = scene_of(o, B.ns, g);
        f(s, B.scenes[s], g - o[s]);
    }
}

// For every active tile of level l over the batch's scenes (B.aoff: the prefix sums of the
// scenes' active-tile counts, built at the solve's start).
DEV uint32_t batch_item(const BatchView& B, int l, int g) {
    const int* o = B.aoff + l * (B.ns + 1);
    const int s = scene_of(o, B.ns, g);
    const DevScene& d = B.scenes[s];
    return ((uint32_t)s << 16) | d.plist[d.lv.toff[l] + (g - o[s])];
}

DEV uint32_t active_tiles_b(const BatchView& B, int l, const TileCache& tc) {
    return l < kCacheLevels ? tc.cnt[l] : *(volatile const uint32_t*)&B.aoff[l * (B.ns + 1) + B.ns];
}
DEV void fill_cache_b(const BatchView& B, TileCache& tc) {
    for (int l = 0; l < kCacheLevels && l < B.max_tail; l++)
        fill_level(tc, l, *(volatile const uint32_t*)&B.aoff[l * (B.ns + 1) + B.ns], [&](uint32_t k) { return batch_item(B, l, (int)k); });
    __syncthreads();
}

template <class F>
DEV void for_active_b(const BatchView& B, int l, const TileCache& tc, F&& f) {
    const uint32_t N = active_tiles_b(B, l, tc);
    for (uint32_t g = blockIdx.x; g < N; g += gridDim.x) {
        const uint32_t it = batch_item(B, l, (int)g);
        const int s = (int)(it >> 16);
        f(s, B.scenes[s], (int)(it & 0xffffu));
    }
}

DEV float2* parity_r(const DevScene& d, int it) { return (it & 1) ? d.mgr2 : d.mgr; }
DEV float2* parity_p(const DevScene& d, int it) { return (it & 1) ? d.cgp2 : d.cgp; }

}  // namespace

size_t pressure_smem(const Levels& lv) {
    return kTileBytes + tail_bytes(tail_cells(lv), lv.w[lv.tail] * lv.h[lv.tail]);
}

template <class M>
__global__ void __launch_bounds__(NT, 2) k_mgpcg_batch(BatchView B, int second) {
    grid_begin(B.K);
    using acc = typename M::acc;
    using acc4 = typename M::acc4;
    __shared__ TileCache tc;
    // the block's tree buffer, in the stages' bytes: no tile is staged while it is used
    static_assert(NT * sizeof(FF4) <= sizeof(TileSmem::stage), "the refinement's checks sum float pairs");
    acc4* const buf = reinterpret_cast<acc4*>(dyn_smem);
    __shared__ int s_run;
    Solve<acc>* KS = reinterpret_cast<Solve<acc>*>(B.scal);
    SolveState* BK = B.K;
    auto tol = [&](const DevScene& d, int c) { return (acc)d.P->tol[c]; };
    // a scene takes part in iteration it while neither converged nor at its limit
    auto running = [&](int s, int it) {
        const Solve<acc>& K = KS[s];
        return !(K.done[0] && K.done[1]) && (uint32_t)it < B.scenes[s].K->cap[second ? 1 : 0];
    };
    if (!second) {
        for_tiles(B, 0, [&](int s, const DevScene& d, int t) { cg_scale_tile<M>(d, t, B.scale[s]); });
        for (int l = 1; l <= B.max_tail; l++) {
            if (!grid_sync(BK)) return;
            for_tiles(B, l, [&](int s, const DevScene& d, int t) { mg_build_tile<M>(d, l - 1, t); });
        }
        if (!grid_sync(BK)) return;
        for (int s = blockIdx.x * NT + threadIdx.x; s < B.ns; s += gridDim.x * NT) B.scenes[s].K->hier = M::kHier;
    }
    // every scene's active-tile lists (a block each level) and the inactive tiles' zero partials
    for (int g = blockIdx.x; g < B.ns * B.max_tail; g += gridDim.x) {
        const DevScene& d = B.scenes[g / B.max_tail];
        const int l = g % B.max_tail;
        if (l < d.lv.tail) build_plist(d, l);
    }
    {
        const int* o = B.off;
        for (int g = blockIdx.x * NT + threadIdx.x; g < o[B.ns]; g += gridDim.x * NT) {
            const int s = scene_of(o, B.ns, g);
            zero_inactive_tile<M>(B.scenes[s], g - o[s]);
        }
    }
    if (!grid_sync(BK)) return;
    // ... and their prefix sums per level over the scenes
    if (blockIdx.x == 0) {
        for (int l = threadIdx.x; l < B.max_tail; l += NT) {
            int* o = B.aoff + l * (B.ns + 1);
            int acc_ = 0;
            o[0] = 0;
            for (int k = 0; k < B.ns; k++) {
                const DevScene& d = B.scenes[k];
                acc_ += l < d.lv.tail ? (int)d.pcount[l] : 0;
                o[k + 1] = acc_;
            }
        }
    }
    if (!grid_sync(BK)) return;
    fill_cache_b(B, tc);
    residual_pass<M>(my_count(active_tiles_b(B, 0, tc)), reinterpret_cast<float4*>(dyn_smem), [&](int k, int& t) -> const DevScene& {
        const uint32_t g = my_item(tc, 0, k, [&](uint32_t q) { return batch_item(B, 0, (int)q); });
        t = (int)(g & 0xffffu);
        return B.scenes[g >> 16];
    });
    if (!grid_sync(BK)) return;
    // b.b of each scene (before the first apply phase reuses those partials)
    for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
        const DevScene& d = B.scenes[s];
        const auto b = M::fin(total(M::part(d) + d.nwg, d.nwg, buf));
        if (threadIdx.x == 0) {
            KS[s].bb[0] = b.x;
            KS[s].bb[1] = b.y;
            KS[s].done[0] = KS[s].done[1] = 0u;
        }
        __syncthreads();
    }
    // one tail per block stays in its shared memory for the whole solve; with more scenes than
    // blocks, each tail phase sets its tail up again
    const bool resident = B.ns <= (int)gridDim.x;
    if (resident && (int)blockIdx.x < B.ns) tail_setup_of<M>(B.scenes + blockIdx.x);
    const Geo geom = geo();
    auto of = [&B](int s) -> const DevScene& { return B.scenes[s]; };
    auto item = [&](int l, int k) { return my_item(tc, l, k, [&](uint32_t g) { return batch_item(B, l, (int)g); }); };
    // One V-cycle on every running scene; it < 0: the start (right-hand side the residual
    // of x0, no update); else the iteration's, fused with its update.
    auto vcycle_all = [&](int it) -> bool {
        const bool fused = it >= 0;
        const int ir = fused ? it : 0;
        // the next of this block's items of level l, from its k-th on, whose scene takes part
        auto live = [&](int l, int count) {
            return [&, l, count](int k) {
                while (k < count && fused && !running((int)(item(l, k) >> 16), it)) k++;
                return k;
            };
        };
#pragma unroll 1
        for (int l = 0; l < B.max_tail; l++) {
            const int count = my_count(active_tiles_b(B, l, tc));
            down_pass<M>(geom, count, l == 0, of, [&](int k) {
                const uint32_t g = item(l, k);
                const int s = (int)(g >> 16);
                const DevScene& d = B.scenes[s];
                DownArgs A{d.mgr, nullptr, 0.0f, 0.0f, nullptr, nullptr};
                if (l == 0) {
                    A.r = parity_r(d, ir);
                    if (fused) A = DownArgs{A.r, d.cgq, (float)KS[s].alpha[0], (float)KS[s].alpha[1], parity_p(d, ir + 1), parity_r(d, ir + 1)};
                }
                return DownTile{s, lev(d.lv, l), lev(d.lv, l + 1), (int)(g & 0xffffu), A};
            }, live(l, count));
            if (!grid_sync(BK)) return false;
        }
        for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
            if (fused && !running(s, it)) continue;
            const DevScene& d = B.scenes[s];
            const Tail tl = make_tail(d);
            if (!resident) tail_setup_of<M>(&d);
            phase_tail(d.mgr + tl.base, d.mgz + tl.base, tl);
            __syncthreads();
        }
        if (!grid_sync(BK)) return false;
#pragma unroll 1
        for (int l = B.max_tail - 1; l >= 0; l--) {
            const int count = my_count(active_tiles_b(B, l, tc));
            up_pass<M>(geom, count, l == 0, of, [&](int k) {
                const uint32_t g = item(l, k);
                const DevScene& d = B.scenes[g >> 16];
                const Lv C = lev(d.lv, l + 1);
                return UpTile{(int)(g >> 16), lev(d.lv, l), C, (int)(g & 0xffffu), l == 0 ? parity_r(d, fused ? ir + 1 : 0) : d.mgr, d.mgz + C.off, nullptr};
            }, live(l, count));
            if (!grid_sync(BK)) return false;
        }
        return true;
    };
    if (!vcycle_all(-1)) return;
    for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
        const DevScene& d = B.scenes[s];
        const auto a = M::fin(total(M::part(d), d.nwg, buf));
        if (threadIdx.x == 0) {
            auto b = a;
            b.x = KS[s].bb[0];
            b.y = KS[s].bb[1];
            scal_start<acc>(KS[s], a, b, tol(d, 0), tol(d, 1), second);
        }
        __syncthreads();
    }
    if (!grid_sync(BK)) return;
    for (int it = 0;; it++) {
        if (threadIdx.x == 0) {
            int run = 0;
            for (int s = 0; s < B.ns && !run; s++) run = running(s, it) ? 1 : 0;
            s_run = run;
        }
        __syncthreads();
        if (!s_run) break;
        if constexpr (M::kMixed) {   // the refinement, as the single-scene solve takes it
            // a scene checks at iteration it when want_check holds at the top of the iteration;
            // one block decides (after the check's barrier) and leaves the outcome in KS[s].adopt
            auto chk = [&](int s) { return it > 0 && running(s, it) && want_check(KS[s]); };
            if (threadIdx.x == 0) {
                int any = 0;
                for (int s = 0; s < B.ns && !any; s++) any = chk(s) ? 1 : 0;
                s_run = any;
            }
            __syncthreads();
            if (s_run) {
                for_active_b(B, 0, tc, [&](int s, const DevScene& d, int t) {
                    if (chk(s)) check_tile(d, t, d.cgq, reinterpret_cast<FF4*>(d.partials64) + d.nwg, reinterpret_cast<FF4*>(dyn_smem));
                });
                if (!grid_sync(BK)) return;
                // each scene's decision by one block (it alone writes KS[s] until the next barrier)
                for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
                    if (!chk(s)) continue;
                    const DevScene& d = B.scenes[s];
                    const Dbl4 tot = to_dbl(total(reinterpret_cast<FF4*>(d.partials64) + d.nwg, d.nwg, reinterpret_cast<FF4*>(dyn_smem)));
                    if (threadIdx.x == 0) KS[s].adopt = decide_check(KS[s], tot) ? 1u : 0u;
                    __syncthreads();
                }
                if (!grid_sync(BK)) return;
                // every block reads the same decisions: without an adoption, the adopt pass
                // and its barrier are skipped by all of them
                if (threadIdx.x == 0) {
                    int adopt = 0;
                    for (int s = 0; s < B.ns && !adopt; s++) adopt = KS[s].adopt ? 1 : 0;
                    s_run = adopt;
                }
                __syncthreads();
                if (s_run) {
                    for_active_b(B, 0, tc, [&](int s, const DevScene& d, int t) {
                        if (KS[s].adopt) adopt_tile(d, t, d.cgq, parity_r(d, it));
                    });
                    if (!grid_sync(BK)) return;
                    for (int s = blockIdx.x; s < B.ns; s += gridDim.x)
                        if (threadIdx.x == 0) KS[s].adopt = 0u;
                }
            }
        }
        {
            const int count = my_count(active_tiles_b(B, 0, tc));
            apply_pass<M>(count, of, [&](int k) {
                const uint32_t g = item(0, k);
                const int s = (int)(g >> 16);
                const DevScene& d = B.scenes[s];
                return ApplyTile{s, lev(d.lv, 0), (int)(g & 0xffffu), (float)KS[s].beta[0], (float)KS[s].beta[1], parity_p(d, it), parity_p(d, it + 1)};
            }, [&](int k) {
                while (k < count && !running((int)(item(0, k) >> 16), it)) k++;
                return k;
            });
        }
        if (!grid_sync(BK)) return;
        for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
            if (!running(s, it)) continue;
            const DevScene& d = B.scenes[s];
            const auto b = M::fin(total(M::part(d) + d.nwg, d.nwg, buf));
            if (threadIdx.x == 0) scal_alpha<acc>(KS[s], b);
            __syncthreads();
        }
        if (!grid_sync(BK)) return;
        if (!vcycle_all(it)) return;
        for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
            if (!running(s, it)) continue;
            const DevScene& d = B.scenes[s];
            const auto a = M::fin(total(M::part(d), d.nwg, buf));
            if (threadIdx.x == 0) scal_beta<acc>(KS[s], a, tol(d, 0), tol(d, 1));
            __syncthreads();
        }
        if (!grid_sync(BK)) return;
    }
    if constexpr (M::kMixed) {
        for_active_b(B, 0, tc, [&](int s, const DevScene& d, int t) {
            true_residual_tile(d, t, reinterpret_cast<FF4*>(d.partials64), reinterpret_cast<FF4*>(dyn_smem));
        });
        if (!grid_sync(BK)) return;
    }
    for (int s = blockIdx.x; s < B.ns; s += gridDim.x) {
        const DevScene& d = B.scenes[s];
        double true_rel = -1.0;
        if constexpr (M::kMixed) {
            const Dbl4 t4 = to_dbl(total(reinterpret_cast<FF4*>(d.partials64), d.nwg, reinterpret_cast<FF4*>(dyn_smem)));
            true_rel = t4.y > 0.0 ? sqrt(t4.x / t4.y) : 0.0;
        }
        if (threadIdx.x == 0) scal_stats<M, acc>(d.K, KS[s], second, true_rel);
        __syncthreads();
    }
    trace_launch_done(BK);
}

namespace {
template <class M>
int blocks_max(int device, size_t smem) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // Opt in to the dynamic shared memory the largest tank so far needs (static + dynamic
    // above 48 KB needs it). The attribute belongs to the kernel on the current device, so
    // it is tracked per device.
    static size_t opted[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices || smem > opted[device]) {
        cudaFuncSetAttribute(k_mgpcg<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (device >= 0 && device < kMaxDevices) opted[device] = smem;
    }
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mgpcg<M>, NT, smem);
    return sms * per;
}
}  // namespace

int pressure_blocks_max(int device, size_t smem, bool mixed) {
    return mixed ? blocks_max<Mixed>(device, smem) : blocks_max<Plain>(device, smem);
}

namespace {
template <class M>
int batch_blocks_max(int device, size_t smem) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    static size_t opted[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices || smem > opted[device]) {
        cudaFuncSetAttribute(k_mgpcg_batch<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (device >= 0 && device < kMaxDevices) opted[device] = smem;
    }
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mgpcg_batch<M>, NT, smem);
    return sms * per;
}
}  // namespace

int pressure_batch_blocks_max(int device, size_t smem, bool mixed) {
    return mixed ? batch_blocks_max<Mixed>(device, smem) : batch_blocks_max<Plain>(device, smem);
}

size_t pressure_batch_scalar_bytes() { return sizeof(Solve<double>); }

cudaError_t launch_pressure_batch(const BatchView& B, bool mixed, int blocks, size_t smem, cudaStream_t st, int second) {
    cudaMemsetAsync(&B.K->bar_count, 0, sizeof(uint32_t), st);
    void* args[] = {(void*)&B, &second};
    const void* fn = mixed ? (const void*)k_mgpcg_batch<Mixed> : (const void*)k_mgpcg_batch<Plain>;
    return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(NT), args, smem, st);
}

// FluidSim::poll_readbacks' adaptation of a recorded iteration count (mod.rs:3100-3106):
// after a frame in which the solve ran out, half again plus two; otherwise the frame's most
// iterations plus the margin's share (truncated, as `as u32`) plus two, within [2, max].
DEV uint32_t adapt_rec(uint32_t rec, uint32_t used, uint32_t unconverged, uint32_t max, float margin) {
    if (unconverged > 0u) return min(rec + rec / 2u + 2u, max);
    const uint32_t v = used + (uint32_t)((float)used * margin) + 2u;
    return v < 2u ? 2u : (v > max ? max : v);
}

// The end of a frame (a step call): the recorded counts adapted from the frame's solves as
// the reference adapts them when the frame's read-back arrives (mod.rs:3093-3114: the second
// solve's follows the first's when it does not run; the viscosity solve's with margin 0.5),
// the next frame's limits, and the frame's statistics cleared.
DEV void frame_end(const DevScene& d) {
    const DevParams* P = d.P;
    SolveState* K = d.K;
    K->rec[0] = adapt_rec(K->rec[0], K->f_it[0], K->f_un[0], P->pressure_max_iters, P->iters_margin);
    if (P->visc_mode == 2 && P->viscous_projection != 0)
        K->rec[1] = adapt_rec(K->rec[1], K->f_it[1], K->f_un[1], P->pressure_max_iters, P->iters_margin);
    else
        K->rec[1] = K->rec[0];
    K->rec[2] = adapt_rec(K->rec[2], K->f_it[2], K->f_un[2], P->viscosity_max_iters, 0.5f);
    for (int k = 0; k < 3; k++) {
        K->cap[k] = recorded_limit(K->rec[k], k == 2, P->viscosity_precond != 0);
        K->f_it[k] = 0u;
        K->f_un[k] = 0u;
    }
}

__global__ void k_frame_end(DevScene d) { frame_end(d); }
__global__ void k_frame_end_many(const DevScene* scenes, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) frame_end(scenes[s]);
}

void launch_frame_end(const DevScene& d, cudaStream_t st) { k_frame_end<<<1, 1, 0, st>>>(d); }
void launch_frame_end_many(const DevScene* scenes, int n, cudaStream_t st) {
    if (n > 0) k_frame_end_many<<<(n + 127) / 128, 128, 0, st>>>(scenes, n);
}

cudaError_t launch_pressure(const DevScene& d, const LaunchCfg& cfg, cudaStream_t st, int second) {
    // (the right-hand side's kernel, k_rhs or k_rhs_visc, has zeroed the barrier)
    // cg_scale mode 1: with the viscosity between two solves, the first starts from last
    // substep's P1 alone (viscous_warm, mod.rs:2979-2983)
    int scale_mode = (!second && cfg.visc_mode == 2 && cfg.twice && cfg.viscous_warm) ? 1 : 0;
    void* args[] = {(void*)&d, &second, &scale_mode};
    const void* fn = cfg.mixed ? (const void*)k_mgpcg<Mixed> : (const void*)k_mgpcg<Plain>;
    const int blocks = cfg.mixed ? cfg.mg_blocks_mixed : cfg.mg_blocks;
    return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(NT), args, pressure_smem(d.lv), st);
}

}  // namespace sprout

namespace sprout {

// ---- the pressure solve on caller buffers, with no allocation ----------------------------
//
// For callers that cannot allocate device memory themselves or through this library: code
// running where cudaMalloc is unavailable or forbidden (a host whose allocator owns the whole
// device, a capture-time or real-time path that must not allocate, an FFI host with a fixed
// memory budget). The multigrid hierarchy, the Krylov vectors and the solve's scalars live
// in one file-scope device array of fixed size, which every GPU that loads this library
// holds until the process exits.

constexpr int kStaticMaxCells = 512 * 288;   // the largest grid the array holds (147,456 cells)
constexpr int kStaticMinSide = 16;           // and its narrowest side

// The most any accepted grid (both sides >= 16, at most kStaticMaxCells cells) needs of each
// part of the array: hierarchy cells, tiles of the levels down to the tail, level-0 tiles.
// For a given width every count grows with the height, so the tallest grid of each width is
// the one to check. Long thin grids need the most hierarchy: once a level is one cell high,
// each further level halves only the width.
struct StaticNeed {
    int total, tiles, nwg;
};
constexpr StaticNeed static_need() {
    StaticNeed m{0, 0, 0};
    for (int w = kStaticMinSide; w <= kStaticMaxCells / kStaticMinSide; w++) {
        const int h = kStaticMaxCells / w;
        const Levels L = make_levels(w, h);
        const int nwg = ((w + 15) / 16) * ((h + 15) / 16);
        if (L.total > m.total) m.total = L.total;
        if (L.tiles > m.tiles) m.tiles = L.tiles;
        if (nwg > m.nwg) m.nwg = nwg;
    }
    return m;
}
constexpr StaticNeed kStaticNeed = static_need();
constexpr size_t kStaticTotal = (size_t)kStaticNeed.total;
constexpr size_t kStaticTiles = (size_t)kStaticNeed.tiles;
constexpr size_t kStaticNwg = (size_t)kStaticNeed.nwg;
static_assert(kStaticTotal >= (size_t)kStaticMaxCells * 4 / 3, "the hierarchy holds at least 4/3 of the grid");
constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t kStaticBytes =
    align256(sizeof(DevParams)) + align256(sizeof(StepState)) + align256(sizeof(SolveState)) +
    align256((size_t)kStaticMaxCells * sizeof(float4)) +          // rhs as the engine lays it out
    align256((size_t)kStaticMaxCells * sizeof(float)) +           // viscous part of the warm start
    align256(kStaticTiles * sizeof(uint32_t)) +                   // tile flags of every level
    align256(kStaticTiles * sizeof(uint32_t)) + align256(kMaxLevels * sizeof(uint32_t)) +   // active-tile lists
    align256(2 * kStaticNwg * sizeof(float4)) +                   // per-tile partial sums
    align256(kStaticTotal * sizeof(float4)) + align256(kStaticTotal * sizeof(float)) +
    4 * align256(kStaticTotal * sizeof(float2)) + 4 * align256((size_t)kStaticMaxCells * sizeof(float2));

static __device__ __align__(256) unsigned char g_solve_scratch[kStaticBytes];

namespace {

// Prepares a solve in the array: the level-0 matrix and right-hand side copied in, every
// coarse matrix and tile flag cleared (a call starts as the first solve of a fresh tank),
// the level-0 tile flags from the diagonal, the scalars reset.
__global__ void k_static_prep(DevScene d, const float4* mga, const float* mgd, const float2* rhs, float tol_p,
                              float tol_psi, uint32_t max_iters) {
    const int n0 = d.W * d.H;
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = t0; i < d.lv.total; i += stride) {
        if (i < n0) {
            // couplings to cells that are no unknowns count for nothing: zero in the copy, whatever
            // the caller's hold (the passes rely on their being finite)
            const int x = i % d.W, y = i / d.W;
            float4 a = mga[i];
            if (!(x > 0 && mgd[i - 1] > 0.0f)) a.x = 0.0f;
            if (!(x + 1 < d.W && mgd[i + 1] > 0.0f)) a.y = 0.0f;
            if (!(y > 0 && mgd[i - d.W] > 0.0f)) a.z = 0.0f;
            if (!(y + 1 < d.H && mgd[i + d.W] > 0.0f)) a.w = 0.0f;
            d.mga[i] = a;
            const float D = mgd[i];
            d.mgd[i] = D;
            float2 b = rhs[i];
            d.prhs[i] = make_float4(b.x, b.y, 0.0f, 0.0f);
            d.p2keep[i] = 0.0f;
            // a cell that is no unknown leaves with zero potentials, also in tiles without
            // unknowns, which the solve itself never visits
            if (!(D > 0.0f)) d.pres[i] = make_float2(0.0f, 0.0f);
        } else {
            d.mga[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            d.mgd[i] = 0.0f;
            d.mgy[i] = make_float2(0.0f, 0.0f);
        }
    }
    const int tw = (d.W + 15) / 16, th = (d.H + 15) / 16;
    for (int t = t0; t < d.lv.tiles; t += stride) {
        uint32_t on = 0u;
        if (t < tw * th) {
            const int x0 = (t % tw) * 16, y0 = (t / tw) * 16;
            for (int y = y0; y < y0 + 16 && y < d.H && !on; y++)
                for (int x = x0; x < x0 + 16 && x < d.W; x++)
                    if (mgd[y * d.W + x] > 0.0f) { on = 1u; break; }
        }
        d.ptile[t] = on;
    }
    if (t0 == 0) {
        DevParams* P = const_cast<DevParams*>(d.P);
        P->tol[0] = tol_p;
        P->tol[1] = tol_psi;
        P->pressure_max_iters = max_iters;
        d.S->dt = 1.0f;
        d.S->dt_prev = 1.0f;
        SolveState* K = d.K;
        unsigned char* k = reinterpret_cast<unsigned char*>(K);
        for (size_t b = 0; b < sizeof(SolveState); b++) k[b] = 0;
        K->cap[0] = K->cap[1] = max_iters;   // the caller's limit, not a recorded count
        K->hier = HIER_PLAIN;                // (cleared above, as the flags say)
    }
}

struct StaticSlot {
    int ready;
    unsigned char* base;
};
StaticSlot g_slots[kMaxDevices];

}  // namespace

void sprout_internal_set_error(const char* msg);

}  // namespace sprout

extern "C" int sprout_pressure_solve_static(uint32_t w, uint32_t h, const float* mga, const float* mgd, const float* rhs,
                                            float* x, float tol_p, float tol_psi, uint32_t max_iters, void* stream,
                                            uint32_t* iters_out, float* residual_out) {
    using namespace sprout;
    if (!mga || !mgd || !rhs || !x) {
        sprout_internal_set_error("null argument");
        return -1;
    }
    if (w < (uint32_t)kStaticMinSide || h < (uint32_t)kStaticMinSide || (size_t)w * h > (size_t)kStaticMaxCells) {
        sprout_internal_set_error("grid outside 16 x 16 .. 147,456 cells, the most the fixed solve array holds");
        return -3;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        sprout_internal_set_error("no current CUDA device");
        return -6;
    }
    StaticSlot& slot = g_slots[dev];
    if (!slot.ready) {
        // With this device current: the array's device address (its host-side name is only
        // a stand-in). Done on the first call on each device.
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_solve_scratch);
        if (e != cudaSuccess || ptr == nullptr) {
            sprout_internal_set_error(cudaGetErrorString(e));
            return -6;
        }
        slot.base = static_cast<unsigned char*>(ptr);
        slot.ready = 1;
    }
    const Levels L = make_levels((int)w, (int)h);
    DevScene d{};
    d.W = (int)w;
    d.H = (int)h;
    d.ncell = (int)(w * h);
    d.lv = L;
    d.nwg = (int)(((w + 15) / 16) * ((h + 15) / 16));
    unsigned char* p = slot.base;
    auto take = [&](size_t bytes) { unsigned char* q = p; p += align256(bytes); return q; };
    DevParams* P = reinterpret_cast<DevParams*>(take(sizeof(DevParams)));
    d.P = P;
    d.S = reinterpret_cast<StepState*>(take(sizeof(StepState)));
    d.K = reinterpret_cast<SolveState*>(take(sizeof(SolveState)));
    d.prhs = reinterpret_cast<float4*>(take((size_t)kStaticMaxCells * sizeof(float4)));
    d.p2keep = reinterpret_cast<float*>(take((size_t)kStaticMaxCells * sizeof(float)));
    d.ptile = reinterpret_cast<uint32_t*>(take(kStaticTiles * sizeof(uint32_t)));
    d.plist = reinterpret_cast<uint32_t*>(take(kStaticTiles * sizeof(uint32_t)));
    d.pcount = reinterpret_cast<uint32_t*>(take(kMaxLevels * sizeof(uint32_t)));
    d.partials = reinterpret_cast<float4*>(take(2 * kStaticNwg * sizeof(float4)));
    d.mga = reinterpret_cast<float4*>(take(kStaticTotal * sizeof(float4)));
    d.mgd = reinterpret_cast<float*>(take(kStaticTotal * sizeof(float)));
    d.mgy = reinterpret_cast<float2*>(take(kStaticTotal * sizeof(float2)));
    d.mgx = reinterpret_cast<float2*>(take(kStaticTotal * sizeof(float2)));
    d.mgz = reinterpret_cast<float2*>(take(kStaticTotal * sizeof(float2)));
    d.mgr = reinterpret_cast<float2*>(take(kStaticTotal * sizeof(float2)));
    d.mgr2 = reinterpret_cast<float2*>(take((size_t)kStaticMaxCells * sizeof(float2)));
    d.cgp = reinterpret_cast<float2*>(take((size_t)kStaticMaxCells * sizeof(float2)));
    d.cgp2 = reinterpret_cast<float2*>(take((size_t)kStaticMaxCells * sizeof(float2)));
    d.cgq = reinterpret_cast<float2*>(take((size_t)kStaticMaxCells * sizeof(float2)));
    d.pres = reinterpret_cast<float2*>(x);
    // (every accepted grid fits by construction of kStaticNeed; checked all the same)
    if ((size_t)(p - slot.base) > kStaticBytes || (size_t)L.total > kStaticTotal || (size_t)L.tiles > kStaticTiles ||
        (size_t)d.nwg > kStaticNwg) {
        sprout_internal_set_error("fixed solve array layout overflow");
        return -3;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_static_prep<<<128, 256, 0, st>>>(d, reinterpret_cast<const float4*>(mga), mgd, reinterpret_cast<const float2*>(rhs),
                                       tol_p, tol_psi, max_iters);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        sprout_internal_set_error(cudaGetErrorString(e));
        return -6;
    }
    const size_t smem = pressure_smem(L);
    int blocks = pressure_blocks_max(dev, smem, false);
    if (blocks > d.nwg) blocks = d.nwg;
    if (blocks < 1) blocks = 1;
    int second = 0, scale_mode = 0;
    void* args[] = {(void*)&d, &second, &scale_mode};
    e = cudaLaunchCooperativeKernel((const void*)k_mgpcg<Plain>, dim3(blocks), dim3(NT), args, smem, st);
    if (e != cudaSuccess) {
        sprout_internal_set_error(cudaGetErrorString(e));
        return -6;
    }
    if (iters_out || residual_out) {
        SolveState K;
        e = cudaMemcpyAsync(&K, d.K, sizeof K, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            sprout_internal_set_error(cudaGetErrorString(e));
            return -6;
        }
        if (K.error & ERR_DIVERGED) {
            sprout_internal_set_error("the solve met a non-finite right-hand side or residual and stopped");
            return -4;
        }
        if (K.error) {
            sprout_internal_set_error("a bounded device-side wait ran out (grid barrier of the pressure solve)");
            return -5;
        }
        if (iters_out) {
            iters_out[0] = K.p_iters[0];
            iters_out[1] = K.p_iters[1];
        }
        if (residual_out) *residual_out = K.p_bb[0] > 0.0f ? sqrtf(K.p_rr[0] / K.p_bb[0]) : 0.0f;
    }
    return 0;
}
