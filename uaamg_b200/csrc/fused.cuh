// Fused V-cycle level kernels: ONE z march for the way down through a level and
// ONE for the way up (uaamg_preconditioner_3d.cpp:183-196; 2D
// uaamg_preconditioner.cpp:162-175), instead of the four marches of march.cuh.
//
//   k_level_down  forward red-black sweep from x = 0 (smooth(L,1,false),
//                 _3d.cpp:123-141), the residual b - A x (restrictResidual,
//                 144-165) and its restriction to the coarse b.  The smoothed x
//                 is never stored: odd cells hold b/d and even cells a function of
//                 the b of their neighbours, so the block recomputes x on its tile
//                 and a 2-cell ring from the staged b, and writes only the coarse b.
//   k_level_up    prolongation x += 2 x_coarse (prolongateAdd, 168-181) and the
//                 reverse sweep (even colour, then odd), writing the final x; on
//                 the finest level also the CG's z sums (pcg_3d.cpp:112-123).
//
// Block: a 32 x 16 column tile (256 threads, each owning the cell pair (i, j),
// (i, j+1) -- one cell of each colour), marching a chunk of z planes.  Every plane
// of b, the cell codes (coarse levels: diagonal and couplings; way up: the parent
// x) arrives by TMA as a box of the tile plus a 2-cell ring, into a ring of
// shared-memory stages.  Step s of the march computes three things:
//   1. the odd-colour value of plane s+1 (tile and 2-cell ring),
//   2. the even-colour value of plane s (tile and 1-cell ring), from the odd
//      values of plane s in shared memory and plane s +- 1 in registers,
//   3. the final result of plane s-1 on the tile (way down: residual and
//      restriction; way up: the odd colour of the reverse sweep and the store).
// A z neighbour is the same column one step up or down, so each thread keeps its
// column's recent values in registers; in-plane neighbours are read from three
// shared x planes written one step earlier, so one block barrier per step
// suffices.  The first 104 threads also own a pair of ring cells (50 pairs of
// the 1-cell ring, 54 of the 2-cell ring).
//
// Arithmetic: every per-cell value is the reference's expression in its order
// (the forward even update (b + sum c_n x_n)/d, the residual b - (d x - sum c_n
// x_n), the restriction's child order), so the FP64 instantiation (built with
// -fmad=false) reproduces the reference's V-cycle bit for bit.  The FP32 forms
// take the residual of the forward sweep from its exact form: an even cell was
// just relaxed, so its residual is 0, and an odd cell's is sum_n c_n x_n over its
// (even) neighbours, since d x = b there; cells with d < 1e-30 (skipped by the
// smoother) keep r = b.
//
// STAR (the FP32 and mixed solves on covering aggregates, engine.cuh): the transfers
// between this level and the next coarser one are not constant per aggregate but
// reach its face neighbours.  A fine cell takes 2 (x_c + w sum_a (x_n - x_c)), x_n the
// coarse neighbour on the cell's own side along axis a where the coarse level couples
// the two, and the restriction is the transpose: the sum of a coarse cell's residuals
// plus w times, over its coupled faces, the difference between the residuals on the
// far and on the near side of the face.  Constant transfers overshoot in directions
// the smoother is weak in; with w = 1/5 the mixed solve of 129 x 97 x 65 with spacings
// 1 : 1.5 : 0.67 takes 15 iterations instead of 45, of 256^3 12 instead of 15.  The
// way down then needs the residual on the tile and a 1-cell ring and one plane either
// side of the chunk, so its boxes have a 3-cell ring; the way up needs the parent
// level's x in boxes one cell wider, two planes deep, and the parent's codes, whose
// low six bits say which neighbours a coarse cell is coupled to.
#pragma once
#include "march.cuh"

namespace uaamg {
namespace {

constexpr float kStarW = 0.2f;  // weight of a coupled face neighbour (1/4 is exact for linear
                                // fields; 1/5 took as many iterations or one fewer)

// Box of element type E around a tile with an R-cell ring: cells
// i in [i0-R, i0+31+R], j in [j0-R, j0+15+R] (i0 = 1 + 32 bx, j0 = 1 + 16 by) of one
// plane.  The start column 32 bx - A is a 16-byte boundary at or below i0 - R.
template <class E, int R = 2>
struct RBox {
    static constexpr int A = 16 / (int)sizeof(E);              // elements per 16 bytes
    static constexpr int W = (A + 33 + R + A - 1) / A * A;      // row width (elements)
    static constexpr int H = kMY + 2 * R;
    static constexpr uint32_t BYTES = (uint32_t)(W * H * sizeof(E));
    // position of the cell (i0 + di, j0 + dj), di in [-R, 31+R], dj in [-R, 15+R]
    __host__ __device__ static constexpr int pos(int di, int dj) { return (dj + R) * W + A + 1 + di; }
    static_assert(A >= R - 1, "the ring's first column lies in the box");
};

// STAR, way up: the parent level's x under a tile with a 2-cell ring and the face
// neighbours of those parents: coarse columns [16 bx - A, ...], of which [16 bx - 1,
// 16 bx + 18] are read, rows [8 by - 1, 8 by + 10], and in 3D the two planes kc - 1, kc
// (odd k) or kc, kc + 1 (even k), kc = (k + 1) / 2; and the parents' codes: columns
// [16 bx, 16 bx + 31], rows [8 by, 8 by + 9] of plane kc.
template <class T, int DIM>
struct SBox {
    static constexpr int A = 16 / (int)sizeof(T);
    static constexpr int W = (A + 19 + A - 1) / A * A;
    static constexpr int H = kMY / 2 + 4;
    static constexpr int PL = W * H;
    static constexpr uint32_t BYTES = (uint32_t)(PL * (DIM == 3 ? 2 : 1) * sizeof(T));
    static constexpr int CW = 32, CH = kMY / 2 + 2;
    static constexpr uint32_t CBYTES = CW * CH;
};

// Tensor maps of a fused march (boxes of RBox geometry; xc: the parent level's x
// in QBox geometry, with STAR xc and pc the parent level's x and codes in SBox geometry).
struct FMaps {
    CUtensorMap b, code, dg, cx, cy, cz, xc, pc;
};

// One ring stage: b, codes, [diagonal, couplings], [parent x, [parent codes]].
template <int DIM, class T, class CS, bool FINE, bool UP, bool STAR>
struct FPlan {
    static constexpr int R = STAR && !UP ? 3 : 2;  // ring cells of the boxes
    using BT = RBox<T, R>;
    using BC = RBox<uint8_t, R>;
    using BS = RBox<CS, R>;
    static constexpr int NC = FINE ? 0 : (DIM == 3 ? 3 : 2);
    static constexpr size_t OFF_B = 0;
    static constexpr size_t OFF_CODE = align128(BT::BYTES);
    static constexpr size_t OFF_DG = OFF_CODE + align128(BC::BYTES);
    static constexpr size_t OFF_CX = OFF_DG + (FINE ? 0 : align128(BT::BYTES));
    static constexpr size_t CB = align128(BS::BYTES);
    static constexpr size_t OFF_CY = OFF_CX + CB, OFF_CZ = OFF_CY + CB;
    static constexpr size_t OFF_XC = OFF_CX + NC * CB;
    static constexpr uint32_t XCB = STAR ? SBox<T, DIM>::BYTES : QBox<T>::BYTES;
    static constexpr size_t OFF_PC = OFF_XC + align128(XCB);
    static constexpr size_t STAGE =
        !UP ? OFF_XC : STAR ? OFF_PC + align128(SBox<T, DIM>::CBYTES) : OFF_PC;
    static constexpr uint32_t TX = BT::BYTES + BC::BYTES + (FINE ? 0u : BT::BYTES + NC * BS::BYTES) +
                                   (UP ? XCB + (STAR ? SBox<T, DIM>::CBYTES : 0u) : 0u);
};

// Ring depth and shared memory.  LAG: planes behind the step that stay resident
// (the coarse levels read the -z coupling of plane s-2 in step 3); S >= LAG + 3
// keeps the plane of the next step in flight during the current one.
template <int DIM, class T, class CS, bool FINE, bool UP, bool STAR = false>
struct FCfg {
    using P = FPlan<DIM, T, CS, FINE, UP, STAR>;
    static constexpr int LAG = FINE ? 1 : 2;
    static constexpr int S = DIM == 2 ? 1 : LAG + 3 + (FINE ? (UP ? 2 : 3) : 1);
    static constexpr int NXP = DIM == 2 ? 1 : 3;  // shared x planes
    static constexpr size_t OFF_LUT = 128;          // after the stage barriers
    // finest level in FP32: the per-code table of the branch-free cell updates
    static constexpr bool LEAN = FINE && sizeof(T) == 4;
    static constexpr size_t OFF_TAB = OFF_LUT + align128(64 * sizeof(T));
    static constexpr size_t OFF_RING = OFF_TAB + (LEAN ? 128 * sizeof(float2) : 0);
    static constexpr size_t OFF_X = OFF_RING + S * P::STAGE;
    static constexpr size_t XB = align128(P::BT::BYTES);
    // STAR, way down: the residuals of a coarse plane's two fine planes, summed over
    // them, on the tile and a 1-cell ring: cell (di, dj) at (dj + 1) RW + di + 2
    static constexpr int RW = kMX + 4;
    static constexpr size_t OFF_R = OFF_X + NXP * XB;
    static constexpr size_t BYTES = OFF_R + (STAR && !UP ? align128(RW * (kMY + 2) * sizeof(T)) : 0);
    // resident blocks per SM the finest FP32 level is compiled for (registers): 3D,
    // five on the way down (its shared memory fits five) and four on the way up (at 48
    // registers the compiler recomputed values: 256^3, 74.3 M against 58.0 M warp
    // instructions, 101 against 89 us a launch; the way down at four, 73 against
    // 69 us); 2D, eight (a full SM of 256-thread
    // blocks; the 2D way up at five blocks and 48 registers: 2048 x 1024 solve 10.24
    // against 9.99 ms)
    static constexpr int MINB = LEAN ? (DIM == 3 ? (UP ? 4 : 5) : 8) : 1;
    static_assert(S <= 16, "stage barriers: 128 bytes");
};

// A cell of a task: box positions in the T, code and coupling boxes, the parent
// box position, its global offset in a level plane, whether it lies in the level,
// and its colour on plane 0 ((i + j) & 1).
struct FCell {
    int qt, qc, qs, qq;
    int qk, side;  // STAR: the parent's code; bits 0 / 1: the cell is on its +x / +y side
    int qr;        // STAR: position in the residual buffer
    int gid;
    bool in;
    int par;
};

template <class P, class T, int DIM, bool STAR>
__device__ __forceinline__ FCell fcell(const Geom& g, int i0, int j0, int di, int dj) {
    FCell c;
    c.qt = P::BT::pos(di, dj);
    c.qc = P::BC::pos(di, dj);
    c.qs = P::BS::pos(di, dj);
    if constexpr (STAR) {
        using B = SBox<T, DIM>;
        c.qq = (((dj + 2) >> 1) + 1) * B::W + B::A + ((di + 2) >> 1);
        c.qk = ((dj + 2) >> 1) * B::CW + ((di + 2) >> 1);
        c.side = (di & 1) | ((dj & 1) << 1);
        c.qr = (dj + 1) * (kMX + 4) + di + 2;
    } else {
        c.qq = ((dj + 2) >> 1) * QBox<T>::W + ((di + 2) >> 1);
        c.qk = c.side = c.qr = 0;
    }
    const int i = i0 + di, j = j0 + dj;
    c.gid = i + j * g.sx;
    c.in = i >= 1 && i <= g.nx && j >= 1 && j <= g.ny;
    c.par = (i + j) & 1;
    return c;
}

// The ring tasks: pair t (t < 104) of the 1-cell ring (t < 50) or the 2-cell ring;
// both cells of a pair are neighbours, so they have opposite colours.
__device__ __forceinline__ void ring_pair(int t, int& d1i, int& d1j, int& d2i, int& d2j) {
    if (t < 17) { d1i = 2 * t - 1; d2i = 2 * t; d1j = d2j = -1; }
    else if (t < 34) { const int u = t - 17; d1i = 2 * u - 1; d2i = 2 * u; d1j = d2j = kMY; }
    else if (t < 42) { const int u = t - 34; d1i = d2i = -1; d1j = 2 * u; d2j = 2 * u + 1; }
    else if (t < 50) { const int u = t - 42; d1i = d2i = kMX; d1j = 2 * u; d2j = 2 * u + 1; }
    else if (t < 68) { const int u = t - 50; d1i = 2 * u - 2; d2i = 2 * u - 1; d1j = d2j = -2; }
    else if (t < 86) { const int u = t - 68; d1i = 2 * u - 2; d2i = 2 * u - 1; d1j = d2j = kMY + 1; }
    else if (t < 95) { const int u = t - 86; d1i = d2i = -2; d1j = 2 * u - 1; d2j = 2 * u; }
    else { const int u = t - 95; d1i = d2i = kMX + 1; d1j = 2 * u - 1; d2j = 2 * u; }
}
constexpr int kRing1Tasks = 50, kRingTasks = 104;

// STAR, way down: the ring tasks of thread t by whole warps, so that no warp mixes
// rings and each scheduler's two warps carry about as much: the 1-cell ring (50 pairs,
// all three phases) on warps 0 and 1, the 2-cell ring (54, two phases) on 2 and 3, the
// 3-cell ring (58, odd values only) on 6 and 7.  Returns the ring (0: none).
__device__ __forceinline__ int star_ring_pair(int t, int& d1i, int& d1j, int& d2i, int& d2j) {
    if (t < kRing1Tasks) { ring_pair(t, d1i, d1j, d2i, d2j); return 1; }
    if (t >= 64 && t < 64 + kRingTasks - kRing1Tasks) {
        ring_pair(t - 64 + kRing1Tasks, d1i, d1j, d2i, d2j);
        return 2;
    }
    if (t >= 192 && t < 192 + 58) {
        const int q = t - 192;
        if (q < 19) { d1i = 2 * q - 3; d2i = 2 * q - 2; d1j = d2j = -3; }
        else if (q < 38) { const int u = q - 19; d1i = 2 * u - 3; d2i = 2 * u - 2; d1j = d2j = kMY + 2; }
        else if (q < 48) { const int u = q - 38; d1i = d2i = -3; d1j = 2 * u - 2; d2j = 2 * u - 1; }
        else { const int u = q - 48; d1i = d2i = kMX + 2; d1j = 2 * u - 2; d2j = 2 * u - 1; }
        return 3;
    }
    return 0;
}

// Part 1 of a plane's loads: the hierarchy's constant arrays (they do not depend on the
// kernel before); part 2: b and the parent's x.  Part 1 announces the bytes of both.
template <int DIM, class T, class CS, bool FINE, bool UP, bool STAR>
__device__ __forceinline__ void f_issue1(const FMaps& M, unsigned char* st, uint64_t* bar, int k) {
    using P = FPlan<DIM, T, CS, FINE, UP, STAR>;
    const int x0 = kMX * (int)blockIdx.x, y0 = kMY * (int)blockIdx.y + 1 - P::R;
    mbar_expect_tx(bar, P::TX);
    tma_load<DIM>(st + P::OFF_CODE, &M.code, x0 - P::BC::A, y0, k, bar);
    if constexpr (!FINE) {
        tma_load<DIM>(st + P::OFF_DG, &M.dg, x0 - P::BT::A, y0, k, bar);
        tma_load<DIM>(st + P::OFF_CX, &M.cx, x0 - P::BS::A, y0, k, bar);
        tma_load<DIM>(st + P::OFF_CY, &M.cy, x0 - P::BS::A, y0, k, bar);
        if constexpr (DIM == 3) tma_load<DIM>(st + P::OFF_CZ, &M.cz, x0 - P::BS::A, y0, k, bar);
    }
    if constexpr (UP && STAR)
        tma_load<DIM>(st + P::OFF_PC, &M.pc, x0 / 2, kMY / 2 * (int)blockIdx.y, (k + 1) >> 1, bar);
}
template <int DIM, class T, class CS, bool FINE, bool UP, bool STAR>
__device__ __forceinline__ void f_issue2(const FMaps& M, unsigned char* st, uint64_t* bar, int k) {
    using P = FPlan<DIM, T, CS, FINE, UP, STAR>;
    const int x0 = kMX * (int)blockIdx.x, y0 = kMY * (int)blockIdx.y + 1 - P::R;
    tma_load<DIM>(st + P::OFF_B, &M.b, x0 - P::BT::A, y0, k, bar);
    if constexpr (UP) {
        const int yc = kMY / 2 * (int)blockIdx.y, kc = (k + 1) >> 1;
        if constexpr (STAR)
            tma_load<DIM>(st + P::OFF_XC, &M.xc, x0 / 2 - SBox<T, DIM>::A, yc - 1, kc - (k & 1), bar);
        else
            tma_load<DIM>(st + P::OFF_XC, &M.xc, x0 / 2, yc, kc, bar);
    }
}

// Planes p0 .. plast pass through S stages; plane p uses stage (p - p0) mod S.
// Thread 0 issues every load and is the only thread that waits on the barriers.
template <int DIM, class T, class CS, bool FINE, bool UP, bool STAR, int S>
struct FRing {
    using P = FPlan<DIM, T, CS, FINE, UP, STAR>;
    uint64_t* bars;
    unsigned char* base;
    int p0, plast;
    // stage of plane p (p >= p0 - S; planes below p0 are never read)
    __device__ unsigned char* at(int p) const {
        return base + (size_t)((p - p0 + 2 * S) % S) * P::STAGE;
    }
    __device__ bool wait(int p) const {
        const int u = p - p0;
        return mbar_wait(&bars[u % S], (uint32_t)((u / S) & 1), kTmaWaitLimit);
    }
    // the first S planes: barriers and part 1, then part 2
    __device__ void start1(const FMaps& M) const {
        for (int s = 0; s < S; ++s) mbar_init(&bars[s], 1);
        fence_proxy_async();
        for (int p = p0; p < p0 + S && p <= plast; ++p)
            f_issue1<DIM, T, CS, FINE, UP, STAR>(M, at(p), &bars[(p - p0) % S], p);
    }
    __device__ void start2(const FMaps& M) const {
        for (int p = p0; p < p0 + S && p <= plast; ++p)
            f_issue2<DIM, T, CS, FINE, UP, STAR>(M, at(p), &bars[(p - p0) % S], p);
    }
    // a block that stops at once waits for the loads it started
    __device__ bool drain() const {
        bool ok = true;
        for (int p = p0; p < p0 + S && p <= plast; ++p) ok = wait(p) && ok;
        return ok;
    }
    // after a block barrier: plane `freed` is no longer read; load plane freed + S
    __device__ void refill(const FMaps& M, int freed) const {
        if (freed >= p0 && freed + S <= plast) {
            fence_proxy_async();
            uint64_t* bar = &bars[(freed - p0) % S];
            f_issue1<DIM, T, CS, FINE, UP, STAR>(M, at(freed + S), bar, freed + S);
            f_issue2<DIM, T, CS, FINE, UP, STAR>(M, at(freed + S), bar, freed + S);
        }
    }
};

// Recent values of one column: the last two odd-colour values and the last
// even-colour value computed for it.
template <class T>
struct FHist {
    T o1, o2, e1;
};

// The dynamic shared memory of a fused march (128-byte aligned; see march.cuh).
#define UAAMG_FUSED_SMEM(sm, err)                                                 \
    extern __shared__ __align__(128) unsigned char smem_raw[];                   \
    unsigned char* sm = smem_raw;                                                \
    if (smem_u32(sm) & 127u) {                                                   \
        if (threadIdx.x == 0) atomicExch(err, 2);                                \
        pdl_wait();                                                              \
        return;                                                                  \
    }

template <int DIM, class T, bool FINE, class CS, bool UP, bool ZDOT, bool STAR = false>
__global__ void __launch_bounds__(kThreads, (FCfg<DIM, T, CS, FINE, UP, STAR>::MINB))
    k_level_fused(const __grid_constant__ FMaps M, MLevel<T> L, T* __restrict__ out,
                  const int* __restrict__ done, int* err, double* partials, CGState* cg) {
    using C = FCfg<DIM, T, CS, FINE, UP, STAR>;
    using P = typename C::P;
    constexpr int S = C::S, WT = P::BT::W, WS = P::BS::W;
    constexpr bool kStarDn = STAR && !UP;
    static_assert(!STAR || sizeof(T) == 4, "the FP64 form keeps the reference's transfers");
    static_assert(!STAR || !FINE, "quad.cuh runs the finest level with STAR transfers");
    constexpr bool kFull = sizeof(T) == 8;  // the reference's residual expression
    UAAMG_FUSED_SMEM(sm, err)
    T* lut = reinterpret_cast<T*>(sm + C::OFF_LUT);
    const Geom& g = L.g;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = 1 + kMX * (int)blockIdx.x, j0 = 1 + kMY * (int)blockIdx.y;
    int kb, ke;
    if constexpr (UP) zrange<DIM>(g, L.zc, kb, ke);
    else zrange_restrict<DIM>(g, L.cg, L.zc, kb, ke);
    // 3D: steps s = s0 .. sl: odd values of planes kb-2 .. ke+1, even values of kb-1 ..
    // ke, final results of kb .. ke-1 (a STAR way down: final results of kb-1 .. ke, so one
    // step more at either end); 2D: the one plane 0
    constexpr int X = kStarDn ? 1 : 0;
    const int s0 = kb - 3 - X, sl = ke + X;
    const FRing<DIM, T, CS, FINE, UP, STAR, S> R{reinterpret_cast<uint64_t*>(sm), sm + C::OFF_RING,
                                                 DIM == 3 ? s0 + 1 : 0, DIM == 3 ? sl + 1 : 0};
    if (tid == 0) {
        tma_prefetch(&M.b);
        if constexpr (UP) tma_prefetch(&M.xc);
        R.start1(M);
    }
    if (FINE) build_lut<DIM, T>(lut, L.idx2, L.idy2, L.idz2);
    // Finest level in FP32 (no Dirichlet walls: those problems take the four-march
    // level): every cell update is a multiply-add driven by the table entry of its
    // code's low 7 bits (neighbour bits, interior-fluid bit): x = 1/d for an interior
    // fluid cell the smoother relaxes (d >= 1e-30), else 0; y = 1 for an interior
    // fluid cell it skips (d < 1e-30), else 0.
    constexpr bool LEAN = C::LEAN;
    const float2* tab = reinterpret_cast<const float2*>(sm + C::OFF_TAB);
    if constexpr (LEAN) {
        if (tid < 128) {
            const uint32_t c = (uint32_t)tid;
            float d = ((c & 1u) ? (float)L.idx2 : 0.f) + ((c & 2u) ? (float)L.idx2 : 0.f) +
                      ((c & 4u) ? (float)L.idy2 : 0.f) + ((c & 8u) ? (float)L.idy2 : 0.f);
            if (DIM == 3) d = d + ((c & 16u) ? (float)L.idz2 : 0.f) + ((c & 32u) ? (float)L.idz2 : 0.f);
            const bool act = (c & kActive) != 0, skip = act && d < 1e-30f;
            float2 e;
            e.x = act && !skip ? mdiv<float, CS>(1.0f, d) : 0.f;
            e.y = skip ? 1.f : 0.f;
            reinterpret_cast<float2*>(sm + C::OFF_TAB)[tid] = e;
        }
    }

    // --- per-cell arithmetic --------------------------------------------------
    auto code_at = [&](const unsigned char* st, const FCell& c) -> uint32_t {
        return st[P::OFF_CODE + c.qc];
    };
    auto b_at = [&](const unsigned char* st, const FCell& c) -> T {
        return reinterpret_cast<const T*>(st + P::OFF_B)[c.qt];
    };
    // (a finest level with Dirichlet walls never runs here: no wall diagonal)
    auto diag_of = [&](const unsigned char* st, const FCell& c, uint32_t code, int k) -> T {
        if constexpr (FINE) {
            return lut[code & 63u];
        } else {
            return reinterpret_cast<const T*>(st + P::OFF_DG)[c.qt];
        }
    };
    // couplings +x, -x, +y, -y, +z, -z (stc: this plane, stm: the plane below)
    auto coup = [&](const unsigned char* stc, const unsigned char* stm, const FCell& c, T (&cc)[6]) {
        if constexpr (FINE) {
            cc[0] = cc[1] = L.idx2;
            cc[2] = cc[3] = L.idy2;
            cc[4] = cc[5] = L.idz2;
        } else {
            const CS* cx = reinterpret_cast<const CS*>(stc + P::OFF_CX);
            const CS* cy = reinterpret_cast<const CS*>(stc + P::OFF_CY);
            cc[0] = coupling<T, CS>(cx[c.qs], L.csx);
            cc[1] = coupling<T, CS>(cx[c.qs - 1], L.csx);
            cc[2] = coupling<T, CS>(cy[c.qs], L.csy);
            cc[3] = coupling<T, CS>(cy[c.qs - WS], L.csy);
            if constexpr (DIM == 3) {
                cc[4] = coupling<T, CS>(reinterpret_cast<const CS*>(stc + P::OFF_CZ)[c.qs], L.csz);
                cc[5] = coupling<T, CS>(reinterpret_cast<const CS*>(stm + P::OFF_CZ)[c.qs], L.csz);
            } else {
                cc[4] = cc[5] = T(0);
            }
        }
    };
    // sum c_n v_n in the reference's order (v: a shared x plane)
    auto nbsum2 = [&](const T (&cc)[6], const T* v, int q, T vp, T vm) -> T {
        T nb = cc[0] * v[q + 1] + cc[1] * v[q - 1] + cc[2] * v[q + WT] + cc[3] * v[q - WT];
        if (DIM == 3) nb = nb + cc[4] * vp + cc[5] * vm;
        return nb;
    };
    // kodd: the plane is odd (3D), i.e. the cell is on its parent's -z side
    auto prolong = [&](const unsigned char* st, const FCell& c, auto kodd) -> T {
        const T* xc = reinterpret_cast<const T*>(st + P::OFF_XC);
        if constexpr (STAR) {
            using B = SBox<T, DIM>;
            constexpr bool KO = decltype(kodd)::value;
            constexpr int own = DIM == 3 && KO ? B::PL : 0, oth = DIM == 3 && !KO ? B::PL : 0;
            const uint32_t pc = st[P::OFF_PC + c.qk];
            const bool px = c.side & 1, py = c.side & 2;
            const T xo = xc[own + c.qq];
            T g = (pc & (px ? 1u : 2u)) ? xc[own + c.qq + (px ? 1 : -1)] - xo : T(0);
            g += (pc & (py ? 4u : 8u)) ? xc[own + c.qq + (py ? B::W : -B::W)] - xo : T(0);
            if constexpr (DIM == 3) g += (pc & (KO ? 32u : 16u)) ? xc[oth + c.qq] - xo : T(0);
            return T(2) * (xo + T(kStarW) * g);
        } else {
            return T(2) * xc[c.qq];
        }
    };
    // odd-colour value at plane k: pre-smoothed (b + 0)/d, plus the prolongation on
    // the way up; 0 on cells that are not interior fluid
    auto oval = [&](const unsigned char* st, const FCell& c, int k, auto kodd) -> T {
        if constexpr (LEAN) {
            const uint32_t code = code_at(st, c);
            const float2 t = tab[code & 127u];
            if constexpr (UP) return b_at(st, c) * t.x + ((code & kActive) ? prolong(st, c, kodd) : T(0));
            else return b_at(st, c) * t.x;
        }
        const uint32_t code = code_at(st, c);
        if (!(code & kActive)) return T(0);
        const T d = diag_of(st, c, code, k);
        const T pre = d < T(1e-30) ? T(0) : mdiv<T, CS>(b_at(st, c) + T(0), d);
        if constexpr (UP) return pre + prolong(st, c, kodd);
        else return pre;
    };
    // even-colour value at plane k from the odd values around it: forward sweep
    // (way down) or first colour of the reverse sweep (way up; a skipped cell keeps
    // 0 + the prolongation)
    auto evalc = [&](const unsigned char* st, const unsigned char* stm, const T* xv, const FCell& c,
                     int k, T op, T om, auto kodd) -> T {
        if constexpr (LEAN) {
            const float2 t = tab[code_at(st, c) & 127u];
            const int q = c.qt;
            T nb = L.idx2 * (xv[q + 1] + xv[q - 1]) + L.idy2 * (xv[q + WT] + xv[q - WT]);
            if (DIM == 3) nb = nb + L.idz2 * (op + om);
            if constexpr (UP) return (b_at(st, c) + nb) * t.x + t.y * prolong(st, c, kodd);
            else return (b_at(st, c) + nb) * t.x;
        }
        const uint32_t code = code_at(st, c);
        if (!(code & kActive)) return T(0);
        const T d = diag_of(st, c, code, k);
        if (d < T(1e-30)) {
            if constexpr (UP) return T(0) + prolong(st, c, kodd);
            else return T(0);
        }
        T cc[6];
        coup(st, stm, c, cc);
        return mdiv<T, CS>(b_at(st, c) + nbsum2(cc, xv, c.qt, op, om), d);
    };

    // --- tasks ---------------------------------------------------------------
    // tile pair: A = (i0 + lane, j0 + 2w), B = (i0 + lane, j0 + 2w + 1)
    const FCell cA = fcell<P, T, DIM, STAR>(g, i0, j0, lane, 2 * w);
    const FCell cB = fcell<P, T, DIM, STAR>(g, i0, j0, lane, 2 * w + 1);
    // this thread's ring pair: ring: it has one; ring_e: with even values; ring_f: with
    // final results (the 1-cell ring of a STAR way down)
    bool ring, ring_e, ring_f = false;
    FCell cR1, cR2;
    {
        int d1i = 0, d1j = 0, d2i = 0, d2j = 0;
        if constexpr (kStarDn) {
            const int r = star_ring_pair(tid, d1i, d1j, d2i, d2j);
            ring = r > 0;
            ring_e = r == 1 || r == 2;
            ring_f = r == 1;
        } else {
            ring = tid < kRingTasks;
            ring_e = tid < kRing1Tasks;
            if (ring) ring_pair(tid, d1i, d1j, d2i, d2j);
        }
        cR1 = fcell<P, T, DIM, STAR>(g, i0, j0, d1i, d1j);
        cR2 = fcell<P, T, DIM, STAR>(g, i0, j0, d2i, d2j);
    }
    T* xpl = reinterpret_cast<T*>(sm + C::OFF_X);
    double acc[3] = {0.0, 0.0, 0.0};
    const int ic = kMX / 2 * (int)blockIdx.x + 1 + (lane >> 1);
    const int jc = kMY / 2 * (int)blockIdx.y + 1 + w;
    const bool writer = !UP && (lane & 1) == 0 && ic <= L.cg.nx && jc <= L.cg.ny;

    // Final values of a pair at a plane, in colour order: cO / cE are its odd and even
    // cells there, vO / vE their x values, zp* / zm* their columns' values one plane up and
    // down.  resO / resE: the final x (way up) or the residuals (way down).
    auto finals = [&](const unsigned char* st, const unsigned char* stm, const T* xv, int k,
                      const FCell& cO, const FCell& cE, T vO, T vE, T zpO, T zmO, T zpE, T zmE,
                      T& resO, T& resE) {
        const uint32_t kO = code_at(st, cO), kE = code_at(st, cE);
        resO = UP ? vO : T(0);
        resE = UP ? vE : T(0);
        if constexpr (LEAN) {
            const float2 tO = tab[kO & 127u];
            const int q = cO.qt;
            T nb = L.idx2 * (xv[q + 1] + xv[q - 1]) + L.idy2 * (xv[q + WT] + xv[q - WT]);
            if (DIM == 3) nb = nb + L.idz2 * (zpO + zmO);
            if constexpr (UP) {
                resO = (b_at(st, cO) + nb) * tO.x + tO.y * vO;  // a skipped cell keeps vO
            } else {
                const float2 tE = tab[kE & 127u];
                resO = (tO.x != 0.f ? nb : T(0)) + tO.y * b_at(st, cO);
                resE = tE.y * b_at(st, cE);
            }
        } else if (kO & kActive) {  // odd cell: reverse-sweep update / residual
            const T d = diag_of(st, cO, kO, k);
            if constexpr (UP) {
                if (!(d < T(1e-30))) {
                    T cc[6];
                    coup(st, stm, cO, cc);
                    resO = mdiv<T, CS>(b_at(st, cO) + nbsum2(cc, xv, cO.qt, zpO, zmO), d);
                }
            } else if constexpr (kFull) {
                T cc[6];
                coup(st, stm, cO, cc);
                T ax = d * vO - cc[0] * xv[cO.qt + 1] - cc[1] * xv[cO.qt - 1] -
                       cc[2] * xv[cO.qt + WT] - cc[3] * xv[cO.qt - WT];
                if (DIM == 3) ax = ax - cc[4] * zpO - cc[5] * zmO;
                resO = b_at(st, cO) - ax;
            } else {
                if (d < T(1e-30)) {
                    resO = b_at(st, cO);
                } else {
                    T cc[6];
                    coup(st, stm, cO, cc);
                    resO = nbsum2(cc, xv, cO.qt, zpO, zmO);
                }
            }
        }
        if constexpr (!UP && !LEAN) {
            if (kE & kActive) {  // even cell: residual (0 after its relaxation in FP32)
                const T d = diag_of(st, cE, kE, k);
                if constexpr (kFull) {
                    T cc[6];
                    coup(st, stm, cE, cc);
                    T ax = d * vE - cc[0] * xv[cE.qt + 1] - cc[1] * xv[cE.qt - 1] -
                           cc[2] * xv[cE.qt + WT] - cc[3] * xv[cE.qt - WT];
                    if (DIM == 3) ax = ax - cc[4] * zpE - cc[5] * zmE;
                    resE = b_at(st, cE) - ax;
                } else {
                    if (d < T(1e-30)) resE = b_at(st, cE);
                }
            }
        }
    };

    // Final step on the tile pair at plane k (finals); aOdd: A is the odd cell.  rlo: the
    // way down's dk = 0 residuals, kept from the odd plane below.
    auto final_pair = [&](auto kodd, const unsigned char* st, const unsigned char* stm, const T* xv,
                          int k, const FCell& cO, const FCell& cE, bool aOdd, T vO, T vE, T zpO,
                          T zmO, T zpE, T zmE, T (&rlo)[2]) {
        [[maybe_unused]] constexpr bool KODD = decltype(kodd)::value;  // plane k is odd (3D)
        T resO, resE;
        finals(st, stm, xv, k, cO, cE, vO, vE, zpO, zmO, zpE, zmE, resO, resE);
        const uint32_t kO = code_at(st, cO), kE = code_at(st, cE);
        if constexpr (UP) {
            const int base = k * g.sxy;
            const bool inO = cO.in, inE = cE.in;
            if (inO) out[cO.gid + base] = resO;
            if (inE) out[cE.gid + base] = resE;
            if (ZDOT) {
                if constexpr (LEAN) {
                    // z and b are 0 on every cell that is not interior fluid (ghosts,
                    // padding and cells past the level included)
                    const double zo = (double)resO, ro = (double)b_at(st, cO);
                    const double ze = (double)resE, re = (double)b_at(st, cE);
                    acc[0] += zo;
                    acc[1] += ro * zo;
                    acc[2] += ro;
                    acc[0] += ze;
                    acc[1] += re * ze;
                    acc[2] += re;
                } else {
                    if ((kO & kActive) && inO) {
                        const double zv = (double)resO, rv = (double)b_at(st, cO);
                        acc[0] += zv;
                        acc[1] += rv * zv;
                        acc[2] += rv;
                    }
                    if ((kE & kActive) && inE) {
                        const double zv = (double)resE, rv = (double)b_at(st, cE);
                        acc[0] += zv;
                        acc[1] += rv * zv;
                        acc[2] += rv;
                    }
                }
            }
        } else {
            const T res[2] = {aOdd ? resO : resE, aOdd ? resE : resO};  // [dj]
            // restriction: children dk = 0 on odd planes; the set is complete on the
            // even plane that follows (2D: one plane)
            if (DIM == 3 && KODD) {
                rlo[0] = res[0];
                rlo[1] = res[1];
            } else {
                T pr[2][2];  // the di = 1 partner's values [dj][dk]
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    pr[e][0] = __shfl_down_sync(0xffffffffu, DIM == 3 ? rlo[e] : res[e], 1);
                    pr[e][1] = __shfl_down_sync(0xffffffffu, res[e], 1);
                }
                if (writer) {
                    const int kc = DIM == 3 ? k / 2 : 0;
                    const int cid = cidx(L.cg, ic, jc, kc);
                    T sum = T(0);
                    if (DIM == 3) {
                        sum += rlo[0]; sum += res[0]; sum += rlo[1]; sum += res[1];
                        sum += pr[0][0]; sum += pr[0][1]; sum += pr[1][0]; sum += pr[1][1];
                    } else {
                        sum += res[0]; sum += res[1];
                        sum += pr[0][1]; sum += pr[1][1];
                    }
                    // also written on solid coarse cells, where no kernel reads b
                    out[cid] = sum;
                }
            }
        }
    };

    // STAR, way down.  rbuf holds the residuals summed over a coarse plane's two fine
    // planes on the tile and its 1-cell ring; a writer lane (an even column) forms its
    // coarse cell's sum and adds w times, per coupled face, the far minus the near
    // side's sums; zt: the two z faces' part, the same way.
    T* rbuf = reinterpret_cast<T*>(sm + C::OFF_R);
    uint32_t ccode = 0;  // code of this writer's coarse cell of the plane in progress
    auto star_write = [&](int kc, T zt) {
        constexpr int RW = C::RW;
        const T* r0 = rbuf + (2 * w + 1) * RW + lane + 2;  // row dj = 2 w, column lane
        const T a0 = r0[0], a1 = r0[1], b0 = r0[RW], b1 = r0[RW + 1];
        T q = (ccode & 2u) ? (r0[-1] + r0[RW - 1]) - (a0 + b0) : T(0);
        q += (ccode & 1u) ? (r0[2] + r0[RW + 2]) - (a1 + b1) : T(0);
        q += (ccode & 8u) ? (r0[-RW] + r0[1 - RW]) - (a0 + a1) : T(0);
        q += (ccode & 4u) ? (r0[2 * RW] + r0[2 * RW + 1]) - (b0 + b1) : T(0);
        out[cidx(L.cg, ic, jc, kc)] = ((a0 + a1) + (b0 + b1)) + T(kStarW) * (q + zt);
    };
    T rlo[2] = {T(0), T(0)};
    // from here on the previous kernel's results: b, the parent's x, the stop flag (read
    // beside the loads, whose blocks then only wait for what they started)
    pdl_wait();
    bool ok = true;
    const int stop = done ? ld_now(done) : 0;
    if (tid == 0) R.start2(M);
    pdl_launch();
    if (stop) {
        if (tid == 0 && !R.drain()) atomicExch(err, 1);
        return;
    }
    if (tid == 0) ok = R.wait(R.p0);
    if (!step_barrier(ok, err)) return;
    if constexpr (DIM == 2) {
        // one plane: odd values, barrier, even values, barrier, final
        unsigned char* st = sm + C::OFF_RING;
        // A is odd when i + j is odd; ring pairs likewise
        const bool oddA = cA.par != 0;
        const FCell tO = oddA ? cA : cB, tE = oddA ? cB : cA;
        const bool odd1 = cR1.par != 0;
        const FCell rO = odd1 ? cR1 : cR2, rE = odd1 ? cR2 : cR1;
        const std::false_type even;
        const T ot = oval(st, tO, 0, even);
        xpl[tO.qt] = ot;
        T otr = T(0), etr = T(0);
        if (ring) {
            otr = oval(st, rO, 0, even);
            xpl[rO.qt] = otr;
        }
        __syncthreads();
        const T et = evalc(st, st, xpl, tE, 0, T(0), T(0), even);
        xpl[tE.qt] = et;
        if (ring_e) {
            etr = evalc(st, st, xpl, rE, 0, T(0), T(0), even);
            xpl[rE.qt] = etr;
        }
        __syncthreads();
        if constexpr (kStarDn) {
            T rA, rB;
            if (writer) ccode = L.ccode[cidx(L.cg, ic, jc, 0)];
            finals(st, st, xpl, 0, tO, tE, ot, et, T(0), T(0), T(0), T(0), rA, rB);
            rbuf[tO.qr] = rA;
            rbuf[tE.qr] = rB;
            if (ring_f) {
                finals(st, st, xpl, 0, rO, rE, otr, etr, T(0), T(0), T(0), T(0), rA, rB);
                rbuf[rO.qr] = rA;
                rbuf[rE.qr] = rB;
            }
            __syncthreads();
            if (writer) star_write(0, T(0));
        } else {
            final_pair(even, st, st, xpl, 0, tO, tE, oddA, ot, et, T(0), T(0), T(0), T(0), rlo);
        }
    } else {
        // role 0 is the cell that is even on planes s0, s0+2, ... (odd on s0+1, ...)
        const bool aRole0 = ((cA.par + s0) & 1) == 0;
        const FCell t0 = aRole0 ? cA : cB, t1 = aRole0 ? cB : cA;
        const bool r1Role0 = ((cR1.par + s0) & 1) == 0;
        const FCell q0 = r1Role0 ? cR1 : cR2, q1 = r1Role0 ? cR2 : cR1;
        FHist<T> ht[2] = {{T(0), T(0), T(0)}, {T(0), T(0), T(0)}};
        T hr[2] = {T(0), T(0)};  // ring columns: last odd value
        // STAR way down: the ring columns' last even value and dk = 0 residuals (by role),
        // the tile pair's residual sum on the even plane below, and on the z face below
        // the coarse plane in progress the difference of the two sides' sums
        T he[2] = {T(0), T(0)}, hlo[2] = {T(0), T(0)}, te = T(0), gz = T(0);
        // stages of planes s+1, s, s-1, s-2 and the shared x planes s+1, s, s-1,
        // rotated once per step (planes below p0 are never read)
        const unsigned char* ring_end = sm + C::OFF_RING + S * P::STAGE;
        const unsigned char* sp1 = R.at(s0 + 1);
        const unsigned char* s00 = R.at(s0);
        const unsigned char* sm1 = R.at(s0 - 1);
        const unsigned char* sm2 = R.at(s0 - 2);
        T* xn = xpl + (size_t)((s0 + 4) % 3) * (C::XB / sizeof(T));
        T* xc = xpl + (size_t)((s0 + 3) % 3) * (C::XB / sizeof(T));
        T* xo = xpl + (size_t)((s0 + 5) % 3) * (C::XB / sizeof(T));
        // one step; R0c: the role whose cell is even at plane s; PHc: the phases it runs
        // (2: odd and even values, 3: all three; 0: decided at run time from s) --
        // compile-time
        auto step = [&](int s, auto R0c, auto PHc) -> bool {
            constexpr int RC = decltype(R0c)::value, RO = 1 - RC, PH = decltype(PHc)::value;
            const bool run_even = PH == 0 ? s >= kb - 1 : PH >= 2;
            const bool run_final = PH == 0 ? s >= kb + 1 : PH == 3;
            // planes s+1 and s-1 are odd, plane s is even, or the other way round (s0 is
            // even, for a STAR way down odd)
            using Odd1 = std::integral_constant<bool, (RC == 0) != (X != 0)>;
            using Odd0 = std::integral_constant<bool, !Odd1::value>;
            const FCell& tc = RC == 0 ? t0 : t1;
            const FCell& qc = RC == 0 ? q0 : q1;
            // 1. odd values of plane s+1
            const T on = oval(sp1, tc, s + 1, Odd1());
            xn[tc.qt] = on;
            T onr = T(0);
            if (ring) {
                onr = oval(sp1, qc, s + 1, Odd1());
                xn[qc.qt] = onr;
            }
            // 2. even values of plane s
            T en = T(0), enr = T(0);
            if (run_even) {
                en = evalc(s00, sm1, xc, tc, s, on, ht[RC].o1, Odd0());
                xc[tc.qt] = en;
                if (ring_e) {
                    enr = evalc(s00, sm1, xc, qc, s, onr, hr[RC], Odd0());
                    xc[qc.qt] = enr;
                }
            }
            // 3. final results of plane s-1: the role-RC cell is odd there
            if constexpr (kStarDn) {
                if (run_final) {
                    const int p = s - 1;
                    constexpr bool KODD = Odd1::value;
                    T rO, rE;
                    finals(sm1, sm2, xo, p, tc, RC == 0 ? t1 : t0, ht[RC].o1, ht[RO].e1, en, ht[RC].e1,
                           ht[RO].o1, ht[RO].o2, rO, rE);
                    const T t = rO + rE;
                    if constexpr (KODD) {  // dk = 0; the coarse plane below is complete
                        const T g = te - t;
                        if (p > kb) {
                            T zt = ((ccode & 32u) ? gz : T(0)) - ((ccode & 16u) ? g : T(0));
                            const uint32_t cn = __shfl_up_sync(0xffffffffu, ccode, 1);
                            const T zo = ((cn & 32u) ? gz : T(0)) - ((cn & 16u) ? g : T(0));
                            zt += __shfl_down_sync(0xffffffffu, zo, 1);
                            if (writer) star_write((p - 1) / 2, zt);
                        }
                        gz = g;
                        rlo[RC] = rO;
                        rlo[RO] = rE;
                    } else {  // dk = 1: the sums over both planes
                        te = t;
                        rbuf[tc.qr] = rlo[RC] + rO;
                        rbuf[(RC == 0 ? t1 : t0).qr] = rlo[RO] + rE;
                        if (writer) ccode = L.ccode[cidx(L.cg, ic, jc, p / 2)];
                    }
                    if (ring_f) {
                        const FCell& qo = RC == 0 ? q1 : q0;
                        finals(sm1, sm2, xo, p, qc, qo, T(0), T(0), enr, he[RC], T(0), T(0), rO, rE);
                        if constexpr (KODD) {
                            hlo[RC] = rO;
                            hlo[RO] = rE;
                        } else {
                            rbuf[qc.qr] = hlo[RC] + rO;
                            rbuf[qo.qr] = hlo[RO] + rE;
                        }
                    }
                }
                he[RC] = enr;
            } else if (run_final) {
                const int p = s - 1;
                const T vR = ht[RC].o1, vO = ht[RO].e1;   // x at p
                const T zpR = en, zmR = ht[RC].e1;         // role RC: even values at p+1, p-1
                const T zpO = ht[RO].o1, zmO = ht[RO].o2;  // role RO: odd values at p+1, p-1
                const FCell& to = RC == 0 ? t1 : t0;
                final_pair(Odd1(), sm1, sm2, xo, p, tc, to,
                           aRole0 == (RC == 0), vR, vO, zpR, zmR, zpO, zmO, rlo);
            }
            ht[RC].o2 = ht[RC].o1;
            ht[RC].o1 = on;
            ht[RC].e1 = en;
            hr[RC] = onr;
            sm2 = sm1;
            sm1 = s00;
            s00 = sp1;
            sp1 += P::STAGE;
            if (sp1 == ring_end) sp1 = sm + C::OFF_RING;
            {
                T* t = xo;
                xo = xc;
                xc = xn;
                xn = t;
            }
            bool okk = true;
            if (tid == 0 && s + 2 <= R.plast) okk = R.wait(s + 2);
            if (!step_barrier(okk, err)) return false;
            if (tid == kRefill) R.refill(M, s - C::LAG);
            return true;
        };
        using R0 = std::integral_constant<int, 0>;
        using R1 = std::integral_constant<int, 1>;
        if constexpr (UP) {
            // one loop, phases by s (fewer registers than two loops here)
#pragma unroll 1
            for (int s = s0; s <= ke; s += 2) {
                if (!step(s, R0(), std::integral_constant<int, 0>())) return;
                if (s + 1 <= ke && !step(s + 1, R1(), std::integral_constant<int, 0>())) return;
            }
        } else {
            // four steps fill the pipeline: odd and even values only (the even values of
            // the first two planes are not needed; their shared positions are written
            // again before any read); then two or more steps run all three
#pragma unroll 1
            for (int s = s0; s < s0 + 4; s += 2) {
                if (!step(s, R0(), std::integral_constant<int, 2>())) return;
                if (!step(s + 1, R1(), std::integral_constant<int, 2>())) return;
            }
#pragma unroll 1
            for (int s = s0 + 4; s <= sl; s += 2) {
                if (!step(s, R0(), std::integral_constant<int, 3>())) return;
                if (s + 1 <= sl && !step(s + 1, R1(), std::integral_constant<int, 3>())) return;
            }
        }
    }
    if constexpr (UP && ZDOT) {
        double tot[3];
        ZdotIn in;
        if (reduce_last<3>(acc, partials, &cg->counter[2], tot, [&] { in.load(cg); }))
            finish_zdot(cg, in, tot);
    }
}

// ---------------------------------------------------------------------------
// Small 3D levels (a few 8^3 tiles): the same two steps per level as whole-tile
// boxes instead of z marches, whose pipeline never fills on a handful of planes.  A
// block owns an 8 x 8 x 8 tile; one TMA load per array brings the tile and a 2-cell
// ring (12^3 cells) into shared memory; then (1) the odd-colour values on the whole
// box, (2) the even-colour values on the tile and the inner ring, (3) the final
// results on the tile (way down: residual and restriction; way up: odd colour of
// the reverse sweep, the store, and on the finest level the z sums), with one block
// barrier between the phases.  Per-cell expressions are those of k_level_fused.
constexpr int kBT = 8;               // tile edge

// Box of element type E: cells i in [i0-R, i0+7+R] (i0 = 1 + 8 bx; R = 2, on the STAR way
// down 3), the start column 8 bx - A rounded to 16 bytes; 8 + 2 R rows and planes.
template <class E, int R = 2>
struct BBox {
    static constexpr int A = 16 / (int)sizeof(E);
    static constexpr int N = kBT + 2 * R;  // box edge
    static constexpr int W = (A + kBT + R + 1 + A - 1) / A * A;
    static constexpr uint32_t BYTES = (uint32_t)(W * N * N * sizeof(E));
    __host__ __device__ static constexpr int pos(int di, int dj, int dk) {
        return ((dk + R) * N + (dj + R)) * W + A + 1 + di;
    }
};
// Parent box (coarse x under the box): coarse cells [4 bx, 4 bx + 5] per axis.
template <class T>
struct BQBox {
    static constexpr int W = (6 * (int)sizeof(T) + 15) / 16 * 16 / (int)sizeof(T);
    static constexpr uint32_t BYTES = (uint32_t)(W * 6 * 6 * sizeof(T));
};
// STAR: parent box with the parents' face neighbours: coarse columns [4 bx - 4, ...], of
// which [4 bx - 1, 4 bx + 6] are read, rows and planes [4 by - 1, 4 by + 6]; and the
// parents' codes: columns from the 16-byte boundary at or below 4 bx, rows and planes
// [4 by, 4 by + 5].
template <class T>
struct BSBox {
    static constexpr int W = 12, N = 8;
    static constexpr uint32_t BYTES = (uint32_t)(W * N * N * sizeof(T));
    static constexpr int CW = 32, CN = 6;
    static constexpr uint32_t CBYTES = CW * CN * CN;
};

template <class T, class CS, bool FINE, bool UP, bool STAR = false>
struct BPlan {
    static constexpr int R = STAR && !UP ? 3 : 2;
    using BT = BBox<T, R>;
    using BC = BBox<uint8_t, R>;
    using BS = BBox<CS, R>;
    static constexpr uint32_t XCB = STAR ? BSBox<T>::BYTES : BQBox<T>::BYTES;
    static constexpr size_t OFF_B = 0;
    static constexpr size_t OFF_CODE = align128(BT::BYTES);
    static constexpr size_t OFF_DG = OFF_CODE + align128(BC::BYTES);
    static constexpr size_t CB = align128(BS::BYTES);
    static constexpr size_t OFF_CX = OFF_DG + (FINE ? 0 : align128(BT::BYTES));
    static constexpr size_t OFF_CY = OFF_CX + CB, OFF_CZ = OFF_CY + CB;
    static constexpr size_t OFF_XC = OFF_CX + (FINE ? 0 : 3 * CB);
    static constexpr size_t OFF_PC = OFF_XC + (UP ? align128(XCB) : 0);
    static constexpr size_t OFF_X = OFF_PC + (UP && STAR ? align128(BSBox<T>::CBYTES) : 0);
    // STAR, way down: residuals on the tile and its 1-cell ring
    static constexpr int RN = kBT + 2;
    static constexpr size_t OFF_R = OFF_X + align128(BT::BYTES);
    static constexpr size_t OFF_BAR = OFF_R + (STAR && !UP ? align128(RN * RN * RN * sizeof(T)) : 0);
    static constexpr size_t OFF_LUT = OFF_BAR + 128;
    static constexpr size_t BYTES = OFF_LUT + align128(64 * sizeof(T));
    // the parent x and codes are loaded for trimmed boxes too
    static constexpr uint32_t TXP = UP ? XCB + (STAR ? BSBox<T>::CBYTES : 0u) : 0u;
    static constexpr uint32_t TX =
        BT::BYTES + BC::BYTES + (FINE ? 0u : BT::BYTES + 3 * BS::BYTES) + TXP;
};

// Tensor maps of a box kernel: b, codes, diagonal, couplings (BBox geometry), and the
// parent level's x (BQBox geometry; STAR: x and codes in BSBox geometry).
struct BMaps {
    CUtensorMap b, code, dg, cx, cy, cz, xc, pc;
    // coarse levels: per box the default stencil {d, c_x, c_y, c_z} (as T) when every
    // cell of the box and its 2-cell ring is interior fluid with that diagonal and
    // those couplings (a trimmed box), else d = 0 (k_box_trim); null: no trimming
    const void* trim;
};

// Trimming of a coarse box level (the reference's tile trimming,
// cuda_uaamg_preconditioner_3d.cu:81-99 and :357-375, on this kernel's 8^3 tiles): a
// box whose 12^3 cells (tile and 2-cell ring) are all interior fluid and share one
// diagonal and one coupling per axis needs none of its diagonal, coupling or code
// boxes: the box kernel loads b (and the parent x) only and uses the four values.
// The values are the stored ones, so results are identical with and without
// trimming.  One block of 256 threads per box; rec[4 box + 0] = d or 0.  (Boxes with a
// 2-cell ring: the solves' STAR boxes are not trimmed.)
template <class E>
__device__ __forceinline__ bool same_bits(E a, E b) {
    if constexpr (sizeof(E) == 2) return __half_as_ushort(a) == __half_as_ushort(b);
    else if constexpr (sizeof(E) == 4) return __float_as_uint(a) == __float_as_uint(b);
    else return __double_as_longlong(a) == __double_as_longlong(b);
}

template <class T, class CS>
__global__ void __launch_bounds__(256) k_box_trim(Geom g, const uint8_t* __restrict__ code,
                                                  const T* __restrict__ dg, const CS* __restrict__ cx,
                                                  const CS* __restrict__ cy, const CS* __restrict__ cz,
                                                  T csx, T csy, T csz, T* rec) {
    pdl_entry();
    const int i0 = 1 + kBT * (int)blockIdx.x, j0 = 1 + kBT * (int)blockIdx.y,
              k0 = 1 + kBT * (int)blockIdx.z;
    constexpr int lo = 2, hi = kBT + 1, nb = BBox<T>::N;
    const bool inside = i0 - lo >= 1 && j0 - lo >= 1 && k0 - lo >= 1 && i0 + hi <= g.nx &&
                        j0 + hi <= g.ny && k0 + hi <= g.nz;
    bool ok = inside;
    T d0 = T(0);
    CS x0{}, y0{}, z0{};
    if (inside) {
        const int id0 = cidx(g, i0, j0, k0);
        d0 = dg[id0];
        x0 = cx[id0];
        y0 = cy[id0];
        z0 = cz[id0];
        ok = !(d0 < T(1e-30));
        for (int c = threadIdx.x; ok && c < nb * nb * nb; c += blockDim.x) {
            const int i = i0 - lo + c % nb, j = j0 - lo + (c / nb) % nb, k = k0 - lo + c / (nb * nb);
            const int id = cidx(g, i, j, k);
            ok = (code[id] & kActive) && same_bits(dg[id], d0) && same_bits(cx[id], x0) &&
                 same_bits(cy[id], y0) && same_bits(cz[id], z0);
        }
    }
    ok = __syncthreads_and(ok) != 0;
    if (threadIdx.x == 0) {
        const size_t r = 4 * (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
        rec[r] = ok ? d0 : T(0);
        rec[r + 1] = ok ? coupling<T, CS>(x0, csx) : T(0);
        rec[r + 2] = ok ? coupling<T, CS>(y0, csy) : T(0);
        rec[r + 3] = ok ? coupling<T, CS>(z0, csz) : T(0);
    }
}

template <class T, bool FINE, class CS, bool UP, bool ZDOT, bool STAR = false>
__global__ void __launch_bounds__(kThreads)
    k_level_box(const __grid_constant__ BMaps M, MLevel<T> L, T* __restrict__ out,
                const int* __restrict__ done, int* err, double* partials, CGState* cg) {
    using P = BPlan<T, CS, FINE, UP, STAR>;
    using BT = typename P::BT;
    using BC = typename P::BC;
    using BS = typename P::BS;
    constexpr int R = P::R, BN = BT::N;          // ring, box edge
    constexpr int WT = BT::W, WS = BS::W;
    constexpr int PT = WT * BN, PS = WS * BN;  // plane strides
    constexpr bool kStarDn = STAR && !UP;
    static_assert(!STAR || sizeof(T) == 4, "the FP64 form keeps the reference's transfers");
    constexpr bool kFull = sizeof(T) == 8;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* sm = smem_raw;
    if (smem_u32(sm) & 127u) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        pdl_wait();
        return;
    }
    const Geom& g = L.g;
    const int tid = threadIdx.x;
    const int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
    const int i0 = 1 + kBT * bx, j0 = 1 + kBT * by, k0 = 1 + kBT * bz;
    T* lut = reinterpret_cast<T*>(sm + P::OFF_LUT);
    T* xs = reinterpret_cast<T*>(sm + P::OFF_X);
    const T* bs = reinterpret_cast<const T*>(sm + P::OFF_B);
    const unsigned char* cs = sm + P::OFF_CODE;
    const T* dgs = reinterpret_cast<const T*>(sm + P::OFF_DG);
    const CS* cxs = reinterpret_cast<const CS*>(sm + P::OFF_CX);
    const CS* cys = reinterpret_cast<const CS*>(sm + P::OFF_CY);
    const CS* czs = reinterpret_cast<const CS*>(sm + P::OFF_CZ);
    const T* xcs = reinterpret_cast<const T*>(sm + P::OFF_XC);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + P::OFF_BAR);
    if (FINE) build_lut<3, T>(lut, L.idx2, L.idy2, L.idz2);
    // a trimmed coarse box: its default stencil (d > 0), read before any load
    T trim[4] = {T(0), T(0), T(0), T(0)};
    if constexpr (!FINE) {
        if (M.trim) {
            const T* r = reinterpret_cast<const T*>(M.trim) + 4 * ((bz * gridDim.y + by) * gridDim.x + bx);
#pragma unroll
            for (int q = 0; q < 4; ++q) trim[q] = r[q];
        }
    }
    const bool tr = !FINE && trim[0] != T(0);
    // The code box starts at the 16-byte boundary at or below its first column (x0 + 1 - R
    // in the padded array): x0 - 16 when bx is even, x0 - 8 when it is odd.  Every other
    // box starts at x0 - A, a 16-byte boundary for its element size.
    const int aC = kBT * bx - 16 * ((kBT * bx + 1 - R) >> 4);
    static_assert(16 + kBT + R < BC::W, "code box: tile and ring at the widest offset");
    // likewise the parents' codes (STAR): from the boundary at or below 4 bx
    const int aP = (kBT / 2 * bx) & 15;
    static_assert(12 + 6 <= BSBox<T>::CW, "parent code box at the widest offset");
    bool ok = true;
    if (tid == 0) {
        mbar_init(bar, 1);
        const int x0 = kBT * bx, y0 = kBT * by + 1 - R, z0 = kBT * bz + 1 - R;
        fence_proxy_async();
        constexpr uint32_t kTrimTX = BT::BYTES + P::TXP;
        mbar_expect_tx(bar, tr ? kTrimTX : P::TX);
        // the hierarchy's constant arrays, ahead of the wait for the previous kernel
        tma_prefetch(&M.b);
        if constexpr (UP) tma_prefetch(&M.xc);
        if (!tr) {
            tma_load<3>(sm + P::OFF_CODE, &M.code, x0 - aC, y0, z0, bar);
            if constexpr (!FINE) {
                tma_load<3>(sm + P::OFF_DG, &M.dg, x0 - BT::A, y0, z0, bar);
                tma_load<3>(sm + P::OFF_CX, &M.cx, x0 - BS::A, y0, z0, bar);
                tma_load<3>(sm + P::OFF_CY, &M.cy, x0 - BS::A, y0, z0, bar);
                tma_load<3>(sm + P::OFF_CZ, &M.cz, x0 - BS::A, y0, z0, bar);
            }
        }
        const int xp = kBT / 2 * bx, yp = kBT / 2 * by, zp = kBT / 2 * bz;
        if constexpr (UP && STAR) tma_load<3>(sm + P::OFF_PC, &M.pc, xp - aP, yp, zp, bar);
        pdl_wait();
        tma_load<3>(sm + P::OFF_B, &M.b, x0 - BT::A, y0, z0, bar);
        if constexpr (UP && STAR) tma_load<3>(sm + P::OFF_XC, &M.xc, xp - 4, yp - 1, zp - 1, bar);
        else if constexpr (UP) tma_load<3>(sm + P::OFF_XC, &M.xc, xp, yp, zp, bar);
    } else {
        pdl_wait();
    }
    const int stop = done ? ld_now(done) : 0;
    pdl_launch();
    if (tid == 0) ok = mbar_wait(bar, 0u, kTmaWaitLimit);
    if (!step_barrier(ok, err)) return;
    if (stop) return;

    // per-cell helpers on box offsets (di, dj, dk) in [-R, 7 + R]
    auto qT = [](int di, int dj, int dk) { return BT::pos(di, dj, dk); };
    auto qC = [aC](int di, int dj, int dk) { return BC::pos(di, dj, dk) - BC::A + aC; };
    auto qS = [](int di, int dj, int dk) { return BS::pos(di, dj, dk); };
    auto nbsum = [&](const T (&cc)[6], int q) -> T {
        return cc[0] * xs[q + 1] + cc[1] * xs[q - 1] + cc[2] * xs[q + WT] + cc[3] * xs[q - WT] +
               cc[4] * xs[q + PT] + cc[5] * xs[q - PT];
    };
    auto prolong = [&](int di, int dj, int dk) -> T {
        if constexpr (STAR) {
            using B = BSBox<T>;
            const int pi = (di + 2) >> 1, pj = (dj + 2) >> 1, pk = (dk + 2) >> 1;
            const int q = ((pk + 1) * B::N + pj + 1) * B::W + pi + 4;
            const uint32_t pc = sm[P::OFF_PC + (pk * B::CN + pj) * B::CW + pi + aP];
            const T xo = xcs[q];
            T g = (pc & ((di & 1) ? 1u : 2u)) ? xcs[q + ((di & 1) ? 1 : -1)] - xo : T(0);
            g += (pc & ((dj & 1) ? 4u : 8u)) ? xcs[q + ((dj & 1) ? B::W : -B::W)] - xo : T(0);
            g += (pc & ((dk & 1) ? 16u : 32u)) ? xcs[q + ((dk & 1) ? B::N * B::W : -B::N * B::W)] - xo
                                              : T(0);
            return T(2) * (xo + T(kStarW) * g);
        }
        return T(2) * xcs[(((dk + 2) >> 1) * 6 + ((dj + 2) >> 1)) * BQBox<T>::W + ((di + 2) >> 1)];
    };
    // colour of a box cell: (i + j + k) & 1 with i0 + j0 + k0 odd
    const int par0 = (i0 + j0 + k0) & 1;

    // The three steps; TR: a trimmed box (every cell interior fluid, the stencil in
    // trim[]), whose codes, diagonals and couplings were not loaded.
    auto run = [&](auto trimc) {
        constexpr bool TR = decltype(trimc)::value;
        auto code_at = [&](int di, int dj, int dk) -> uint32_t {
            if constexpr (TR) return kActive;
            else return cs[qC(di, dj, dk)];
        };
        auto diag = [&](uint32_t code, int q) -> T {
            if constexpr (TR) return trim[0];
            else if constexpr (FINE) return lut[code & 63u];
            else return dgs[q];
        };
        auto coup = [&](int qs, T (&cc)[6]) {
            if constexpr (TR) {
                cc[0] = cc[1] = trim[1];
                cc[2] = cc[3] = trim[2];
                cc[4] = cc[5] = trim[3];
            } else if constexpr (FINE) {
                cc[0] = cc[1] = L.idx2;
                cc[2] = cc[3] = L.idy2;
                cc[4] = cc[5] = L.idz2;
            } else {
                cc[0] = coupling<T, CS>(cxs[qs], L.csx);
                cc[1] = coupling<T, CS>(cxs[qs - 1], L.csx);
                cc[2] = coupling<T, CS>(cys[qs], L.csy);
                cc[3] = coupling<T, CS>(cys[qs - WS], L.csy);
                cc[4] = coupling<T, CS>(czs[qs], L.csz);
                cc[5] = coupling<T, CS>(czs[qs - PS], L.csz);
            }
        };

        // Cells are enumerated by colour: the rows (dj, dk) of a region hold
        // alternating colours, so the k-th cell of a colour in a row is di = first +
        // 2 m + s with s fixed by the row's parity.  A thread steps its enumeration
        // index by the block size, updating (m, row) incrementally.
        static_assert(kThreads == 256, "incremental colour enumeration assumes 256 threads");
        // 1. odd values on the whole box: BN^2 rows of BN cells, H = BN / 2 odd per row; a
        // step of 256 is SK planes, SJ rows and SM cells (BN = 12: 3, 6 and 4)
        {
            constexpr int H = BN / 2, SM = 256 % H, SJ = 256 / H % BN, SK = 256 / H / BN;
            int m = tid % H, jj = (tid / H) % BN, kk = tid / (H * BN);
            while (kk < BN) {
                const int dj = jj - R, dk = kk - R;
                const int di = -R + 2 * m + ((1 + dj + dk + par0 + R) & 1);
                const int q = qT(di, dj, dk);
                const uint32_t code = code_at(di, dj, dk);
                T v = T(0);
                if (code & kActive) {
                    const T d = diag(code, q);
                    v = d < T(1e-30) ? T(0) : mdiv<T, CS>(bs[q] + T(0), d);
                    if constexpr (UP) v = v + prolong(di, dj, dk);
                }
                xs[q] = v;
                m += SM;
                jj += SJ;
                kk += SK;
                if (m >= H) { m -= H; jj += 1; }
                if (jj >= BN) { jj -= BN; kk += 1; }
            }
        }
        __syncthreads();
        // 2. even values on the tile and all rings but the outermost: EN = BN - 2 (BN = 12:
        // a step of 256 is 5 planes, 1 row and 1 cell)
        {
            constexpr int EN = BN - 2, H = EN / 2, SM = 256 % H, SJ = 256 / H % EN, SK = 256 / H / EN;
            int m = tid % H, jj = (tid / H) % EN, kk = tid / (H * EN);
            while (kk < EN) {
                const int dj = jj - (R - 1), dk = kk - (R - 1);
                const int di = -(R - 1) + 2 * m + ((1 + dj + dk + par0 + R) & 1);
                const int q = qT(di, dj, dk);
                const uint32_t code = code_at(di, dj, dk);
                T v = T(0);
                if (code & kActive) {
                    const T d = diag(code, q);
                    if (d < T(1e-30)) {
                        if constexpr (UP) v = T(0) + prolong(di, dj, dk);
                    } else {
                        T cc[6];
                        coup(qS(di, dj, dk), cc);
                        v = mdiv<T, CS>(bs[q] + nbsum(cc, q), d);
                    }
                }
                xs[q] = v;
                m += SM;
                jj += SJ;
                kk += SK;
                if (m >= H) { m -= H; jj += 1; }
                if (jj >= EN) { jj -= EN; kk += 1; }
            }
        }
        __syncthreads();
        // 3. final results on the tile: thread = the x pair (2 m, 2 m + 1) of row (dj,
        // dk); u = 0 its odd cell, u = 1 its even cell (no lane diverges on colour)
        double acc[3] = {0.0, 0.0, 0.0};
        if constexpr (kStarDn) {
            // residuals of the tile and the six faces of its 1-cell ring; even cells were
            // just relaxed (0, or b where the smoother skips them)
            constexpr int RN = P::RN;
            T* rr = reinterpret_cast<T*>(sm + P::OFF_R);
            auto resid = [&](int di, int dj, int dk, bool odd) {
                const int q = qT(di, dj, dk);
                const uint32_t code = code_at(di, dj, dk);
                T v = T(0);
                if (code & kActive) {
                    if (diag(code, q) < T(1e-30)) {
                        v = bs[q];
                    } else if (odd) {
                        T cc[6];
                        coup(qS(di, dj, dk), cc);
                        v = nbsum(cc, q);
                    }
                }
                rr[((dk + 1) * RN + dj + 1) * RN + di + 1] = v;
            };
            {  // thread = the x pair (2 m, 2 m + 1) of row (dj, dk)
                const int pm = tid & 3, pj = (tid >> 2) & 7, pk = tid >> 5;
                const int sO = (1 + pj + pk + par0) & 1;  // the odd cell is di = 2 pm + sO
                resid(2 * pm + sO, pj, pk, true);
                resid(2 * pm + 1 - sO, pj, pk, false);
            }
            for (int t = tid; t < 6 * 32; t += kThreads) {  // pairs of the faces
                const int f = t >> 5, m = (t & 31) >> 3, r = t & 7;
                const int e = (f & 1) ? kBT : -1;
                int di, dj, dk;
                if (f < 2) { di = e; dj = 2 * m; dk = r; }
                else if (f < 4) { dj = e; di = 2 * m; dk = r; }
                else { dk = e; di = 2 * m; dj = r; }
                const int o = (1 + di + dj + dk + par0) & 1;  // 1: the pair's second cell is odd
                // (i + j + k and di + dj + dk + par0 have one parity)
                const int si = f < 2 ? 0 : 1, sj = f < 2 ? 1 : 0;
                resid(di + si * o, dj + sj * o, dk, true);
                resid(di + si * (1 - o), dj + sj * (1 - o), dk, false);
            }
            __syncthreads();
            if (tid < (kBT / 2) * (kBT / 2) * (kBT / 2)) {
                const int ci = tid % 4, cj = (tid / 4) % 4, ck = tid / 16;
                const int ic = kBT / 2 * bx + 1 + ci, jc = kBT / 2 * by + 1 + cj,
                          kc = kBT / 2 * bz + 1 + ck;
                if (ic <= L.cg.nx && jc <= L.cg.ny && kc <= L.cg.nz) {
                    const int cid = cidx(L.cg, ic, jc, kc);
                    const uint32_t cc = L.ccode[cid];
                    const T* r0 = rr + ((2 * ck + 1) * RN + 2 * cj + 1) * RN + 2 * ci + 1;
                    auto four = [&](int o, int a, int b2) {  // a face's four cells from offset o
                        return (r0[o] + r0[o + a]) + (r0[o + b2] + r0[o + a + b2]);
                    };
                    constexpr int X = 1, Y = RN, Z = RN * RN;
                    const T xl = four(0, Y, Z), xr = four(X, Y, Z);
                    T q = (cc & 2u) ? four(-X, Y, Z) - xl : T(0);
                    q += (cc & 1u) ? four(2 * X, Y, Z) - xr : T(0);
                    q += (cc & 8u) ? four(-Y, X, Z) - four(0, X, Z) : T(0);
                    q += (cc & 4u) ? four(2 * Y, X, Z) - four(Y, X, Z) : T(0);
                    q += (cc & 32u) ? four(-Z, X, Y) - four(0, X, Y) : T(0);
                    q += (cc & 16u) ? four(2 * Z, X, Y) - four(Z, X, Y) : T(0);
                    out[cid] = (xl + xr) + T(kStarW) * q;
                }
            }
            return;
        }
        T* rs = reinterpret_cast<T*>(sm + P::OFF_B);  // way down: residuals replace b (tile only)
        T res[2];
        int resq[2];
        const int pm = tid & 3, pj = (tid >> 2) & 7, pk = tid >> 5;
        const int sO = (1 + pj + pk + par0) & 1;  // the odd cell is di = 2 pm + sO
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool odd = u == 0;
            const int di = 2 * pm + (u == 0 ? sO : 1 - sO), dj = pj, dk = pk;
            const int q = qT(di, dj, dk);
            const uint32_t code = code_at(di, dj, dk);
            const T x0 = xs[q];
            T v = UP ? x0 : T(0);
            if (code & kActive) {
                const T d = diag(code, q);
                if constexpr (UP) {
                    if (odd && !(d < T(1e-30))) {
                        T cc[6];
                        coup(qS(di, dj, dk), cc);
                        v = mdiv<T, CS>(bs[q] + nbsum(cc, q), d);
                    }
                } else if constexpr (kFull) {
                    T cc[6];
                    coup(qS(di, dj, dk), cc);
                    const T ax = d * x0 - cc[0] * xs[q + 1] - cc[1] * xs[q - 1] - cc[2] * xs[q + WT] -
                                 cc[3] * xs[q - WT] - cc[4] * xs[q + PT] - cc[5] * xs[q - PT];
                    v = bs[q] - ax;
                } else {
                    if (d < T(1e-30)) {
                        v = bs[q];
                    } else if (odd) {
                        T cc[6];
                        coup(qS(di, dj, dk), cc);
                        v = nbsum(cc, q);
                    }
                }
            }
            res[u] = v;
            resq[u] = q;
            if constexpr (UP) {
                const int i = i0 + di, j = j0 + dj, k = k0 + dk;
                if (i <= g.nx && j <= g.ny && k <= g.nz) {
                    out[cidx(g, i, j, k)] = v;
                    if (ZDOT && (code & kActive)) {
                        const double zv = (double)v, rv = (double)bs[q];
                        acc[0] += zv;
                        acc[1] += rv * zv;
                        acc[2] += rv;
                    }
                }
            }
        }
        if constexpr (!UP) {
            __syncthreads();  // every b of the tile has been read
#pragma unroll
            for (int u = 0; u < 2; ++u) rs[resq[u]] = res[u];
            __syncthreads();
            // restriction: 4^3 coarse cells, the 2x2x2 children in (di, dj, dk) order
            if (tid < (kBT / 2) * (kBT / 2) * (kBT / 2)) {
                const int ci = tid % 4, cj = (tid / 4) % 4, ck = tid / 16;
                const int ic = kBT / 2 * bx + 1 + ci, jc = kBT / 2 * by + 1 + cj,
                          kc = kBT / 2 * bz + 1 + ck;
                if (ic <= L.cg.nx && jc <= L.cg.ny && kc <= L.cg.nz) {
                    T sum = T(0);
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
                            for (int e = 0; e < 2; ++e) sum += rs[qT(2 * ci + a, 2 * cj + b2, 2 * ck + e)];
                    // also written on solid coarse cells, where no kernel reads b
                    out[cidx(L.cg, ic, jc, kc)] = sum;
                }
            }
        }
        if constexpr (UP && ZDOT) {
            double tot[3];
            ZdotIn in;
        if (reduce_last<3>(acc, partials, &cg->counter[2], tot, [&] { in.load(cg); }))
            finish_zdot(cg, in, tot);
        }
    };
    if constexpr (FINE) {
        run(std::false_type{});
    } else {
        if (tr) run(std::true_type{});
        else run(std::false_type{});
    }
}

#undef UAAMG_FUSED_SMEM

}  // namespace
}  // namespace uaamg
