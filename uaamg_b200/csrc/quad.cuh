// The finest level's V-cycle marches of the FP32 and mixed solves (STAR transfers,
// fused.cuh), four cells of a row a thread.
//
// k_level_fused gives a thread one vertical cell pair of the tile and lets some threads
// own ring pairs beside it: 184 (way down) and 264 (way up) warp instructions a plane,
// most of them addresses, table look-ups and single-word shared-memory accesses, on
// marches that are bound by instruction issue (large levels) or by one step's chain of
// them (middle ones).  Here a thread owns a quad, four consecutive cells 4 m .. 4 m + 3 of
// a row, and the block's 2 x 128 threads cover the tile and its ring alike, every thread
// running the same phases (values outside a phase's region are computed from whatever is
// there and never used).  A quad holds two cells of each colour, which alternate with the
// row and the plane; rows of one parity share a thread group, so the colours' positions
// are the same for a whole warp.  The two colours' values are kept apart: in shared
// memory the odd (O) and the even (E) cells of a row lie packed, so a quad's neighbours
// in y are one 8-byte load, in x its own pair and one word, in z its own registers; and
// the arithmetic runs on pairs (add / mul / fma.f32x2).  b and the codes of a plane are
// read once, 16 and 4 bytes a quad, and carried in registers through the three phases,
// so a ring stage is free after one step.  1/d comes from a table by code only where the
// quad is not interior fluid on all sides.
//
// The phases of step s are those of k_level_fused: odd values of plane s+1, even values
// of plane s, final results of plane s-1, one block barrier a step.  Per-cell values are
// the same expressions up to rounding, except that a fluid cell without any coupling
// (d < 1e-30) counts as solid: z = 0 there, and its residual is not restricted.
#pragma once
#include "fused.cuh"

namespace uaamg {
namespace {

constexpr int kQuads = 10;  // quads of a row: columns [i0 - 5, i0 + 34]
constexpr int kPackW = 26;  // row stride of a packed colour plane (words): the 8-byte loads
                            // of a half warp, which spans rows of one parity, hit all banks

struct F2 {
    float x, y;
};
__device__ __forceinline__ unsigned long long f2_bits(F2 a) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a.x), "f"(a.y));
    return v;
}
__device__ __forceinline__ F2 f2_of(unsigned long long v) {
    F2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(v));
    return a;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return f2_of(v);
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(f2_bits(a)), "l"(f2_bits(b)));
    return f2_of(v);
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    unsigned long long v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
    return f2_of(v);
}

template <int DIM, class CS, bool UP>
struct QCfg {
    using P = FPlan<DIM, float, CS, true, UP, true>;
    static constexpr int R = P::R;
    static constexpr int ROWS = kMY + 2 * R;
    static constexpr int S = DIM == 2 ? 1 : 4;  // a stage is read in one step only
    static constexpr size_t OFF_TAB = 128;
    static constexpr size_t OFF_RING = OFF_TAB + 128 * sizeof(float);
    // packed colour planes with a row of padding before and after; 3D: O and E alternate
    // between two each
    static constexpr int PLANE = (ROWS + 2) * kPackW + 2;
    static constexpr size_t OFF_PK = OFF_RING + S * P::STAGE;
    static constexpr int NPK = DIM == 2 ? 2 : 4;
    // way down: residuals of the tile and its 1-cell ring in natural order, cell (di, dj)
    // at (dj + 1) 40 + di + 5; 3D: of two coarse planes in turn
    static constexpr int RB = (kMY + 2) * 4 * kQuads;
    static constexpr size_t OFF_R = OFF_PK + align128(NPK * PLANE * sizeof(float));
    static constexpr size_t BYTES = OFF_R + (UP ? 0 : (DIM == 2 ? 1 : 2) * align128(RB * sizeof(float)));
    static_assert(ROWS / 2 * kQuads <= 128, "a row parity's quads fit its thread group");
};

template <int DIM, class CS, bool UP, bool ZDOT>
__global__ void __launch_bounds__(kThreads, DIM == 3 ? (UP ? 3 : 4) : 5)
    k_level_quad(const __grid_constant__ FMaps M, MLevel<float> L, float* __restrict__ out,
                 const int* __restrict__ done, int* err, double* partials, CGState* cg) {
    using T = float;
    using C = QCfg<DIM, CS, UP>;
    using P = typename C::P;
    constexpr int R = C::R, S = C::S;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* sm = smem_raw;
    if (smem_u32(sm) & 127u) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        pdl_wait();
        return;
    }
    const Geom& g = L.g;
    const int tid = threadIdx.x;
    int kb, ke;
    if constexpr (UP) zrange<DIM>(g, L.zc, kb, ke);
    else zrange_restrict<DIM>(g, L.cg, L.zc, kb, ke);
    // steps and planes as k_level_fused
    constexpr int X = UP ? 0 : 1;
    const int s0 = kb - 3 - X, sl = ke + X;
    const FRing<DIM, T, CS, true, UP, true, S> RG{reinterpret_cast<uint64_t*>(sm), sm + C::OFF_RING,
                                                  DIM == 3 ? s0 + 1 : 0, DIM == 3 ? sl + 1 : 0};
    if (tid == 0) {
        tma_prefetch(&M.b);
        if constexpr (UP) tma_prefetch(&M.xc);
        RG.start1(M);
    }
    float* tab = reinterpret_cast<float*>(sm + C::OFF_TAB);
    if (tid < 128) {  // 1/d by code: 0 unless an interior fluid cell with a coupling
        const uint32_t c = (uint32_t)tid;
        float d = ((c & 1u) ? L.idx2 : 0.f) + ((c & 2u) ? L.idx2 : 0.f) + ((c & 4u) ? L.idy2 : 0.f) +
                  ((c & 8u) ? L.idy2 : 0.f);
        if (DIM == 3) d = d + ((c & 16u) ? L.idz2 : 0.f) + ((c & 32u) ? L.idz2 : 0.f);
        tab[tid] = (c & kActive) && !(d < 1e-30f) ? mdiv<float, CS>(1.0f, d) : 0.f;
    }
    // the code of a cell with all neighbours, four times, and its 1/d
    constexpr uint32_t kFullCode = DIM == 3 ? 0x7f7f7f7fu : 0x4f4f4f4fu;
    const float dfull = DIM == 3 ? L.idx2 + L.idx2 + L.idy2 + L.idy2 + L.idz2 + L.idz2
                                 : L.idx2 + L.idx2 + L.idy2 + L.idy2;
    const float rfull = mdiv<float, CS>(1.0f, dfull);

    // this thread's quad: row r (of parity grp) of the box, quad q of the row
    const int grp = tid >> 7, l = tid & 127;
    const int m = l / kQuads, q = l - kQuads * m;
    const bool live = m < C::ROWS / 2;
    const int r = live ? 2 * m + grp : grp, dj = r - R;
    const bool trow = live && dj >= 0 && dj < kMY;        // a tile row
    const bool frow = live && dj >= -1 && dj <= kMY;      // a row with residuals
    // word offsets: b in its box, codes in theirs (bytes), the pair in a packed plane
    const int ob = r * P::BT::W + 4 * q, oc = r * P::BC::W + P::BC::A - 4 + 4 * q;
    const int op = (r + 1) * kPackW + 2 * q + 1;  // (a plane starts at an odd word: 8-byte aligned)
    float* pk = reinterpret_cast<float*>(sm + C::OFF_PK);
    const F2 ix{L.idx2, L.idx2}, iy{L.idy2, L.idy2}, iz{L.idz2, L.idz2};

    struct Quad {
        F2 o, e;    // b of the odd and the even cells
        F2 ro, re;  // their 1/d
    };
    // Odd cells sit at e = PO, PO + 2 of the quad.
    auto split = [](const float4& v, auto po, F2& o, F2& e) {
        if constexpr (decltype(po)::value == 0) {
            o = F2{v.x, v.z};
            e = F2{v.y, v.w};
        } else {
            o = F2{v.y, v.w};
            e = F2{v.x, v.z};
        }
    };
    auto rcp4 = [&](uint32_t c, float4& v) {
        v = make_float4(rfull, rfull, rfull, rfull);
        if ((c & 0x7f7f7f7fu) != kFullCode) {
            v.x = tab[c & 127u];
            v.y = tab[(c >> 8) & 127u];
            v.z = tab[(c >> 16) & 127u];
            v.w = tab[(c >> 24) & 127u];
        }
    };
    // 2 (x_c + w sum (x_n - x_c)) of the two odd cells from the staged parent planes; PO as
    // above, KO: the plane is odd (the cells are on their parents' -z side)
    auto prolong2 = [&](const unsigned char* st, auto po, auto kodd) -> F2 {
        using B = SBox<T, DIM>;
        constexpr int PO = decltype(po)::value;
        constexpr bool KO = decltype(kodd)::value;
        const T* xc = reinterpret_cast<const T*>(st + P::OFF_XC);
        constexpr int own = DIM == 3 && KO ? B::PL : 0, oth = DIM == 3 && !KO ? B::PL : 0;
        // parents c0 (cell 0), c0 + 1 (cells 1, 2), c0 + 2 (cell 3); row (dj + 2) >> 1
        const int pr = (dj + 2) >> 1;
        const int a = (pr + 1) * B::W + B::A - 2 + 2 * q + PO;  // the odd cells' parents: a, a + 1
        const unsigned char* pcs = st + P::OFF_PC + pr * B::CW - 2 + 2 * q + PO;
        const uint32_t c0 = pcs[0], c1 = pcs[1];
        const T o0 = xc[own + a], o1 = xc[own + a + 1];
        // x neighbour: + side (PO = 0) or - side
        const T x0 = PO == 0 ? o1 : xc[own + a - 1], x1 = PO == 0 ? xc[own + a + 2] : o0;
        const int ys = (dj & 1) ? B::W : -B::W;
        const T y0 = xc[own + a + ys], y1 = xc[own + a + 1 + ys];
        T z0 = T(0), z1 = T(0);
        if constexpr (DIM == 3) {
            z0 = xc[oth + a];
            z1 = xc[oth + a + 1];
        }
        constexpr uint32_t mx = PO == 0 ? 1u : 2u, mz = DIM == 3 ? (KO ? 32u : 16u) : 0u;
        const uint32_t my = (dj & 1) ? 4u : 8u, all = mx | my | mz;
        F2 v;
        if ((c0 & c1 & all) == all) {
            constexpr float wc = DIM == 3 ? 2.f * (1.f - 3.f * kStarW) : 2.f * (1.f - 2.f * kStarW);
            F2 n = add2(F2{x0, x1}, F2{y0, y1});
            if constexpr (DIM == 3) n = add2(n, F2{z0, z1});
            v = fma2(F2{2.f * kStarW, 2.f * kStarW}, n, mul2(F2{wc, wc}, F2{o0, o1}));
        } else {
            T g0 = (c0 & mx) ? x0 - o0 : T(0), g1 = (c1 & mx) ? x1 - o1 : T(0);
            g0 += (c0 & my) ? y0 - o0 : T(0);
            g1 += (c1 & my) ? y1 - o1 : T(0);
            if constexpr (DIM == 3) {
                g0 += (c0 & mz) ? z0 - o0 : T(0);
                g1 += (c1 & mz) ? z1 - o1 : T(0);
            }
            v = F2{T(2) * (o0 + T(kStarW) * g0), T(2) * (o1 + T(kStarW) * g1)};
        }
        return v;
    };
    // phase 1: the staged plane: b and 1/d by colour, the odd cells' values into `plane`
    auto odd_phase = [&](const unsigned char* st, float* plane, auto po, auto kodd, Quad& Q) -> F2 {
        const float4 b4 = *reinterpret_cast<const float4*>(reinterpret_cast<const T*>(st + P::OFF_B) + ob);
        const uint32_t c = *reinterpret_cast<const uint32_t*>(st + P::OFF_CODE + oc);
        float4 r4;
        rcp4(c, r4);
        split(b4, po, Q.o, Q.e);
        split(r4, po, Q.ro, Q.re);
        F2 v{Q.o.x * Q.ro.x, Q.o.y * Q.ro.y};
        if constexpr (UP) {
            const F2 p = prolong2(st, po, kodd);
            v.x = Q.ro.x != 0.f ? v.x + p.x : v.x;
            v.y = Q.ro.y != 0.f ? v.y + p.y : v.y;
        }
        *reinterpret_cast<float2*>(plane + op) = make_float2(v.x, v.y);
        return v;
    };
    // (b + nb) / d of a pair
    auto relax = [](F2 b, F2 nb, F2 rd) -> F2 { return F2{(b.x + nb.x) * rd.x, (b.y + nb.y) * rd.y}; };
    // sum c_n x_n of the pair at positions NP, NP + 2 (NP = 0 or 1) over the other colour's
    // packed plane; mine: that colour's pair of this quad, zs: the z neighbours' sum
    auto nbsum = [&](const float* plane, auto np, F2 mine, F2 zs) -> F2 {
        const float2 yd = *reinterpret_cast<const float2*>(plane + op - kPackW);
        const float2 yu = *reinterpret_cast<const float2*>(plane + op + kPackW);
        // x neighbours: positions 0, 2: (prev, 1), (1, 3); positions 1, 3: (0, 2), (2, next)
        const float mid = mine.x + mine.y;
        F2 n;
        if constexpr (decltype(np)::value == 0) n = F2{plane[op - 1] + mine.x, mid};
        else n = F2{mid, mine.y + plane[op + 2]};
        n = mul2(ix, n);
        n = fma2(iy, add2(F2{yd.x, yd.y}, F2{yu.x, yu.y}), n);
        if constexpr (DIM == 3) n = fma2(iz, zs, n);
        return n;
    };

    const int i4 = kMX * (int)blockIdx.x - 4 + 4 * q;  // the quad's first cell
    const int j = 1 + kMY * (int)blockIdx.y + dj;
    const bool srow = trow && j <= g.ny;
    double acc[3] = {0.0, 0.0, 0.0};
    // bits 0-3: the quad's cells that lie in the tile; vec: stored as one vector; bits 4-7:
    // else the cells stored one by one (tile edges, the level's last quad)
    const bool vec = q >= 2 && q <= 8 && i4 + 3 <= g.nx;
    int keep = q == 1 ? 14 : q == 9 ? 1 : q >= 2 ? 15 : 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (!vec && (keep & (1 << e)) && i4 + e <= g.nx) keep |= 16 << e;
    // way up, phase 3: the pair's final odd values and the even ones stored (and summed)
    auto store_up = [&](auto po, int k, F2 fo, F2 fe, F2 bo, F2 be) {
        float v[4], b[4];
        constexpr int PO = decltype(po)::value;
        v[PO] = fo.x; v[PO + 2] = fo.y; v[1 - PO] = fe.x; v[3 - PO] = fe.y;
        b[PO] = bo.x; b[PO + 2] = bo.y; b[1 - PO] = be.x; b[3 - PO] = be.y;
        float* dst = out + (size_t)(j * g.sx + k * g.sxy) + i4;
        if (vec) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (keep & (16 << e)) dst[e] = v[e];
        if constexpr (ZDOT) {
            // tile cells; z and b are 0 on every cell that is not interior fluid (cells past
            // the level included)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (!(keep & (1 << e))) continue;
                const double zv = (double)v[e], rv = (double)b[e];
                acc[0] += zv;
                acc[1] += rv * zv;
                acc[2] += rv;
            }
        }
    };
    // way down: the coarse cell (ci, cj) of the tile, from the residual buffer rb of its
    // plane; zt: the coupled z faces' part
    const int ci = tid & 15, cj = tid >> 4;
    const int ic = kMX / 2 * (int)blockIdx.x + 1 + ci, jc = kMY / 2 * (int)blockIdx.y + 1 + cj;
    const bool writer = !UP && tid < 128 && ic <= L.cg.nx && jc <= L.cg.ny;
    const int orb = (2 * cj + 1) * 4 * kQuads + 2 * ci + 5;  // its cell (0, 0)
    auto star_write = [&](const float* rb, uint32_t cc, int kc, T zt) {
        constexpr int RW = 4 * kQuads;
        const T* r0 = rb + orb;
        const T a0 = r0[0], a1 = r0[1], b0 = r0[RW], b1 = r0[RW + 1];
        T s = (cc & 2u) ? (r0[-1] + r0[RW - 1]) - (a0 + b0) : T(0);
        s += (cc & 1u) ? (r0[2] + r0[RW + 2]) - (a1 + b1) : T(0);
        s += (cc & 8u) ? (r0[-RW] + r0[1 - RW]) - (a0 + a1) : T(0);
        s += (cc & 4u) ? (r0[2 * RW] + r0[2 * RW + 1]) - (b0 + b1) : T(0);
        out[cidx(L.cg, ic, jc, kc)] = ((a0 + a1) + (b0 + b1)) + T(kStarW) * (s + zt);
    };
    float* rbuf = reinterpret_cast<float*>(sm + C::OFF_R);

    // the previous kernel's results from here on (see k_level_fused)
    pdl_wait();
    bool ok = true;
    const int stop = done ? ld_now(done) : 0;
    if (tid == 0) RG.start2(M);
    pdl_launch();
    if (stop) {
        if (tid == 0 && !RG.drain()) atomicExch(err, 1);
        return;
    }
    if (tid == 0) ok = RG.wait(RG.p0);
    if (!step_barrier(ok, err)) return;

    using B0 = std::integral_constant<int, 0>;
    using B1 = std::integral_constant<int, 1>;
    if constexpr (DIM == 2) {
        const unsigned char* st = sm + C::OFF_RING;
        float *O = pk + 1, *E = pk + C::PLANE + 1;
        auto run = [&](auto po) {
            constexpr int PO = decltype(po)::value;
            using PE = std::integral_constant<int, 1 - PO>;
            const F2 zero{0.f, 0.f};
            Quad Q{};
            F2 vo = zero, ve = zero;
            if (live) vo = odd_phase(st, O, po, std::false_type(), Q);
            __syncthreads();
            if (live) {
                ve = relax(Q.e, nbsum(O, PE(), vo, zero), Q.re);
                *reinterpret_cast<float2*>(E + op) = make_float2(ve.x, ve.y);
            }
            __syncthreads();
            if constexpr (UP) {
                if (srow && q >= 1) store_up(po, 0, relax(Q.o, nbsum(E, po, ve, zero), Q.ro), ve, Q.o, Q.e);
            } else if (frow) {
                F2 f = nbsum(E, po, ve, zero);
                f.x = Q.ro.x != 0.f ? f.x : 0.f;
                f.y = Q.ro.y != 0.f ? f.y : 0.f;
                // the even cells were just relaxed: 0
                *reinterpret_cast<float4*>(rbuf + (dj + 1) * 4 * kQuads + 4 * q) =
                    PO == 0 ? make_float4(f.x, 0.f, f.y, 0.f) : make_float4(0.f, f.x, 0.f, f.y);
            }
        };
        // odd cells at (1 + j) & 1, j = 1 + 16 by + r - R
        if ((R + grp) & 1) run(B1());
        else run(B0());
        if constexpr (!UP) {
            const uint32_t cc = writer ? L.ccode[cidx(L.cg, ic, jc, 0)] : 0u;
            __syncthreads();
            if (writer) star_write(rbuf, cc, 0, T(0));
        }
    } else {
        // Registers by step parity (H: this step's): everything a step needs from earlier
        // ones was made one step ago (the other parity's slot) or two (its own, about to be
        // overwritten), so nothing moves.  o / ro: b and 1/d of plane s+1's odd cells, used
        // again two steps on; e / re: of its even cells, used in the next (e: and in the one
        // after, for the z sums); vo, ve: odd
        // values of plane s+1, even values of plane s.
        F2 o[2] = {}, ro[2] = {}, e[2] = {}, re[2] = {}, vo[2] = {}, ve[2] = {};
        T zh = T(0);  // way down: the coarse plane below's upper sum
        uint32_t cc = 0u;
        const unsigned char* st = sm + C::OFF_RING;  // stage of plane s+1
        // PN: the odd cells' position on plane s+1 (and s-1); KO: planes s+1 and s-1 are odd
        auto work = [&](int s, auto hc, auto pn, auto kodd) {
            constexpr int H = decltype(hc)::value, PN = decltype(pn)::value;
            using PO1 = std::integral_constant<int, PN>;
            float* On = pk + H * C::PLANE + 1;
            const float* Oc = pk + (1 - H) * C::PLANE + 1;
            float* En = pk + (2 + H) * C::PLANE + 1;
            const float* Ec = pk + (3 - H) * C::PLANE + 1;
            const F2 bo = o[H], be = e[H], rbo = ro[H], o2 = vo[H], e2 = ve[H];  // planes s-1; e2: s-2
            Quad Q;
            vo[H] = odd_phase(st, On, pn, kodd, Q);
            // even cells of plane s sit where plane s+1's odd ones do
            const F2 en = relax(e[1 - H], nbsum(Oc, PO1(), vo[1 - H], add2(vo[H], o2)), re[1 - H]);
            *reinterpret_cast<float2*>(En + op) = make_float2(en.x, en.y);
            const int p = s - 1;
            if constexpr (UP) {
                if (p >= kb && srow && q >= 1) {
                    const F2 f = relax(bo, nbsum(Ec, PO1(), ve[1 - H], add2(en, e2)), rbo);
                    store_up(PO1(), p, f, ve[1 - H], bo, be);
                }
            } else if (p >= kb - 1 && frow) {
                const F2 f = nbsum(Ec, PO1(), ve[1 - H], add2(en, e2));
                float* rb = rbuf + (((p + 1) >> 1) & 1) * (align128(C::RB * sizeof(float)) / sizeof(float)) +
                            (dj + 1) * 4 * kQuads + 4 * q + PN;
                rb[0] = rbo.x != 0.f ? f.x : 0.f;
                rb[2] = rbo.y != 0.f ? f.y : 0.f;
            }
            o[H] = Q.o;
            ro[H] = Q.ro;
            e[H] = Q.e;
            re[H] = Q.re;
            ve[H] = en;
        };
        // way down, beside an even plane p's step: coarse plane kc = p / 2 - 1, whose fine
        // planes and the one above it are in the buffers.  Its children's residuals: (0,0)
        // and (1,1) come from its lower plane, the others from its upper one (a cell is odd
        // on one of them).
        auto coarse = [&](int p) {
            const int kc = p / 2 - 1;
            constexpr size_t NB = align128(C::RB * sizeof(float)) / sizeof(float);
            const float* rb = rbuf + (kc & 1) * NB;
            const float* rn = rbuf + ((kc + 1) & 1) * NB;
            if (writer) {
                const T lo = rb[orb] + rb[orb + 4 * kQuads + 1], hi = rb[orb + 1] + rb[orb + 4 * kQuads];
                const T nx = rn[orb] + rn[orb + 4 * kQuads + 1];
                if (kc >= (kb + 1) / 2)
                    star_write(rb, cc, kc, ((cc & 32u) ? zh - lo : T(0)) + ((cc & 16u) ? nx - hi : T(0)));
                zh = hi;
                // the next plane's code, an iteration of two steps ahead
                if (2 * (kc + 1) <= ke) cc = L.ccode[cidx(L.cg, ic, jc, kc + 1)];
            }
        };
        using KE = std::integral_constant<bool, X != 0>;  // is s0 odd?
        // step s = s0 + (0 or 1) + 2 u: plane s+1 is odd when s is even
        // position of plane k's odd cells: (R + grp + k) & 1
        auto step = [&](int s, auto first) -> bool {
            constexpr bool SODD = decltype(first)::value ? KE::value : !KE::value;
            using KO = std::integral_constant<bool, !SODD>;  // plane s+1 is odd
            using H = std::integral_constant<int, decltype(first)::value ? 0 : 1>;
            if (live) {
                if ((R + grp + (SODD ? 0 : 1)) & 1) work(s, H(), B1(), KO());
                else work(s, H(), B0(), KO());
            }
            if constexpr (!UP && SODD) {  // plane s-1 is even
                if (s - 1 >= kb + 1) coarse(s - 1);
            }
            bool okk = true;
            if (tid == 0 && s + 2 <= RG.plast) okk = RG.wait(s + 2);
            if (!step_barrier(okk, err)) return false;
            if (tid == kRefill) RG.refill(M, s + 1);
            st += P::STAGE;
            if (st == sm + C::OFF_RING + S * P::STAGE) st = sm + C::OFF_RING;
            return true;
        };
#pragma unroll 1
        for (int s = s0; s <= sl; s += 2) {
            if (!step(s, std::true_type())) return;
            if (s + 1 <= sl && !step(s + 1, std::false_type())) return;
        }
        if constexpr (!UP) coarse(ke + 1);  // the last coarse plane (ke is odd)
    }
    if constexpr (UP && ZDOT) {
        double tot[3];
        ZdotIn in;
        if (reduce_last<3>(acc, partials, &cg->counter[2], tot, [&] { in.load(cg); }))
            finish_zdot(cg, in, tot);
    }
}

}  // namespace
}  // namespace uaamg
