// The curl + CPML half steps from plain loads, four x cells (a quad) a thread.
//
// A thread marches a few z planes of one quad: every array is one aligned
// 16-byte access a plane, the field below (E) or above (H) stays in registers,
// and the y and x neighbours are L1 or L2 hits.  Consecutive quads in row order
// fill the warps, so a row's end wastes no lane.  The CPML slabs a quad meets
// are known from three small tables (per quad of x cells, row and plane), and
// a psi row is padded to whole quads, so a correction moves 16 bytes as well.
#pragma once
#include "stencil.cuh"

namespace sgpu {

// Inverse steps, P_b / P_c and the slabs (of a side's 12) that meet the quad
// or hold it whole; a row's or a plane's inverse step, P_b, P_c and the slabs
// that hold it.
struct alignas(16) QuadX {
    float id[4], pb[4], pc[4];
    unsigned meet, whole, pad[2];
};
struct alignas(16) QuadLine {
    float id, pb, pc;
    unsigned hold;
};
// A psi slab by absolute local indices: the psi of (i, j, k) is base[i + px*j + pn*k].
struct SlabRef {
    float* base;
    int px, pn;
    int xlo, xhi;
};
// One side's half step.
struct QuadSide {
    const QuadX* x;
    const QuadLine *y, *z;
    const float2* tab;     // (G1, G2) or (GM1, GM2) of every medium
    int nmed1;
    int y0, ny, z0, nz, nq;  // rows, planes and quads a row of the union of the sweeps
    // the first xlo and last xhi quads of a row meet the slabs of x corrections;
    // they are numbered after all others (from `inner`, a multiple of 32), so
    // that a warp has either none or only such quads
    int xlo, xhi, inner, threads;
    SlabRef slab[12];
};
struct QuadView {
    float* F[6];
    const uint8_t* M8[6];
    int pitch, plane;
    int sw[6][6];
};

// Views of a context, and its tables (built on first use).
QuadView quad_view(const sgpu_ctx* c);
QuadSide quad_side(const sgpu_ctx* c, int side);
sgpu_status quad_prepare(sgpu_ctx* c);

namespace dev {

// The quad of thread p of a side: its first cell and row; false past the last
// (which then names a valid quad all the same).
__device__ __forceinline__ bool quad_at(const QuadSide& s, int p, int& i, int& j) {
    const bool inner = p < s.inner;
    if (!inner) p -= s.inner;
    const int w = inner ? s.nq - s.xlo - s.xhi : s.xlo + s.xhi, r = w ? p / w : s.ny;
    const bool valid = r < s.ny;
    int q = valid ? p - r * w : 0;
    q = inner ? q + s.xlo : q < s.xlo ? q : q + (s.nq - w);
    j = s.y0 + (valid ? r : s.ny - 1);
    i = 4 * q;
    return valid;
}

__device__ __forceinline__ void ld4(float (&v)[4], const float* p) {
    const float4 q = *(const float4*)p;
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) { *(float4*)p = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ QuadLine ldl(const QuadLine* p) {
    const float4 q = *(const float4*)p;
    return QuadLine{q.x, q.y, q.z, __float_as_uint(q.w)};
}
// The cells i .. i+3 inside [lo, hi], as bits.
__device__ __forceinline__ unsigned in_range4(int i, int lo, int hi) {
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) m |= (i + e >= lo && i + e <= hi) ? 1u << e : 0u;
    return m;
}
// Store a quad, the cells outside `ok` with their old values (no one else
// writes them in this phase).
__device__ __forceinline__ void put4(float* p, unsigned ok, float (&v)[4], const float (&old)[4]) {
    if (ok == 0) return;
    if (ok != 15u) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (!((ok >> e) & 1u)) v[e] = old[e];
    }
    st4(p, v);
}
// The coefficient pairs of a quad's four media: most quads have one medium.
__device__ __forceinline__ void quad_tab(float2 (&t)[4], const float2* tab, unsigned m) {
    t[0] = tab[m & 255u];
    t[1] = t[2] = t[3] = t[0];
    if (m != (m & 255u) * 0x01010101u) {
        t[1] = tab[(m >> 8) & 255u];
        t[2] = tab[(m >> 16) & 255u];
        t[3] = tab[m >> 24];
    }
}
// The old psi of one correction of a quad: slab pair N, N + 1, whose live bits
// (at most one: quads_apart) are in `live`.  Loaded with the plane's fields, before any store of the
// plane: a load behind a store would wait for memory once per correction.
struct QuadPsi {
    float v[4];
    float* p;
    unsigned cells;  // the quad's cells inside the slab
};
template <int N>
__device__ __forceinline__ void psi_load(QuadPsi& s, const SlabRef* slab, unsigned live, unsigned whole, int i, int j, int k) {
    const unsigned b = (live >> N) & 3u;
    s.cells = 0;
    if (b) {
        const bool lo = b & 1u;
        const SlabRef &u = slab[N], &w = slab[N + 1];
        s.p = (lo ? u.base : w.base) + (i + (lo ? u.px : w.px) * j + (lo ? u.pn : w.pn) * k);
        ld4(s.v, s.p);
        s.cells = (whole >> (lo ? N : N + 1)) & 1u ? 15u : in_range4(i, lo ? u.xlo : w.xlo, lo ? u.xhi : w.xhi);
    }
}
// psi = P_b psi + diff P_c ; F = F +- g psi, cell by cell as cpml_pair; pb / pc
// per cell (x) or one value.
template <bool ADD, int NP>
__device__ __forceinline__ void psi_apply(QuadPsi& s, const float (&pb)[NP], const float (&pc)[NP], const float (&diff)[4],
                                          const float2 (&t)[4], float (&v)[4]) {
    if (s.cells) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float q = pb[NP == 4 ? e : 0] * s.v[e] + diff[e] * pc[NP == 4 ? e : 0];
            if ((s.cells >> e) & 1u) {
                s.v[e] = q;
                v[e] = ADD ? v[e] + t[e].y * q : v[e] - t[e].y * q;
            }
        }
        st4(s.p, s.v);
    }
}

// Advance_E (SIDE 0, timestepping.F90:2165-2285) + AdvanceelectricCPML or
// Advance_H (SIDE 1, :2294-2409) + AdvanceMagneticCPML of the quad at (i, j)
// over planes kb..ke, in the order of efield_column / hfield_column.  Both
// sides march so that the z neighbour is the plane before: up on the E side,
// down on the H side.  MODE (kBulk, kCpml, kCx ..): only the curl, only the
// corrections, only some components, for the routines called one by one.
template <int SIDE, bool CP, int MODE = kBulk | kCpml | kAll>
__device__ __forceinline__ void quad_march(const QuadView& g, const QuadSide& s, const float2* tab, const QuadLine* zl, const QuadX* X, const QuadLine& Y,
                                           const float (&idx)[4], unsigned meet, unsigned whole, int i, int j, int kb, int ke,
                                           bool valid) {
    constexpr int O = 3 * SIDE, S = 3 - O;  // own and other field
    const int pitch = g.pitch, plane = g.plane;
    const SlabRef* slab = s.slab;
    int k = SIDE ? ke : kb;
    int c = i + pitch * j + plane * k;
    const int dz = SIDE ? plane : -plane, dy = SIDE ? pitch : -pitch;
    float xk[4], yk[4];  // the other field's x and y components at the plane before
    if (MODE & kCy) ld4(xk, g.F[S] + (c + dz));
    if (MODE & kCx) ld4(yk, g.F[S + 1] + (c + dz));
    unsigned ok0 = 0, ok1 = 0, ok2 = 0;
    if (valid) {
        ok0 = j >= g.sw[O][2] && j <= g.sw[O][3] ? in_range4(i, g.sw[O][0], g.sw[O][1]) : 0u;
        ok1 = j >= g.sw[O + 1][2] && j <= g.sw[O + 1][3] ? in_range4(i, g.sw[O + 1][0], g.sw[O + 1][1]) : 0u;
        ok2 = j >= g.sw[O + 2][2] && j <= g.sw[O + 2][3] ? in_range4(i, g.sw[O + 2][0], g.sw[O + 2][1]) : 0u;
    }
    const int planes = ke - kb + 1;
#pragma unroll 1
    for (int n = 0; n < planes; ++n, k += SIDE ? -1 : 1, c -= dz) {
        float x[4], y[4], z[4], xj[4], zj[4], f0[4], f1[4], f2[4];
        const QuadLine Z = ldl(zl + (k - kb));
        const unsigned live = CP ? meet & Z.hold : 0u;
        if (!(MODE & kBulk) && !live) continue;  // the carried planes are loaded again below
        if (MODE & (kCy | kCz)) ld4(x, g.F[S] + c);
        if (MODE & (kCx | kCz)) ld4(y, g.F[S + 1] + c);
        if (MODE & (kCx | kCy)) ld4(z, g.F[S + 2] + c);
        if (MODE & kCz) ld4(xj, g.F[S] + (c + dy));
        if (MODE & kCx) ld4(zj, g.F[S + 2] + (c + dy));
        if (MODE & kCx) ld4(f0, g.F[O] + c);
        if (MODE & kCy) ld4(f1, g.F[O + 1] + c);
        if (MODE & kCz) ld4(f2, g.F[O + 2] + c);
        if (!(MODE & kBulk)) {
            ld4(xk, g.F[S] + (c + dz));
            ld4(yk, g.F[S + 1] + (c + dz));
        }
        float yi = 0.0f, zi = 0.0f;
        if (MODE & kCz) yi = g.F[S + 1][c + (SIDE ? 4 : -1)];
        if (MODE & kCy) zi = g.F[S + 2][c + (SIDE ? 4 : -1)];
        unsigned m0 = 0, m1 = 0, m2 = 0;
        if (MODE & kCx) m0 = *(const unsigned*)(g.M8[O] + c);
        if (MODE & kCy) m1 = *(const unsigned*)(g.M8[O + 1] + c);
        if (MODE & kCz) m2 = *(const unsigned*)(g.M8[O + 2] + c);
        const unsigned on0 = k >= g.sw[O][4] && k <= g.sw[O][5] ? ok0 : 0u;
        const unsigned on1 = k >= g.sw[O + 1][4] && k <= g.sw[O + 1][5] ? ok1 : 0u;
        const unsigned on2 = k >= g.sw[O + 2][4] && k <= g.sw[O + 2][5] ? ok2 : 0u;
        QuadPsi p0, p1, p2, p3, p4, p5;
        if (CP) {
            psi_load<0>(p0, slab, on0 ? live : 0u, whole, i, j, k);
            psi_load<2>(p1, slab, on0 ? live : 0u, whole, i, j, k);
            psi_load<4>(p2, slab, on1 ? live : 0u, whole, i, j, k);
            psi_load<6>(p3, slab, on1 ? live : 0u, whole, i, j, k);
            psi_load<8>(p4, slab, on2 ? live : 0u, whole, i, j, k);
            psi_load<10>(p5, slab, on2 ? live : 0u, whole, i, j, k);
        }
        // differences along an axis: backward (E) or forward (H)
        auto dif = [](float at, float next) { return SIDE ? next - at : at - next; };
        auto nx = [&](const float (&v)[4], float edge_v, int e) {
            return SIDE ? (e < 3 ? v[e < 3 ? e + 1 : 3] : edge_v) : (e ? v[e ? e - 1 : 0] : edge_v);
        };
        float d1[4], d2[4], v[4];
        float2 t[4];
        const float yb[1] = {Y.pb}, yc[1] = {Y.pc}, zb[1] = {Z.pb}, zc[1] = {Z.pc};
        if (MODE & kCx) {  // x: y derivative of the z component, z derivative of the y component
            quad_tab(t, tab, m0);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                d1[e] = dif(z[e], zj[e]);
                d2[e] = dif(y[e], yk[e]);
                v[e] = !(MODE & kBulk) ? f0[e] : t[e].x * f0[e] + t[e].y * (SIDE ? d2[e] * Z.id - d1[e] * Y.id : d1[e] * Y.id - d2[e] * Z.id);
            }
            if (CP && live) {
                psi_apply<SIDE == 0>(p0, yb, yc, d1, t, v);
                psi_apply<SIDE == 1>(p1, zb, zc, d2, t, v);
            }
            put4(g.F[O] + c, on0, v, f0);
        }
        if (MODE & kCy) {  // y: z derivative of the x component, x derivative of the z component
            quad_tab(t, tab, m1);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                d1[e] = dif(x[e], xk[e]);
                d2[e] = dif(z[e], nx(z, zi, e));
                v[e] = !(MODE & kBulk) ? f1[e] : t[e].x * f1[e] + t[e].y * (SIDE ? d2[e] * idx[e] - d1[e] * Z.id : d1[e] * Z.id - d2[e] * idx[e]);
            }
            if (CP && live) {
                psi_apply<SIDE == 0>(p2, zb, zc, d1, t, v);
                psi_apply<SIDE == 1>(p3, X->pb, X->pc, d2, t, v);
            }
            put4(g.F[O + 1] + c, on1, v, f1);
        }
        if (MODE & kCz) {  // z: x derivative of the y component, y derivative of the x component
            quad_tab(t, tab, m2);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                d1[e] = dif(y[e], nx(y, yi, e));
                d2[e] = dif(x[e], xj[e]);
                v[e] = !(MODE & kBulk) ? f2[e] : t[e].x * f2[e] + t[e].y * (SIDE ? d2[e] * Y.id - d1[e] * idx[e] : d1[e] * idx[e] - d2[e] * Y.id);
            }
            if (CP && live) {
                psi_apply<SIDE == 1>(p4, yb, yc, d2, t, v);
                psi_apply<SIDE == 0>(p5, X->pb, X->pc, d1, t, v);
            }
            put4(g.F[O + 2] + c, on2, v, f2);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            xk[e] = x[e];
            yk[e] = y[e];
        }
    }
}

}  // namespace dev
}  // namespace sgpu
