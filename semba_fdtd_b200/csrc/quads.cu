// The quad half-step kernels (quads.cuh) and their tables.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "quads.cuh"
#include "sgpu_internal.h"

using namespace sgpu;
using namespace sgpu::dev;

namespace {

constexpr int kQuadThreads = 64;  // 8 blocks an SM at 128 registers: 10 blocks spill and take 1.3 times as long
// Planes a thread marches: few, for many blocks in flight (4 against 16 planes
// at 220^3: 191 / 207 us a step).
constexpr int kQuadChunk = 4;
// Up to here (padded cells) the quads are the faster half step.  Beyond, DRAM
// streaming decides, the TMA ring's deeper prefetch catches up, and its blocks
// leave room for another stream's.  One step of cubes with CPML 10 alone on the
// GPU, quads against ring: 60^3 10.2 / 24.4 us, 150^3 67.8 / 91.7, 220^3
// 191 / 209, 276^3 359 / 376, 400^3 988 / 956; 280^3 cubes of three streams
// taking turns: 395 / 353..387.
constexpr long long kQuadCells = 16ll << 20;

template <int SIDE>
__global__ void __launch_bounds__(kQuadThreads, 8)
    k_quad(const __grid_constant__ QuadView g, const __grid_constant__ QuadSide s, int chunk) {
    // everything before grid_wait is constant over the run: it overlaps the
    // kernel before
    __shared__ float2 tab[256];
    __shared__ QuadLine zl[kQuadChunk];
    for (int m = threadIdx.x; m < s.nmed1; m += kQuadThreads) tab[m] = s.tab[m];
    int p = blockIdx.x * kQuadThreads + threadIdx.x;
    const bool inner = p < s.inner;
    if (!inner) p -= s.inner;
    const int w = inner ? s.nq - s.xlo - s.xhi : s.xlo + s.xhi, r = p / w;
    const bool valid = r < s.ny;
    int q = p - r * w;
    q = inner ? q + s.xlo : q < s.xlo ? q : q + (s.nq - w);
    const int j = s.y0 + (valid ? r : s.ny - 1), i = 4 * q;
    const int kb = s.z0 + blockIdx.y * chunk, ke = min(kb + chunk, s.z0 + s.nz) - 1;
    for (int m = threadIdx.x; m <= ke - kb; m += kQuadThreads) zl[m] = s.z[kb + m];
    const QuadX* X = s.x + (i >> 2);
    const QuadLine Y = ldl(s.y + j);
    float idx[4];
    ld4(idx, X->id);
    const unsigned meet = valid ? X->meet & Y.hold : 0u, whole = X->whole;
    __syncthreads();
    grid_wait();
    if (__any_sync(0xffffffffu, meet != 0)) quad_march<SIDE, true>(g, s, tab, zl, X, Y, idx, meet, whole, i, j, kb, ke, valid);
    else quad_march<SIDE, false>(g, s, tab, zl, X, Y, idx, meet, whole, i, j, kb, ke, valid);
}

__global__ void k_quad_tables(KGrid g, KCpml cp, int nxa, int nya, int nza, int side, QuadX* x, QuadLine* y, QuadLine* z,
                              float2* tab) {
    const int nq = g.pitch / 4, q = blockIdx.x * blockDim.x + threadIdx.x;
    for (int m = q; m < g.nmed1; m += gridDim.x * blockDim.x)
        tab[m] = side ? make_float2(g.gm1[m], g.gm2[m]) : make_float2(g.g1[m], g.g2[m]);
    if (q >= nq + nya + nza) return;
    const int ax = q < nq ? 0 : q < nq + nya ? 1 : 2, at = ax == 0 ? 4 * q : ax == 1 ? q - nq : q - nq - nya;
    unsigned meet = 0, whole = 0;
    if (cp.on)
        for (int n = 0; n < 12; ++n) {
            const Slab& s = cp.s[3 * side + (n >> 2)][(n >> 1) & 1][n & 1];
            if (!s.psi) continue;
            const int lo = ax == 0 ? s.xlo : ax == 1 ? s.ylo : s.zlo, hi = ax == 0 ? s.xhi : ax == 1 ? s.yhi : s.zhi;
            if ((ax == 0 ? at + 3 : at) >= lo && at <= hi) meet |= 1u << n;
            if (at >= lo && at + 3 <= hi) whole |= 1u << n;
        }
    if (ax == 0) {
        QuadX r{};
        for (int e = 0; e < 4; ++e) {
            const bool in = cp.on && at + e < nxa;  // the CPML vectors end at the box, the x metrics at the pitch
            r.id[e] = (side ? g.idxe : g.idxh)[at + e];
            r.pb[e] = in ? (side ? cp.pbm[0] : cp.pbe[0])[at + e] : 1.0f;
            r.pc[e] = in ? (side ? cp.pcm[0] : cp.pce[0])[at + e] : 0.0f;
        }
        r.meet = meet;
        r.whole = whole;
        x[q] = r;
    } else {
        QuadLine r;
        r.id = (ax == 1 ? (side ? g.idye : g.idyh) : (side ? g.idze : g.idzh))[at];
        r.pb = cp.on ? (side ? cp.pbm[ax] : cp.pbe[ax])[at] : 1.0f;
        r.pc = cp.on ? (side ? cp.pcm[ax] : cp.pce[ax])[at] : 0.0f;
        r.hold = meet;
        (ax == 1 ? y : z)[at] = r;
    }
}

sgpu_status cuda_error(sgpu_ctx* c, const char* what, cudaError_t e) {
    return set_error(c, SGPU_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// One side's tables: x quads, rows, planes, the pairs of up to 256 media.
size_t table_bytes(const sgpu_ctx* c) {
    return c->pitch / 4 * sizeof(QuadX) + (size_t)(c->nya + c->nza) * sizeof(QuadLine) + 256 * sizeof(float2);
}

}  // namespace

namespace sgpu {

bool quads_usable(const sgpu_ctx* c) { return tma_usable(c) && c->vol <= kQuadCells && !c->wait_drill; }

QuadView quad_view(const sgpu_ctx* c) {
    QuadView v{};
    const KGrid g = kgrid(c);
    for (int f = 0; f < 6; ++f) {
        v.F[f] = c->F[f];
        v.M8[f] = c->M8[f];
        for (int q = 0; q < 6; ++q) v.sw[f][q] = g.sw[f][q];
    }
    v.pitch = c->pitch;
    v.plane = (int)c->plane;
    return v;
}

// The tables are built on first use and again after sgpu_init_cpml; before
// steps are captured, so that a graph holds no allocation.
sgpu_status quad_prepare(sgpu_ctx* c) {
    if (c->quad_ok) return SGPU_OK;
    const size_t nx = c->pitch / 4, one = table_bytes(c);
    if (!c->quad_mem) {
        c->quad_mem = ctx_malloc(c, 2 * one);
        if (!c->quad_mem) return set_error(c, SGPU_ERR_OOM, "quad tables");
    }
    for (int h = 0; h < 2; ++h) {
        QuadX* x = (QuadX*)((char*)c->quad_mem + h * one);
        QuadLine* y = (QuadLine*)(x + nx);
        const int n = (int)nx + c->nya + c->nza;
        k_quad_tables<<<(n + 127) / 128, 128, 0, c->stream>>>(kgrid(c), c->cpml, c->nxa, c->nya, c->nza, h, x, y, y + c->nya,
                                                         (float2*)(y + c->nya + c->nza));
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_error(c, "k_quad_tables", e);
    }
    c->quad_ok = true;
    return SGPU_OK;
}

QuadSide quad_side(const sgpu_ctx* c, int side) {
    const KGrid g = kgrid(c);
    const size_t nx = c->pitch / 4, one = table_bytes(c);
    QuadSide s{};
    s.x = (const QuadX*)((const char*)c->quad_mem + side * one);
    s.y = (const QuadLine*)(s.x + nx);
    s.z = s.y + c->nya;
    s.tab = (const float2*)(s.z + c->nza);
    s.nmed1 = c->num_media + 1;
    int x1 = -1, y0 = 1 << 30, y1 = -1, z0 = 1 << 30, z1 = -1;
    for (int f = 3 * side; f < 3 * side + 3; ++f) {
        x1 = std::max(x1, g.sw[f][1]);
        y0 = std::min(y0, g.sw[f][2]); y1 = std::max(y1, g.sw[f][3]);
        z0 = std::min(z0, g.sw[f][4]); z1 = std::max(z1, g.sw[f][5]);
    }
    s.y0 = y0; s.ny = y1 - y0 + 1;
    s.z0 = z0; s.nz = z1 - z0 + 1;
    s.nq = x1 / 4 + 1;
    for (int n = 0; n < 12; ++n) {
        const Slab& q = c->cpml.s[3 * side + (n >> 2)][(n >> 1) & 1][n & 1];
        if (!c->cpml.on || !q.psi) continue;
        const int pn = q.px * (q.yhi - q.ylo + 1);
        if ((kCpmlX >> n) & 1u) {  // a correction along x: the quads up to its low side, or from its high side on
            if (n & 1) s.xhi = std::max(s.xhi, s.nq - q.xlo / 4);
            else s.xlo = std::max(s.xlo, q.xhi / 4 + 1);
        }
        s.slab[n] = SlabRef{q.psi - q.xb - (long long)q.px * q.ylo - (long long)pn * q.zlo, q.px, pn, q.xlo, q.xhi};
    }
    // a grid whose two x sides meet: one group
    if (s.xlo < 0 || s.xhi < 0 || s.xlo + s.xhi >= s.nq) s.xlo = s.xhi = 0;
    s.inner = (int)(((long long)s.ny * (s.nq - s.xlo - s.xhi) + 31) / 32 * 32);
    s.threads = s.inner + s.ny * (s.xlo + s.xhi);
    return s;
}

sgpu_status launch_quad(sgpu_ctx* c, int side) {
    const sgpu_status st = quad_prepare(c);
    if (st) return st;
    const QuadSide s = quad_side(c, side);
    const int bx = (s.threads + kQuadThreads - 1) / kQuadThreads;
    int chunk = kQuadChunk;
    while (chunk > 2 && (long long)bx * ((s.nz + chunk - 1) / chunk) < 148 * 16) chunk /= 2;
    const dim3 grid(bx, (s.nz + chunk - 1) / chunk);
    const QuadView v = quad_view(c);
    const cudaError_t e = side ? launch_after(c->stream, grid, kQuadThreads, k_quad<1>, v, s, chunk)
                               : launch_after(c->stream, grid, kQuadThreads, k_quad<0>, v, s, chunk);
    return e == cudaSuccess ? SGPU_OK : cuda_error(c, "k_quad", e);
}

}  // namespace sgpu
