// The quad half-step kernels (quads.cuh) and their tables.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <type_traits>
#include <vector>

#include "observe.cuh"
#include "quads.cuh"
#include "sgpu_internal.h"

using namespace sgpu;
using namespace sgpu::dev;

namespace {

constexpr int kQuadThreads = 64;  // 8 blocks an SM at 128 registers: 10 blocks spill and take 1.3 times as long
// Planes a thread marches: few, for many blocks in flight (4 against 16 planes
// at 220^3: 191 / 207 us a step).
constexpr int kQuadChunk = 4;
// Up to here (padded cells) the quads, beyond the TMA ring.  The line lies between
// two uses: alone on the GPU the quads are the faster half step to 30 Mi and more
// (their blocks start sooner), with three solvers taking turns on streams of their
// own the ring is from 10 Mi on (its blocks leave room for another stream's).  A
// step of cubes with CPML 10, quads / ring, alone (spread 2 to 4 %) and of three
// (6 %): 8.8 Mi 155 / 170 and 147 / 148 us, 10.6 Mi 191 / 213 and 186 / 174, 15.4 Mi
// 270 / 290 and 263 / 248, 19.9 Mi 327 / 369 and 324 / 315, 29.9 Mi 492 / 511 and
// 493 / 458.
constexpr long long kQuadCells = 16ll << 20;

constexpr int kQuadVol = 4;  // volume probes the arguments hold

// A source row with its first contribution beside it.
struct QuadRow {
    int node, comp, count, first;
    SrcEntry e;
};
// The nodal source rows of a half step by (warp's quads, plane), and what a row needs.
struct QuadSrc {
    const int* ptr;  // null: none
    const QuadRow* row;
    KSrc s;
    const double* tiempo;
    int t_n0;
    double dt;
    StepRef sr;
};
// A row's node, its first contribution and where the others stand.
struct RowTerm {
    float* f;
    SrcTerm first;
    int p, end;
};
// Nodal source rows ride in the half step, a launch less, while no plane wave acts
// and they are at most one on 128 cells (denser was not measured).  One step alone
// on the GPU against k_sources, spread below 1 %: 86x76x82 cells, a line of 60 nodes
// 13.9 / 15.4 us; 170^3, a line of 128 100.8 / 103.5; 42x45x40, a plate of 64
// 11.1 / 21.3, where k_sources also looks through 64 waveforms for a plane wave's.
// The rows of an acting wave do not ride: where a z face of its box passes they are
// two on each of a warp's 128 cells, with five dependent loads each, and held the
// half step up, where k_sources has a thread a row (riding / not, 86x76x82 cells,
// one row on 70 cells 22.4 / 17.3 us; 104^3, on 81 33.1 / 30.4; 170^3, on 84
// 133 / 107, on 26 162 / 109).  Past, they change nothing and take no launch
// (86x76x82 cells 13.8 us against 17.2 with k_sources, 170^3 100 / 109).
constexpr int kRowsAtOnce = 4;
constexpr long long kCellsARow = 128;
constexpr int kNodalTerms = (1 << kSrcNodalSoft) | (1 << kSrcNodalHard);
// Observations of one side's fields after step sr, one thread a point probe, a
// volume probe's node or a surface sample.
struct QuadObs {
    KProbes probes;
    int first_n;
    int nvol;
    VolProbe vol[kQuadVol];
    int nfar;
    FarArgs far;
    int ox, oy, oz;
    StepRef sr;
};

__device__ __forceinline__ void observe(const KGrid& g, const QuadObs& o, int side, long long q) {
    const int n = step_of(o.sr);
    if (q < o.probes.n) {
        if ((o.probes.comp[q] >= 3) == (side == 1)) probe_one(g, o.probes, n, o.first_n, (int)q);
        return;
    }
    q -= o.probes.n;
    for (int v = 0; v < o.nvol; ++v) {
        const VolProbe& p = o.vol[v];
        if ((p.magnetic != 0) != (side == 1)) continue;
        const long long nodes = (long long)p.ni * p.nj * p.nk;
        if (q < nodes) {
            if (p.kind == 0) vol_probe_node<true>(g, p, n, o.ox, o.oy, o.oz, nodes, q);
            else vol_probe_node<false>(g, p, n, o.ox, o.oy, o.oz, nodes, q);
            return;
        }
        q -= nodes;
    }
    int m;
    if (o.nfar && q < o.far.samples && far_step(o.far, n, m)) far_sample(g, o.far, m, side ? 2 : 1, o.ox, o.oy, o.oz, (int)q);
}

// The observations of H after a call's last step, which no half step follows.
__global__ void __launch_bounds__(kQuadThreads) k_observe_h(const __grid_constant__ KGrid g, const __grid_constant__ QuadObs o) {
    grid_wait();
    observe(g, o, 1, blockIdx.x * (long long)kQuadThreads + threadIdx.x);
}

// One half step: blocks below `blocks` march quads (bx of them a chunk of
// planes) and apply the nodal source rows on their cells; with OBS the blocks from
// there on observe the other field, which this half step leaves alone.  A step
// is then two launches, where the sources and each kind of observation took one
// each (84^3 cells with probes and a plane wave that is past: 5 launches, 24.0 us a
// step alone, against 20.1).
template <int SIDE, bool OBS>
__global__ void __launch_bounds__(kQuadThreads, 8)
    k_quad(const __grid_constant__ QuadView g, const __grid_constant__ QuadSide s, const __grid_constant__ KGrid kg,
           const __grid_constant__ QuadSrc src, const __grid_constant__ std::conditional_t<OBS, QuadObs, char> obs, int chunk, int bx,
           int blocks) {
    if constexpr (OBS) {
        if ((int)blockIdx.x >= blocks) {
            grid_wait();
            observe(kg, obs, 1 - SIDE, (blockIdx.x - blocks) * (long long)kQuadThreads + threadIdx.x);
            return;
        }
    }
    // everything before grid_wait is constant over the run: it overlaps the
    // kernel before
    __shared__ float2 tab[256];
    __shared__ QuadLine zl[kQuadChunk];
    __shared__ RowTerm ahead[kQuadThreads];
    for (int m = threadIdx.x; m < s.nmed1; m += kQuadThreads) tab[m] = s.tab[m];
    const int by = blockIdx.x / bx;
    const int p = (blockIdx.x - by * bx) * kQuadThreads + threadIdx.x;
    const int k0 = by * chunk, k1 = min(k0 + chunk, s.nz), kb = s.z0 + k0, ke = s.z0 + k1 - 1;
    for (int m = threadIdx.x; m <= ke - kb; m += kQuadThreads) zl[m] = s.z[kb + m];
    // the warp's source rows: their first contributions are formed here
    int r0 = 0, r1 = 0;
    const int lane = threadIdx.x & 31;
    if (src.ptr && p - lane < s.threads) {
        const int* sp = src.ptr + (p >> 5) * s.nz;
        r0 = sp[k0];
        r1 = sp[k1];
    }
    float t = 0.0f;
    if (r0 < r1) {
        const double tn = src.tiempo[step_of(src.sr) - src.t_n0];
        t = SIDE ? (float)(tn + (double)0.5f * src.dt) : (float)tn;
    }
    auto term = [&](const SrcEntry& e) { return source_term(src.s, e, t, 0.0f, kNodalTerms, false); };
    auto row_of = [&](int r) {
        const QuadRow q = src.row[r];
        return RowTerm{kg.F[q.comp] + q.node, term(q.e), q.first + 1, q.first + q.count};
    };
    if (r0 + lane < r1) ahead[threadIdx.x] = row_of(r0 + lane);
    int i, j;
    const bool valid = quad_at(s, p, i, j);
    const QuadX* X = s.x + (i >> 2);
    const QuadLine Y = ldl(s.y + j);
    float idx[4];
    ld4(idx, X->id);
    const unsigned meet = valid ? X->meet & Y.hold : 0u, whole = X->whole;
    __syncthreads();
    grid_wait();
    if (__any_sync(0xffffffffu, meet != 0)) quad_march<SIDE, true>(g, s, tab, zl, X, Y, idx, meet, whole, i, j, kb, ke, valid);
    else quad_march<SIDE, false>(g, s, tab, zl, X, Y, idx, meet, whole, i, j, kb, ke, valid);
    if (r0 < r1) {
        __syncwarp();  // the warp's cells are stored
        if (r0 + lane < r1) {
            const RowTerm row = ahead[threadIdx.x];
            float v = source_add(*row.f, row.first);
            for (int e = row.p; e < row.end; ++e) v = source_add(v, term(src.s.e[e]));
            *row.f = v;
        }
        for (int r = r0 + 32 + lane; r < r1; r += 32 * kRowsAtOnce) {
            // on distinct nodes: the loads of several rows, then their stores
            RowTerm row[kRowsAtOnce];
            float v[kRowsAtOnce];
#pragma unroll
            for (int u = 0; u < kRowsAtOnce; ++u) {
                row[u].f = nullptr;
                if (r + 32 * u < r1) {
                    row[u] = row_of(r + 32 * u);
                    v[u] = *row[u].f;
                }
            }
#pragma unroll
            for (int u = 0; u < kRowsAtOnce; ++u)
                if (row[u].f) {
                    v[u] = source_add(v[u], row[u].first);
                    for (int e = row[u].p; e < row[u].end; ++e) v[u] = source_add(v[u], term(src.s.e[e]));
                    *row[u].f = v[u];
                }
        }
    }
}

// One routine of a half step alone (MODE as quad_march's): one call per routine
// of 120x110x130 swept cells, 142 us a step with the register-marching kernels,
// 68 with these.
template <int SIDE, int MODE>
__global__ void __launch_bounds__(kQuadThreads, 8)
    k_quad_part(const __grid_constant__ QuadView g, const __grid_constant__ QuadSide s, int chunk, int bx) {
    __shared__ float2 tab[256];
    __shared__ QuadLine zl[kQuadChunk];
    for (int m = threadIdx.x; m < s.nmed1; m += kQuadThreads) tab[m] = s.tab[m];
    const int by = blockIdx.x / bx;
    const int kb = s.z0 + by * chunk, ke = min(kb + chunk, s.z0 + s.nz) - 1;
    for (int m = threadIdx.x; m <= ke - kb; m += kQuadThreads) zl[m] = s.z[kb + m];
    int i, j;
    const bool valid = quad_at(s, (blockIdx.x - by * bx) * kQuadThreads + threadIdx.x, i, j);
    const QuadX* X = s.x + (i >> 2);
    const QuadLine Y = ldl(s.y + j);
    float idx[4];
    ld4(idx, X->id);
    const unsigned meet = (MODE & kCpml) && valid ? X->meet & Y.hold : 0u, whole = X->whole;
    __syncthreads();
    grid_wait();
    if ((MODE & kBulk) || __any_sync(0xffffffffu, meet != 0))
        quad_march<SIDE, (MODE & kCpml) != 0, MODE>(g, s, tab, zl, X, Y, idx, meet, whole, i, j, kb, ke, valid);
}

// Side blockIdx.y's tables, `one` bytes a side (table_bytes).
__global__ void k_quad_tables(KGrid g, KCpml cp, int nxa, int nya, int nza, char* mem, size_t one) {
    const int side = blockIdx.y, nq = g.pitch / 4, q = blockIdx.x * blockDim.x + threadIdx.x;
    QuadX* const x = (QuadX*)(mem + side * one);
    QuadLine *const y = (QuadLine*)(x + nq), *const z = y + nya;
    float2* const tab = (float2*)(z + nza);
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

// Launched plainly after the tables: it begins when they are complete and
// visible, so the quad kernel that follows it may read them before grid_wait.
__global__ void k_tables_done() {}

sgpu_status cuda_error(sgpu_ctx* c, const char* what, cudaError_t e) {
    return set_error(c, SGPU_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// One side's tables: x quads, rows, planes, the pairs of up to 256 media.
size_t table_bytes(const sgpu_ctx* c) {
    return c->pitch / 4 * sizeof(QuadX) + (size_t)(c->nya + c->nza) * sizeof(QuadLine) + 256 * sizeof(float2);
}

}  // namespace

namespace sgpu {

// A quad takes one slab of a pair (psi_load).  Grids where some quad meets both,
// those of two cells in x between two CPML sides, go to the ring or the register
// kernels, which choose the slab cell by cell.
bool quads_apart(const KCpml& cp) {
    for (int f = 0; f < 6 && cp.on; ++f)
        for (int w = 0; w < 2; ++w) {
            const Slab &a = cp.s[f][w][0], &b = cp.s[f][w][1];
            auto meet = [](int alo, int ahi, int blo, int bhi) { return alo <= bhi && blo <= ahi; };
            if (a.psi && b.psi && meet(a.xlo / 4, a.xhi / 4, b.xlo / 4, b.xhi / 4) && meet(a.ylo, a.yhi, b.ylo, b.yhi) &&
                meet(a.zlo, a.zhi, b.zlo, b.zhi))
                return false;
        }
    return true;
}

bool quads_usable(const sgpu_ctx* c) {
    return c->family == 1 && tma_usable(c) && c->vol <= kQuadCells && c->quad_apart && !c->wait_drill && c->quad_mem;
}

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

// Room for the tables, taken with the context's other buffers, so that a
// context set up after another finds the pool's free blocks whole.  In a batch,
// too, from the device's pool: the arena holds what an instance's footprint
// counts.  Where the pool has none left the ring serves the context.
void quad_alloc(sgpu_ctx* c) {
    if (c->vol <= kQuadCells) c->quad_mem = ctx_pool_malloc(c, 2 * table_bytes(c));
}

// The tables are built on first use and again after sgpu_init_cpml.
sgpu_status quad_prepare(sgpu_ctx* c) {
    if (c->quad_ok) return SGPU_OK;
    const int n = c->pitch / 4 + c->nya + c->nza;
    k_quad_tables<<<dim3((n + 127) / 128, 2), 128, 0, c->stream>>>(kgrid(c), c->cpml, c->nxa, c->nya, c->nza, (char*)c->quad_mem,
                                                                   table_bytes(c));
    k_tables_done<<<1, 1, 0, c->stream>>>();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(c, "k_quad_tables", e);
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

// The nodal source rows grouped by (warp's quads, plane) of their node, in the
// kernel's numbering of the quads.  A side whose rows were not kept, or of which
// one lies on no cell the side's kernel updates, gets no groups.
static sgpu_status quad_sources(sgpu_ctx* c) {
    if (c->quad_src_ok) return SGPU_OK;
    for (void* q : c->quad_src_allocs) ctx_free(c, q);
    c->quad_src_allocs.clear();
    for (int side = 0; side < 2; ++side) {
        c->quad_sptr[side] = nullptr;
        c->quad_srow[side] = nullptr;
        const SrcRows& h = c->src_rows[side];
        const size_t n = h.node.size();
        c->quad_src_all[side] = h.kept && n == 0;
        if (n == 0) continue;
        const QuadSide s = quad_side(c, side);
        const int we = s.xlo + s.xhi, wi = s.nq - we;
        const size_t keys = (size_t)((s.threads + 31) / 32) * s.nz;
        std::vector<int> ptr(keys + 1, 0), key(n);
        bool fits = true;
        for (size_t r = 0; r < n; ++r) {
            const int q = h.node[r] % c->pitch / 4, j = (int)(h.node[r] % c->plane) / c->pitch - s.y0,
                      k = (int)(h.node[r] / c->plane) - s.z0;
            if (h.comp[r] / 3 != side || q >= s.nq || j < 0 || j >= s.ny || k < 0 || k >= s.nz) {
                fits = false;  // no thread of the side updates this cell
                break;
            }
            const bool in = q >= s.xlo && q < s.nq - s.xhi;
            const int p = in ? j * wi + (q - s.xlo) : s.inner + j * we + (q < s.xlo ? q : q - wi);
            key[r] = p / 32 * s.nz + k;
            ++ptr[key[r] + 1];
        }
        if (!fits) continue;
        for (size_t q = 0; q < keys; ++q) ptr[q + 1] += ptr[q];
        std::vector<int> at(ptr.begin(), ptr.end() - 1);
        std::vector<QuadRow> row(n);
        for (size_t r = 0; r < n; ++r) row[at[key[r]]++] = QuadRow{h.node[r], h.comp[r], h.count[r], h.start[r], h.first[r]};
        int* dp = (int*)ctx_malloc(c, ptr.size() * sizeof(int));
        if (dp) c->quad_src_allocs.push_back(dp);
        void* dr = ctx_malloc(c, n * sizeof(QuadRow));
        if (dr) c->quad_src_allocs.push_back(dr);
        if (!dp || !dr) continue;  // no room for groups: the rows stay with k_sources
        cudaError_t e = cudaMemcpyAsync(dp, ptr.data(), ptr.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dr, row.data(), n * sizeof(QuadRow), cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) return cuda_error(c, "source rows by warp", e);
        c->quad_sptr[side] = dp;
        c->quad_srow[side] = dr;
        c->quad_src_all[side] = true;
    }
    c->quad_src_ok = true;
    return SGPU_OK;
}

bool rows_ride(const sgpu_ctx* c, int side, long long rows) {
    const QuadSide s = quad_side(c, side);
    return kCellsARow * rows <= 4ll * s.nq * s.ny * s.nz;
}

bool rows_grouped(const sgpu_ctx* c, int side) { return c->quad_src_ok && c->quad_src_all[side]; }

bool observers_ride(const sgpu_ctx* c) { return (int)c->vprobes.size() <= kQuadVol && c->farfields.size() <= 1; }

// The observers of one side's fields and their threads (0: none).
static QuadObs quad_obs(const sgpu_ctx* c, int side, StepRef sr, long long* threads) {
    QuadObs o{};
    o.probes = c->probes;
    o.first_n = c->probe_first_n;
    o.ox = c->ox; o.oy = c->oy; o.oz = c->oz;
    o.sr = sr;
    *threads = c->probes.n;
    for (const VolProbe& v : c->vprobes) {
        if ((v.magnetic != 0) != (side == 1)) continue;
        o.vol[o.nvol++] = v;
        *threads += (long long)v.ni * v.nj * v.nk;
    }
    for (const FarField& f : c->farfields)
        if (f.samples) {
            o.far = far_args(f);
            o.nfar = 1;
            *threads += f.samples;
        }
    return o;
}

sgpu_status launch_observe_h(sgpu_ctx* c, StepRef sr) {
    long long threads;
    const QuadObs o = quad_obs(c, 1, sr, &threads);
    if (threads == 0) return SGPU_OK;
    const unsigned blocks = (unsigned)((threads + kQuadThreads - 1) / kQuadThreads);
    const cudaError_t e = launch_after(c->stream, blocks, kQuadThreads, k_observe_h, kgrid(c), o);
    return e == cudaSuccess ? SGPU_OK : cuda_error(c, "k_observe_h", e);
}

// Planes a thread of `bx` blocks' columns marches: fewer on grids with less than
// 16 blocks an SM (148 of them).
static int quad_chunk(int bx, int nz) {
    int chunk = kQuadChunk;
    while (chunk > 2 && (long long)bx * ((nz + chunk - 1) / chunk) < 148 * 16) chunk /= 2;
    return chunk;
}

sgpu_status launch_quad(sgpu_ctx* c, int side, StepRef sr, bool sources, const StepRef* obs, bool* applied) {
    sgpu_status st = quad_prepare(c);
    if (st) return st;
    const QuadSide s = quad_side(c, side);
    const int bx = (s.threads + kQuadThreads - 1) / kQuadThreads;
    const int chunk = quad_chunk(bx, s.nz);
    const int blocks = bx * ((s.nz + chunk - 1) / chunk);
    const QuadView v = quad_view(c);
    const KGrid g = kgrid(c);
    QuadSrc src{};
    // grouped before they are needed: a later call may be under capture
    if (c->src[side].nrows && (st = quad_sources(c))) return st;
    if (sources && c->src[side].nrows && rows_grouped(c, side)) {
        if (c->quad_sptr[side])
            src = QuadSrc{c->quad_sptr[side], (const QuadRow*)c->quad_srow[side], c->src[side], c->d_tiempo, c->t_n0, c->dt, sr};
        *applied = true;
    }
    cudaError_t e;
    long long threads = 0;
    QuadObs o{};
    if (obs) o = quad_obs(c, 1 - side, *obs, &threads);
    if (threads) {
        const int all = blocks + (int)((threads + kQuadThreads - 1) / kQuadThreads);
        e = side ? launch_after(c->stream, all, kQuadThreads, k_quad<1, true>, v, s, g, src, o, chunk, bx, blocks)
                 : launch_after(c->stream, all, kQuadThreads, k_quad<0, true>, v, s, g, src, o, chunk, bx, blocks);
    } else {
        e = side ? launch_after(c->stream, blocks, kQuadThreads, k_quad<1, false>, v, s, g, src, '\0', chunk, bx, blocks)
                 : launch_after(c->stream, blocks, kQuadThreads, k_quad<0, false>, v, s, g, src, '\0', chunk, bx, blocks);
    }
    return e == cudaSuccess ? SGPU_OK : cuda_error(c, "k_quad", e);
}

template <int SIDE, int MODE> static cudaError_t launch_part(sgpu_ctx* c) {
    const QuadSide s = quad_side(c, SIDE);
    const int bx = (s.threads + kQuadThreads - 1) / kQuadThreads;
    const int chunk = quad_chunk(bx, s.nz);
    return launch_after(c->stream, bx * ((s.nz + chunk - 1) / chunk), kQuadThreads, k_quad_part<SIDE, MODE>, quad_view(c), s, chunk, bx);
}

sgpu_status launch_quad_part(sgpu_ctx* c, int side, int what) {
    const sgpu_status st = quad_prepare(c);
    if (st) return st;
    cudaError_t e;
    switch (4 * side + what) {
        case 0: e = launch_part<0, kBulk | kCx>(c); break;
        case 1: e = launch_part<0, kBulk | kCy>(c); break;
        case 2: e = launch_part<0, kBulk | kCz>(c); break;
        case 3: e = launch_part<0, kCpml | kAll>(c); break;
        case 4: e = launch_part<1, kBulk | kCx>(c); break;
        case 5: e = launch_part<1, kBulk | kCy>(c); break;
        case 6: e = launch_part<1, kBulk | kCz>(c); break;
        default: e = launch_part<1, kCpml | kAll>(c); break;
    }
    return e == cudaSuccess ? SGPU_OK : cuda_error(c, "k_quad_part", e);
}

// What steps need on the device before they are captured: a graph holds no
// allocation.
sgpu_status quad_ready(sgpu_ctx* c) {
    const sgpu_status st = quad_prepare(c);
    return st ? st : quad_sources(c);
}

}  // namespace sgpu
