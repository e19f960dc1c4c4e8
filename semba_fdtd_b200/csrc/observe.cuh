// Per-node device code of the volume probes and the far-field surface
// transform, shared by their own kernels (kernels.cu, farfield.cu) and the
// quad kernels (quads.cu).
#pragma once
#include "sgpu_internal.h"

namespace sgpu {

// What the surface transform needs of a FarField on the device.
struct FarArgs {
    FarPatch patch[kFarPatches];
    int npatch, samples, nf, ndecim, w_m;
    double2* acc;
    const double2* wE;
    const double2* wH;
};

namespace dev {

// Sampled node q of a volume probe after step n.  Frequency domain:
// V = V + w * F in complex(8) per frequency, component and node
// (observation.F90:3527-3600); else the node's three values go into the frame
// of step n.
template <bool FREQ>
__device__ __forceinline__ void vol_probe_node(const KGrid& g, const VolProbe& p, int n, int ox, int oy, int oz,
                                               long long nodes, long long q) {
    const int ii = (int)(q % p.ni), jj = (int)((q / p.ni) % p.nj), kk = (int)(q / ((long long)p.ni * p.nj));
    const long long c = (long long)((p.i0 + ii) * p.tr[0] - ox) + (long long)g.pitch * ((p.j0 + jj) * p.tr[1] - oy) +
                        g.plane * (long long)((p.k0 + kk) * p.tr[2] - oz);
    const int f0 = p.magnetic ? 3 : 0;
    const float v[3] = {g.F[f0][c], g.F[f0 + 1][c], g.F[f0 + 2][c]};
    if (FREQ) {
        const int m = n - p.w_n0;
        if (m < 0 || m >= p.w_steps) return;
        for (int f = 0; f < p.nf; ++f) {
            const double2 w = p.w[(long long)m * p.nf + f];
            for (int comp = 0; comp < 3; ++comp) {
                double2* a = p.acc + (((long long)f * 3 + comp) * nodes + q);
                double2 x = *a;
                x.x = x.x + w.x * (double)v[comp];
                x.y = x.y + w.y * (double)v[comp];
                *a = x;
            }
        }
    } else {
        if (n < p.n_first || n >= p.n_last || (n - p.n_first) % p.every) return;
        const long long slot = (long long)((n - p.n_first) / p.every) % p.cap;
        for (int comp = 0; comp < 3; ++comp) p.ring[(slot * 3 + comp) * nodes + q] = v[comp];
    }
}

// Whether step n is sampled by the surface transform, and its weight index.
__device__ __forceinline__ bool far_step(const FarArgs& a, int n, int& m) {
    if ((n - 1) % a.ndecim) return false;  // mod(ntime-1, Ndecim) /= 0 (Fortran MOD keeps the dividend's sign)
    // sampled steps before this one since step 0: the weight index
    m = a.ndecim == 1 ? n : (n - 1) / a.ndecim;
    return m >= 0 && m < a.w_m;
}

// Sample q of the surface at weight index m, when its component's side is in
// `sides` (1 electric, 2 magnetic, 3 both): S += w * F for every frequency.
__device__ __forceinline__ void far_sample(const KGrid& g, const FarArgs& a, int m, int sides, int ox, int oy, int oz, int q) {
    int p = 0;
    while (p + 1 < a.npatch && q >= a.patch[p + 1].off) ++p;
    const FarPatch& P = a.patch[p];
    if (!((P.comp >= 3 ? 2 : 1) & sides)) return;
    const int r = q - P.off, w2 = P.hi2 - P.lo2 + 1;
    const int o = P.lo1 + r / w2, u = P.lo2 + r % w2;
    int i, j, k;
    if (P.axis == 0) { i = P.plane; j = u; k = o; }
    else if (P.axis == 1) { i = u; j = P.plane; k = o; }
    else { i = u; j = o; k = P.plane; }
    const long long c = (long long)(i - ox) + (long long)g.pitch * (j - oy) + g.plane * (long long)(k - oz);
    const double v = (double)g.F[P.comp][c];
    const double2* w = (P.comp >= 3 ? a.wH : a.wE) + (long long)m * a.nf;
    for (int f = 0; f < a.nf; ++f) {
        double2* s = a.acc + (long long)f * a.samples + q;
        double2 x = *s;
        const double2 wf = w[f];
        x.x = x.x + wf.x * v;
        x.y = x.y + wf.y * v;
        *s = x;
    }
}

}  // namespace dev
}  // namespace sgpu
