// SH (toroidal) engine: replaces src/SGTsh/SGTsh-MPI.f90:404-555.
//
// Kernels (this file is compiled without fused multiply-add, so scalar
// operations round as the Fortran's do; the band solves spell fused operations
// and a refined reciprocal out, and k_sh_coef and k_sh_epi multiply by
// reciprocals):
//   k_sh_omega   per-omega band pieces a0, a2 (cala0, cala2, overlap,
//                src/SGTsh/calmat.f90:267-304, 386-423; calcoef,
//                src/SGTsh/others.f90:772-800)
//   k_sh_factor, k_sh_join, k_sh_walk
//                assembly a = a0 + l(l+1) a2 (cala, calmat.f90:309-324) and
//                the complex-symmetric tridiagonal solve (dclisb0,
//                dcsbsub0, src/SGTsh/dclib.f90:1-137) of three basis
//                right-hand sides, the two source rows and the surface row,
//                in segments of rows.
//   k_sh_coef    source terms (calga, calg2, calmat.f90:329-353, 427-479),
//                back-propagation sources (calbveczero, trial.f90:120-157):
//                each slot's weights of the basis solutions, and the cutoff
//                probe |g0(nn)| of imt = 3.
//   k_sh_fields  receiver interpolation (interpolate, others.f90:843-891):
//                the per-order receiver fields of every active (m, source)
//                slot.
//   k_sh_scan    the cutoff test (calamp, others.f90:805-824, and the
//                ismall > 20 rule, SGTsh-MPI.f90:431-436) in the
//                reference's order.
//   k_sh_epi     turns the l-contractions into TSGT / RSGT / SYNN
//                (calu, locallyCartesianDerivatives, udertotsgtSH,
//                udertorsgtSH, utosynnSH, others.f90:132-367, 829-838).
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cmath>

#include "engine.cuh"

namespace dsm {
namespace {

constexpr int SH_NSLOT1 = 8;  // |m| = 1: m = -1, +1 x {imt 4, imt 5, back 2, back 3}
constexpr int SH_NSLOT2 = 6;  // |m| = 2: m = -2, +2 x {imt 2, imt 3, imt 6}
constexpr int SH_NF = 3;      // fields: W/lsq, W'/lsq, l(l+1) W/lsq

struct ShDev {
    int nn, nzone, R, ncap, srow, ins, spn;
    double spo, r0, mu0, tlen, omegai;
    const int *nlayer, *isp, *jsp;
    const double *qmu;
    const double *t, *h1, *h2, *h3, *h4;  // [4*nnlayer]
    const double *g;                      // gt, gh1..gh4: [5][8]
    const int* rcap;                      // [R][3] capture index of the stencil nodes
    int cap_nn;                           // capture index of the surface row
    const double *wv, *wd;                // [R][3]
};

__device__ __forceinline__ cd calcoef1(double omega, double q) {
    if (q <= 0.0) return mk(1.0);
    double aa = (omega == 0.0) ? 1.0 : 1.0 + log(omega / (2.0 * kPi)) / (kPi * q);
    double bb = 1.0 / (2.0 * q);
    return mk(aa, bb) * mk(aa, bb);
}

// a0/a2 of one frequency: layout [(nn+1)][2] (k = 0 off-diagonal, 1 diagonal)
__global__ void k_sh_omega(ShDev d, const int* __restrict__ freqs, cd* __restrict__ a0,
                           cd* __restrict__ a2) {
    int w = blockIdx.y;
    int jj = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (jj > d.nn) return;
    double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
    cd comega2 = mk(omega, -d.omegai) * mk(omega, -d.omegai);
    cd s0d = mk(0.0), s0o = mk(0.0), s2d = mk(0.0), s2o = mk(0.0);
    for (int z = 0; z < d.nzone; ++z) {
        int nl = d.nlayer[z], i = jj - d.isp[z] + 1;
        if (i < 1 || i > nl + 1) continue;
        cd coef = calcoef1(omega, d.qmu[z]);
        const int o = d.jsp[z] - 2;  // element entry n (1-based) -> array index o + n
        auto e0 = [&](int n) {
            double h = d.h1[o + n] - d.h2[o + n] + d.h3[o + n] - 2.0 * d.h4[o + n];
            return comega2 * mk(d.t[o + n]) - coef * mk(h);
        };
        auto e2 = [&](int n) { return -coef * mk(d.h4[o + n]); };
        int nsize = nl + 1;
        if (i == 1) {
            s0d = s0d + e0(1);
            s2d = s2d + e2(1);
        } else if (i == nsize) {
            s0d = s0d + e0(4 * nl);
            s2d = s2d + e2(4 * nl);
        } else {
            s0d = s0d + e0(4 * i - 4) + e0(4 * i - 3);
            s2d = s2d + e2(4 * i - 4) + e2(4 * i - 3);
        }
        if (i >= 2) {
            s0o = s0o + e0(4 * i - 6);
            s2o = s2o + e2(4 * i - 6);
        }
    }
    size_t base = ((size_t)w * (d.nn + 1) + jj) * 2;
    a0[base + 0] = s0o;
    a0[base + 1] = s0d;
    a2[base + 0] = s2o;
    a2[base + 1] = s2d;
}

// ---- the tridiagonal solves, cut into segments of rows by one-row
// separators; the two source rows and the surface row are separators too, so
// no segment holds a right-hand side.  As psv_seg.cu, with half-width 1: a
// thread eliminates one segment of one system upward, carrying the fill-in f
// to the separator below it, and keeps the product of the back-substitution
// steps since the last captured row, x_low = p x_high + q x_left.  16 slices
// of the 256-frequency grid (17 824 systems): 1.96 ms with one chain of all
// rows per thread and the multipliers in memory, 0.24 ms so.
constexpr int SH_MAXSEG = 16;
constexpr int SH_RECS = 2;  // records of a captured row (w, wf), of a gap (p, q)
struct ShPlan {
    int nseg;                           // >= 2, the last one above the source rows s, s+1
    int a[SH_MAXSEG], b[SH_MAXSEG];     // rows [a, b] of each
    int clo[SH_MAXSEG], chi[SH_MAXSEG]; // its captured rows [clo, chi) in ascending order
    int merged;                         // 1: source row s+1 is the surface row
    int ifcap[SH_MAXSEG + 2];           // capture slot of each separator, source row, surface row, or -1
};
struct ShSeg {
    const int *caprow, *capslot;  // captured rows ascending (ended by INT_MAX), their slots
    cd *Lrec, *Grec, *Send, *Xif; // [row][2], [row][2], [segment][3], [interface row][3], each [nsys] last
};

// fused complex operations
__device__ __forceinline__ cd fmul(cd a, cd b) {
    return mk(fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re));
}
__device__ __forceinline__ cd fnmul(cd a, cd b) {  // -a b
    return mk(fma(-a.re, b.re, a.im * b.im), fma(-a.re, b.im, -a.im * b.re));
}
// c + a b, c - a b: the real part of the product is rounded first, the sum
// that follows cancels and is then mostly exact
__device__ __forceinline__ cd fmac(cd c, cd a, cd b) {
    return mk(__dadd_rn(c.re, fma(a.re, b.re, -__dmul_rn(a.im, b.im))), fma(a.re, b.im, fma(a.im, b.re, c.im)));
}
__device__ __forceinline__ cd fmsub(cd c, cd a, cd b) {
    return mk(__dsub_rn(c.re, fma(a.re, b.re, -__dmul_rn(a.im, b.im))), fma(-a.re, b.im, fma(-a.im, b.re, c.im)));
}
// c - m m / D, a pivot's update, with w = m / D and w's own rounding taken out
// of the real part: the pivots' errors add up along the rows.  FP64 outputs
// beyond 90 degrees against 80-bit arithmetic (56 models x 3 frequencies),
// as a geometric mean over the sequential solve's error: products added to c
// one by one 1.05, rounded first 1.00, with this 0.94 (+- 0.01).
__device__ __forceinline__ cd pivot_sub(cd c, cd w, cd m, cd D) {
    const double q = fma(w.im, D.im, fma(-w.re, D.re, m.re));
    return mk(__dsub_rn(c.re, fma(w.re, m.re, fma(q, w.re, -__dmul_rn(w.im, m.im)))),
              fma(-w.re, m.im, fma(-w.im, m.re, c.im)));
}
// band entry k (0 off-diagonal, 1 diagonal) of row j at l(l+1) = xl2
__device__ __forceinline__ cd sh_band(const cd* A0, const cd* A2, int j, int k, double xl2) {
    const cd x = A0[2 * j + k], y = A2[2 * j + k];
    return mk(fma(xl2, y.re, x.re), fma(xl2, y.im, x.im));
}

__global__ void __launch_bounds__(128) k_sh_factor(ShDev d, ShPlan pl, ShSeg g, const cd* __restrict__ a0,
                                                   const cd* __restrict__ a2, WorkList wl, int nsys) {
    const int sys = blockIdx.x * blockDim.x + threadIdx.x;
    if (sys >= nsys) return;
    const int seg = blockIdx.y;
    int w, l;
    wl_map(wl, sys, w, l);
    const cd* A0 = a0 + (size_t)w * (d.nn + 1) * 2;
    const cd* A2 = a2 + (size_t)w * (d.nn + 1) * 2;
    const double xl2 = (double)l * (double)(l + 1);
    const int a = pl.a[seg], b = pl.b[seg];
    // (a > nn above source rows that are the surface's: nothing is eliminated)
    cd dg = mk(1.0), f = mk(0.0), s = mk(0.0), p = mk(0.0), q = mk(0.0);
    if (a <= d.nn) {
        dg = sh_band(A0, A2, a, 1, xl2);
        if (seg > 0) f = sh_band(A0, A2, a, 0, xl2);
    }
    int ci = pl.clo[seg];
    const int chi = pl.chi[seg];
    int next = ci < chi ? g.caprow[ci] : INT_MAX;
    bool low = false, gap = false;
    auto flush = [&] {
        cd* G = g.Grec + (size_t)(ci - 1) * SH_RECS * nsys + sys;
        G[0] = p;
        G[nsys] = q;
    };
    // entries of the next row, one row ahead of use
    cd off = a < d.nn ? sh_band(A0, A2, a + 1, 0, xl2) : mk(0.0), dn = a < d.nn ? sh_band(A0, A2, a + 1, 1, xl2) : mk(0.0);
    for (int j = a; j <= b; ++j) {
        const cd c = off, dc = dn;
        const int jn = min(j + 2, d.nn);
        off = sh_band(A0, A2, jn, 0, xl2);
        dn = sh_band(A0, A2, jn, 1, xl2);
        const cd r = crcp(dg), wv = fmul(c, r), wf = fmul(f, r);
        dg = pivot_sub(dc, wv, c, dg);
        s = fmsub(s, wf, f);
        f = fnmul(wv, f);
        if (j == next) {
            if (gap) flush();
            cd* L = g.Lrec + (size_t)ci * SH_RECS * nsys + sys;
            L[0] = wv;
            L[nsys] = wf;
            ++ci;
            next = ci < chi ? g.caprow[ci] : INT_MAX;
            low = true;
            gap = false;
            p = mk(1.0);
            q = mk(0.0);
        } else if (low) {
            gap = true;
            q = fmsub(q, p, wf);
            p = fnmul(p, wv);
        }
    }
    if (gap) flush();
    cd* S = g.Send + (size_t)seg * 3 * nsys + sys;
    S[0] = dg;
    S[nsys] = f;
    S[2 * (size_t)nsys] = s;
}

// Separators, source rows and surface row of one system: chain elimination up
// to the source, 3x3 system for the unit vectors, and back down.
__global__ void __launch_bounds__(128) k_sh_join(ShDev d, ShPlan pl, ShSeg g, const cd* __restrict__ a0,
                                                 const cd* __restrict__ a2, WorkList wl, int nsys,
                                                 cd* __restrict__ Xcap) {
    const int sys = blockIdx.x * blockDim.x + threadIdx.x;
    if (sys >= nsys) return;
    int w, l;
    wl_map(wl, sys, w, l);
    const cd* A0 = a0 + (size_t)w * (d.nn + 1) * 2;
    const cd* A2 = a2 + (size_t)w * (d.nn + 1) * 2;
    const double xl2 = (double)l * (double)(l + 1);
    const int G = pl.nseg - 2;
    auto E = [&](int seg, int i) { return g.Send[((size_t)seg * 3 + i) * nsys + sys]; };
    cd t[SH_MAXSEG - 2];
    cd A = E(0, 0);
    for (int i = 0; i < G; ++i) {
        const cd f = E(i + 1, 1);
        t[i] = fmul(f, crcp(A + E(i + 1, 2)));
        A = fmsub(E(i + 1, 0), f, t[i]);
    }
    const cd m10 = sh_band(A0, A2, d.srow + 1, 0, xl2);
    cd m11 = sh_band(A0, A2, d.srow + 1, 1, xl2), m21 = mk(0.0), m22 = mk(1.0);
    if (!pl.merged) {
        m11 = m11 + E(G + 1, 2);
        m21 = E(G + 1, 1);
        m22 = E(G + 1, 0);
    }
    const cd r0 = crcp(A), l10 = fmul(m10, r0), r1 = crcp(fmsub(m11, l10, m10)), l21 = fmul(m21, r1);
    const cd r2 = crcp(fmsub(m22, l21, m21));
    for (int k = 0; k < 3; ++k) {
        const int unit = pl.merged && k == 2 ? 1 : k;
        cd x0 = mk(unit == 0 ? 1.0 : 0.0), x1 = mk(unit == 1 ? 1.0 : 0.0), x2 = mk(unit == 2 ? 1.0 : 0.0);
        x1 = fmsub(x1, l10, x0);
        x2 = fmsub(x2, l21, x1);
        x2 = fmul(x2, r2);
        x1 = fmsub(fmul(x1, r1), l21, x2);
        x0 = fmsub(fmul(x0, r0), l10, x1);
        auto put = [&](int slot, cd v) {
            g.Xif[((size_t)slot * 3 + k) * nsys + sys] = v;
            if (pl.ifcap[slot] >= 0) Xcap[((size_t)pl.ifcap[slot] * 3 + k) * nsys + sys] = v;
        };
        put(G, x0);
        put(G + 1, x1);
        if (!pl.merged) put(G + 2, x2);
        cd x = x0;
        for (int i = G - 1; i >= 0; --i) {
            x = fnmul(t[i], x);
            put(i, x);
        }
    }
}

// captured rows of one segment, from its upper separator down
__global__ void __launch_bounds__(128) k_sh_walk(ShDev d, ShPlan pl, ShSeg g, int nsys, cd* __restrict__ Xcap) {
    const int sys = blockIdx.x * blockDim.x + threadIdx.x, seg = blockIdx.y;
    if (sys >= nsys) return;
    const int G = pl.nseg - 2, clo = pl.clo[seg];
    int c = pl.chi[seg] - 1;
    if (c < clo) return;
    cd x[3], y[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int up = seg > G ? G + 2 : seg, lo = seg > G ? G + 1 : seg - 1;
        x[k] = g.Xif[((size_t)up * 3 + k) * nsys + sys];
        y[k] = seg > 0 ? g.Xif[((size_t)lo * 3 + k) * nsys + sys] : mk(0.0);
    }
    for (; c >= clo; --c) {
        const int row = g.caprow[c], slot = g.capslot[c];
        const cd* L = g.Lrec + (size_t)c * SH_RECS * nsys + sys;
        const cd wv = L[0], wf = L[nsys];
        if (row < pl.b[seg] && g.caprow[c + 1] != row + 1) {
            const cd* P = g.Grec + (size_t)c * SH_RECS * nsys + sys;
            const cd p = P[0], q = P[nsys];
#pragma unroll
            for (int k = 0; k < 3; ++k) x[k] = fmac(fmul(p, x[k]), q, y[k]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = fmsub(fnmul(wv, x[k]), wf, y[k]);
            Xcap[((size_t)slot * 3 + k) * nsys + sys] = x[k];
        }
    }
}

// calga for one element set (nl elements, 4 entries each), calmat.f90:329-353
__device__ void calga(int nl, cd comega2, double xl2m2, const double* t, const double* h1,
                      const double* h2, const double* h3, const double* h4, cd coef, cd* a) {
    for (int i = 0; i < 4 * nl; ++i) {
        double h = h1[i] - h2[i] + h3[i] + xl2m2 * h4[i];
        a[i] = comega2 * mk(t[i]) - coef * mk(h);
    }
}

// rvec of calbveczero for |m| = 1 (src/SGTsh/trial.f90:120-157)
__device__ cd sh_rvec(int l, int icomp, int m) {
    double xl2 = (double)l * (double)(l + 1);
    double fact = (double)l * (double)(l + 1);
    double coef = sqrt((double)(2 * l + 1) / (4.0 * kPi) / fact);
    cd v;
    if (icomp == 2) v = mk(0.0, 1.0) * xl2 * coef / 2.0;
    else v = -(mk(1.0, 0.0) * xl2 * coef / 2.0);
    if (m < 0) v = -conj(v);
    return v;
}

// Per (omega, l): the slots' weights of the basis solutions, over lsq
// (co[k][sys]: k = 4 sg + 2 q + b for the forward |m| = 1 slots, 8 + 6 sg + 2 q
// + b for |m| = 2, b = 0, 1 of the solutions of the source's two rows; 20 + 2 sg
// + q for the back-propagated |m| = 1 slots, of the third) and the cutoff
// probe.  A warp of the block takes |m| and the sign of m (role = 2 (|m| - 1) +
// sg) of the block's 32 systems; the source matrix is factored in each.
constexpr int SH_NCO = 24;
__global__ void __launch_bounds__(128) k_sh_coef(ShDev d, const int* __restrict__ freqs, WorkList wl, int nsys,
                                                 const cd* __restrict__ Xcap, cd* __restrict__ co, int Lcap,
                                                 double* __restrict__ amps) {
    const int sys = blockIdx.x * 32 + (threadIdx.x & 31), role = threadIdx.x >> 5;
    const int ma = 1 + role / 2, sg = role & 1, m = sg == 0 ? -ma : ma;
    if (sys >= nsys) return;
    int w, l;
    wl_map(wl, sys, w, l);
    // probe: |g0(nn)| of imt = 3 for m = -2, -1, 1, 2
    double* ap = amps + ((size_t)w * Lcap + l) * 4 + (sg == 0 ? 2 - ma : 1 + ma);
    auto put = [&](int k, cd v) { co[(size_t)k * nsys + sys] = v; };
    if (l == 0) {  // the SH m loop is empty at l = 0: fields are zero
        *ap = 0.0;
        return;
    }
    const double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
    const cd comega2 = mk(omega, -d.omegai) * mk(omega, -d.omegai);
    const cd coef = calcoef1(omega, d.qmu[d.spn - 1]);
    const double xl2 = (double)l * (double)(l + 1), lsq = sqrt(xl2), ilsq = 1.0 / lsq;
    // source element matrices (calga) and the 3x3 band of the split element
    cd aa[4], ga[8];
    calga(1, comega2, xl2 - 2.0, d.t + d.ins - 1, d.h1 + d.ins - 1, d.h2 + d.ins - 1,
          d.h3 + d.ins - 1, d.h4 + d.ins - 1, coef, aa);
    calga(2, comega2, xl2 - 2.0, d.g, d.g + 8, d.g + 16, d.g + 24, d.g + 32, coef, ga);
    // overlap(2, ga, ga2): ga2(1,j) off-diagonal, ga2(2,j) diagonal, j = 1..3
    cd o2 = ga[1], o3 = ga[5];
    cd d1 = ga[0], d2 = mk(0.0) + ga[3] + ga[4], d3 = ga[7];
    // dclisb0 on the 3x3 band (nud = 1)
    cd dr1 = mk(1.0) / d1;
    cd L2 = o2 * dr1;
    cd dr2 = mk(1.0) / (d2 - o2 * L2);
    cd L3 = o3 * dr2;
    cd dr3 = mk(1.0) / (d3 - o3 * L3);
    const double b1a = sqrt((double)(2 * l + 1) / (16.0 * kPi));
    const double b1b = (l >= 2) ? sqrt((double)(2 * l + 1) * (double)(l - 1) * (double)(l + 2) / (64.0 * kPi)) : 0.0;
    const double sgn = (m >= 0) ? 1.0 : -1.0;
    double amp = 0.0;
    // slot coefficients (c_s, c_{s+1}) of the forward slots: g2(itmp+1),
    // g2(itmp+2) of calg2 for a unit right-hand side weight
    const cd dmu = mk(d.r0 * d.r0 * d.mu0) * coef;
    for (int k = 0; k < ma + 1; ++k) {
        int imt = (ma == 1) ? (k == 0 ? 4 : 5) : (k == 0 ? 2 : (k == 1 ? 3 : 6));
        double mt12 = imt == 4, mt13 = imt == 5, mt22 = imt == 2, mt33 = imt == 3, mt23 = imt == 6;
        cd c2 = mk(0.0), c3 = mk(0.0), dd = mk(0.0);
        if (ma == 1) {
            dd = mk(b1a) * mk(sgn * mt13, mt12) / dmu;
            c2 = -dd * (ga[4] + ga[5]);
            c3 = -dd * (ga[6] + ga[7]);
        } else if (l >= 2) {
            c2 = mk(b1b / d.r0) * mk(2.0 * mt23, sgn * (mt22 - mt33));
        }
        // dcsbsub0 on the factored 3x3 band (no right-hand side in its first row)
        cd y2 = c2, y3 = c3 - L3 * y2;
        y2 = y2 * dr2;
        y3 = y3 * dr3;
        cd x3 = y3, x2 = y2 - L3 * x3, x1 = mk(0.0) - L2 * x2;
        x3 = x3 + dd;
        cd gs = aa[0] * x1 + aa[1] * x3;
        cd gs1 = aa[2] * x1 + aa[3] * x3;
        if (ma == 2 && l < 2) gs = gs1 = mk(0.0);
        if (imt == 3 && l >= 2)
            amp = cabs_(gs * Xcap[(size_t)d.cap_nn * 3 * nsys + sys] + gs1 * Xcap[((size_t)d.cap_nn * 3 + 1) * nsys + sys]);
        const int k0 = ma == 1 ? 4 * sg + 2 * k : 8 + 6 * sg + 2 * k;
        put(k0, ilsq * gs);
        put(k0 + 1, ilsq * gs1);
    }
    if (ma == 1)
        for (int q = 0; q < 2; ++q) put(20 + 2 * sg + q, ilsq * (-conj(sh_rvec(l, 2 + q, m)) / mk(lsq)));
    *ap = amp;
}

// Receiver fields: a warp takes 32 orders at one receiver (R: the surface).
//
// Bound: the 84 doubles written per order and receiver.  One thread formed the
// weights of an order, dozens of divisions and square roots, and walked 32
// receivers with them, four more divisions per slot: 0.62 ms for 14 600
// systems, 0.23 ms for the 1700 of a second range (14 blocks, one thread's
// chain).  With the weights in their own kernel and a thread per receiver:
// 0.28 and 0.02 ms.
__global__ void __launch_bounds__(128) k_sh_fields(ShDev d, WorkList wl, int nsys, const cd* __restrict__ Xcap,
                                                   const cd* __restrict__ co, double* __restrict__ A1,
                                                   double* __restrict__ A2f, int Lcap) {
    const int sys = blockIdx.x * 32 + (threadIdx.x & 31), r = blockIdx.y * 4 + (threadIdx.x >> 5);
    const int R = d.R;
    if (sys >= nsys || r > R) return;
    int w, l;
    wl_map(wl, sys, w, l);
    // rows ordered (slot, field, re/im, receiver): receivers contiguous
    const size_t rs = (size_t)(R + 1) * Lcap;
    double* A1w = A1 + (size_t)w * (SH_NSLOT1 * SH_NF * 2) * rs + (size_t)r * Lcap + l;
    double* A2w = A2f + (size_t)w * (SH_NSLOT2 * SH_NF * 2) * rs + (size_t)r * Lcap + l;
    const bool surf = r == R;
    auto X = [&](int cap, int k) { return Xcap[((size_t)cap * 3 + k) * nsys + sys]; };
    auto C = [&](int k) { return co[(size_t)k * nsys + sys]; };
    const double xl2 = (double)l * (double)(l + 1);
    auto put3 = [&](double* A, cd Wh, cd Wdh) {
        if (surf) Wdh = mk(0.0);
        const double x2 = surf ? 0.0 : xl2;
        A[0] = Wh.re;
        A[rs] = Wh.im;
        A[2 * rs] = Wdh.re;
        A[3 * rs] = Wdh.im;
        A[4 * rs] = x2 * Wh.re;
        A[5 * rs] = x2 * Wh.im;
    };
    // basis values interpolated at the receiver (value, derivative)
    cd bv[3], bd[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) bv[k] = bd[k] = mk(0.0);
    if (l > 0 && surf) {
#pragma unroll
        for (int k = 0; k < 3; ++k) bv[k] = X(d.cap_nn, k);
    } else if (l > 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int c = d.rcap[3 * r + i];
            const double wvi = d.wv[3 * r + i], wdi = d.wd[3 * r + i];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const cd xv = X(c, k);
                bv[k] = bv[k] + wvi * xv;
                bd[k] = bd[k] + wdi * xv;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < SH_NSLOT1; ++q) {  // |m| = 1: forward, forward, back, back of m = -1, of m = 1
        cd Wh = mk(0.0), Wdh = mk(0.0);
        const int sg = q / 4, k = q % 4;
        if (l > 0 && k < 2) {
            const cd c0 = C(4 * sg + 2 * k), c1 = C(4 * sg + 2 * k + 1);
            Wh = c0 * bv[0] + c1 * bv[1];
            Wdh = c0 * bd[0] + c1 * bd[1];
        } else if (l > 0 && !surf) {  // SYNN takes forward sources only
            const cd cb = C(20 + 2 * sg + k - 2);
            Wh = cb * bv[2];
            Wdh = cb * bd[2];
        }
        put3(A1w + (size_t)q * (SH_NF * 2) * rs, Wh, Wdh);
    }
#pragma unroll
    for (int q = 0; q < SH_NSLOT2; ++q) {  // |m| = 2
        cd Wh = mk(0.0), Wdh = mk(0.0);
        if (l >= 2) {
            const cd c0 = C(8 + 2 * q), c1 = C(8 + 2 * q + 1);
            Wh = c0 * bv[0] + c1 * bv[1];
            Wdh = c0 * bd[0] + c1 * bd[1];
        }
        put3(A2w + (size_t)q * (SH_NF * 2) * rs, Wh, Wdh);
    }
}

// Cutoff scan, one warp per frequency, SCAN_K consecutive orders a lane, with
// the results of the sequential rule (one thread walking the orders took 1.4
// ms for 1100 orders; with one order a lane a warp took 0.05, now 0.02).  Per order l >= 1 the updates are m = -2, -1, 1, 2 (|m| <= l);
// only |m| = 2 has an amplitude, so an order maps ismall v -> ra v + rb:
// all counts reset up to lsuf; above it m = 2 not small resets, else m = -2
// not small leaves 3, else v + 4 (order 1: v + 2).  A prefix maximum gives
// maxamp at each update, a prefix composition of the maps ismall before each
// order; the exit fires at the first order whose ismall exceeds 20.
__global__ void k_sh_scan(int nf, WorkList wl, int Lcap, int maxlmax, double ratl, double tlen,
                          double vtop, double rtop, const int* __restrict__ freqs,
                          const double* __restrict__ amps, CutState* __restrict__ cut,
                          int* __restrict__ status) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= nf) return;
    CutState c = cut[w];
    if (c.done) return;
    const double omega = 2.0 * kPi * (double)freqs[w] / tlen;
    const int lsuf = (int)(omega * rtop / vtop - 0.5) + 1;  // callsuf
    const int l0 = wl.lb[w], l1 = l0 + wl.off[w + 1] - wl.off[w];
    double mx = c.maxamp;
    int v = c.ismall;
    for (int base = l0; base < l1; base += 32 * SCAN_K) {
        const int lf = base + lane * SCAN_K;
        double am[SCAN_K], ap[SCAN_K];  // m = -2, m = 2
        int badpos = INT_MAX;
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            am[j] = ap[j] = 0.0;
            if (lf + j < l1 && lf + j >= 2) {
                const double* p = amps + ((size_t)w * Lcap + lf + j) * 4;
                am[j] = p[0];
                ap[j] = p[3];
            }
        }
        double pm = -1.0;
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            if (!isfinite(am[j]) || !isfinite(ap[j])) {
                badpos = min(badpos, lf + j);
                am[j] = ap[j] = 0.0;
            }
            if (lf + j < l1 && lf + j >= 1) pm = fmax(pm, fmax(fmax(am[j], ap[j]), 0.0));
        }
        badpos = __reduce_min_sync(0xffffffffu, badpos);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, pm, o);
            if (lane >= o) pm = fmax(pm, y);
        }
        // maxamp before this lane's orders, and before each of them
        double run0 = __shfl_up_sync(0xffffffffu, pm, 1);
        run0 = lane == 0 ? mx : fmax(mx, run0);
        double run = run0;
        int ra[SCAN_K], rb[SCAN_K], A = 1, B = 0;  // each order's map v -> ra v + rb, and the lane's
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            const int l = lf + j;
            ra[j] = 1;
            rb[j] = 0;
            if (l < l1 && l >= 1) {
                const double m0 = fmax(run, am[j]), m3 = fmax(fmax(m0, 0.0), ap[j]);
                const double q0 = am[j] != 0.0 && m0 != 0.0 ? am[j] / m0 : 0.0;
                const double q3 = ap[j] != 0.0 && m3 != 0.0 ? ap[j] / m3 : 0.0;
                if (l <= lsuf || !(q3 < ratl)) ra[j] = 0;
                else if (l == 1) rb[j] = 2;
                else if (q0 < ratl) rb[j] = 4;
                else { ra[j] = 0; rb[j] = 3; }
                run = fmax(run, fmax(fmax(am[j], ap[j]), 0.0));
            }
            B = ra[j] * B + rb[j];
            A = ra[j] * A;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int pa = __shfl_up_sync(0xffffffffu, A, o), pb = __shfl_up_sync(0xffffffffu, B, o);
            if (lane >= o) { B = A * pb + B; A = A * pa; }
        }
        const int vafter = A * v + B;
        int vb = __shfl_up_sync(0xffffffffu, vafter, 1);
        if (lane == 0) vb = v;
        int hit = INT_MAX, vhit = 0;
        double mhit = run0;
        run = run0;
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            const int l = lf + j;
            if (hit == INT_MAX && l < l1 && vb > 20) {
                hit = l;
                vhit = vb;
                mhit = run;
            }
            vb = ra[j] * vb + rb[j];
            if (l < l1 && l >= 1) run = fmax(run, fmax(fmax(am[j], ap[j]), 0.0));
        }
        const unsigned ex = __ballot_sync(0xffffffffu, hit != INT_MAX);
        const int e = ex ? __ffs(ex) - 1 : 0, le = __shfl_sync(0xffffffffu, hit, e);
        // an Inf/NaN probe before the exit: the solves broke down (llog -1)
        if (badpos != INT_MAX && (!ex || badpos < le)) {
            if (lane == 0) {
                flag_nonfinite(status, true);
                c.done = 1;
                c.norders = l1;
                c.llog = -1;
                cut[w] = c;
            }
            return;
        }
        if (ex) {
            c.ismall = __shfl_sync(0xffffffffu, vhit, e);
            c.maxamp = __shfl_sync(0xffffffffu, mhit, e);
            if (c.llog > le) c.llog = le;
            c.done = 1;
            c.norders = le;
            if (lane == 0) cut[w] = c;
            return;
        }
        mx = fmax(mx, __shfl_sync(0xffffffffu, pm, 31));
        v = __shfl_sync(0xffffffffu, vafter, 31);
        if (base <= maxlmax && maxlmax < base + 32 * SCAN_K && maxlmax < l1) {
            c.done = 1;
            c.norders = maxlmax + 1;
        }
    }
    c.maxamp = mx;
    c.ismall = v;
    if (lane == 0) cut[w] = c;
}

// Epilogue of the frequencies of a launch (grid.y): thread per (itheta,
// receiver); receiver R is the surface (SYNN).
// TC: double (FP64 contraction) or float (tensor-core contraction)
//
// Bound: a thread's chain through its 14 slots, 285 blocks a frequency for 101
// receivers and 361 distances.  With some twenty divisions a slot and a launch
// per frequency 0.047 ms each; the divisors' reciprocals once per thread and
// the frequencies of a group in one launch: 0.054 ms for two.
constexpr int SH_EPI_W = 32;
__device__ __forceinline__ void put_out(double* p, cd v) { *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im); }
__device__ __forceinline__ void put_out(float* p, cd v) {
    *reinterpret_cast<float2*>(p) = make_float2((float)v.re, (float)v.im);
}
struct ShEpiW {
    int w[SH_EPI_W];
    size_t c1, c2;  // elements from a frequency's outputs to the next's
};
template <class TC, class OT>
__global__ void k_sh_epi(ShDev d, ShEpiW ws, int Th, int Tb, int Thalf, const double* __restrict__ thx,
                         const double* __restrict__ ths, const int* __restrict__ pole,
                         const double* __restrict__ rr, const TC* __restrict__ C1b,
                         const TC* __restrict__ C2b, OT* __restrict__ tsgt,
                         OT* __restrict__ rsgt, OT* __restrict__ synn, int* __restrict__ status) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int R = d.R;
    if (idx >= Th * (R + 1)) return;
    const int w = ws.w[blockIdx.y];
    const TC *C1 = C1b + (size_t)w * ws.c1, *C2 = C2b + (size_t)w * ws.c2;
    int it = idx / (R + 1), r = idx % (R + 1);
    bool surf = r == R;
    const int ic = it < Thalf ? it : 2 * Tb + Th - 1 - it;  // column of basis function 0
    const int M1 = SH_NSLOT1 * (R + 1) * SH_NF * 2, M2 = SH_NSLOT2 * (R + 1) * SH_NF * 2;
    cd T[10], Rg[5], S[5];
    for (auto& v : T) v = mk(0.0);
    for (auto& v : Rg) v = mk(0.0);
    for (auto& v : S) v = mk(0.0);
    if (!pole[it]) {  // at the poles every SH vector harmonic is zero
        const double x = thx[it], s = ths[it];
        const double tc = x / s;  // thetacot = cos/sin
        const double is = 1.0 / s, iri = surf ? 1.0 : 1.0 / rr[r];
        const double i1 = 1.0 / (1 - x * x), xs2 = x * i1;
        for (int ma = 1; ma <= 2; ++ma) {
            const TC* C = ma == 1 ? C1 : C2;
            const int M = ma == 1 ? M1 : M2;
            const int nslot = ma == 1 ? SH_NSLOT1 : SH_NSLOT2;
            for (int q = 0; q < nslot; ++q) {
                int per = ma == 1 ? 4 : 3;
                int sg = q / per, k = q % per;
                int m = sg == 0 ? -ma : ma;
                double sigma = (m < 0 && (ma & 1)) ? -1.0 : 1.0;
                auto G = [&](int f, int b) {
                    size_t row = ((size_t)(q * SH_NF + f) * 2) * (R + 1) + r;
                    size_t col = (size_t)b * Tb + ic;
                    return mk((double)C[row + (size_t)M * col], (double)C[row + (R + 1) + (size_t)M * col]);
                };
                cd P = G(0, 0), D = G(0, 1);
                double mm = (double)m, m2 = mm * mm;
                // u = W bvec / lsq with bvec(2,m) = i m/sin Pbar, bvec(3,m) = -Dbar
                cd u2 = sigma * cmul_i(mm * is, P);
                cd u3 = sigma * (-D);
                if (surf) {
                    if ((ma == 1 && k >= 2)) continue;  // back slots: no SYNN
                    int imt = ma == 1 ? (k == 0 ? 4 : 5) : (k == 0 ? 2 : (k == 1 ? 3 : 6));
                    if (imt == 2) { S[0] = S[0] - 5.e-1 * u2; S[1] = S[1] - 5.e-1 * u2; }
                    if (imt == 3) { S[0] = S[0] - 5.e-1 * u2; S[1] = S[1] + 5.e-1 * u2; }
                    if (imt == 4) { S[3] = S[3] + u2; }
                    if (imt == 5) { S[4] = S[4] + u3; }
                    if (imt == 6) { S[2] = S[2] - u3; }
                    continue;
                }
                cd Pd = G(1, 0), Dd = G(1, 1), LP = G(2, 0);
                cd udr2 = sigma * cmul_i(mm * is, Pd);
                cd udr3 = sigma * (-Dd);
                cd udt2 = sigma * cmul_i(mm, is * D - xs2 * P);
                cd udt3 = sigma * (tc * D - (m2 * i1) * P + LP);
                cd udp2 = sigma * ((-m2 * is) * P);
                cd udp3 = sigma * cmul_i(-mm, D);
                // locallyCartesianDerivatives (u(1) = 0 for SH)
                cd d12 = iri * (mk(0.0) - u2);
                cd d13 = iri * (mk(0.0) - u3);
                cd d21 = udr2;
                cd d22 = iri * udt2;
                cd d23 = iri * (is * udp2 - tc * u3);
                cd d31 = udr3;
                cd d32 = iri * udt3;
                cd d33 = iri * (is * udp3 + tc * u2);
                if (ma == 1 && k >= 2) {
                    int icomp = k == 2 ? 2 : 3;
                    if (icomp == 2) {
                        Rg[0] = Rg[0] - 5.e-1 * d22 - 5.e-1 * d33;
                        Rg[1] = Rg[1] - 5.e-1 * d22 + 5.e-1 * d33;
                        Rg[3] = Rg[3] - 5.e-1 * d12 - 5.e-1 * d21;
                    } else {
                        Rg[2] = Rg[2] - 5.e-1 * d23 - 5.e-1 * d32;
                        Rg[4] = Rg[4] + 5.e-1 * d13 + 5.e-1 * d31;
                    }
                    continue;
                }
                int imt = ma == 1 ? (k == 0 ? 4 : 5) : (k == 0 ? 2 : (k == 1 ? 3 : 6));
                if (imt == 2) {
                    T[1] = T[1] - 2.5e-1 * d22 - 2.5e-1 * d33;
                    T[6] = T[6] - 1.25e-1 * d12 - 1.25e-1 * d21;
                    T[7] = T[7] + 1.25e-1 * d12 + 1.25e-1 * d21;
                    T[8] = T[8] + 1.25e-1 * d22 - 1.25e-1 * d33;
                    T[9] = T[9] + 1.25e-1 * d22 - 1.25e-1 * d33;
                } else if (imt == 3) {
                    T[1] = T[1] + 2.5e-1 * d22 + 2.5e-1 * d33;
                    T[6] = T[6] - 1.25e-1 * d12 - 1.25e-1 * d21;
                    T[7] = T[7] + 1.25e-1 * d12 + 1.25e-1 * d21;
                    T[8] = T[8] - 1.25e-1 * d22 + 1.25e-1 * d33;
                    T[9] = T[9] - 1.25e-1 * d22 + 1.25e-1 * d33;
                } else if (imt == 4) {
                    T[0] = T[0] - 5.e-1 * d22 - 5.e-1 * d33;
                    T[2] = T[2] - 2.5e-1 * d12 - 2.5e-1 * d21;
                    T[3] = T[3] + 2.5e-1 * d12 + 2.5e-1 * d21;
                    T[4] = T[4] + 2.5e-1 * d22 - 2.5e-1 * d33;
                    T[5] = T[5] - 2.5e-1 * d22 + 2.5e-1 * d33;
                } else if (imt == 5) {
                    T[2] = T[2] + 2.5e-1 * d13 + 2.5e-1 * d31;
                    T[3] = T[3] + 2.5e-1 * d13 + 2.5e-1 * d31;
                    T[4] = T[4] - 2.5e-1 * d23 - 2.5e-1 * d32;
                    T[5] = T[5] - 2.5e-1 * d23 - 2.5e-1 * d32;
                } else if (imt == 6) {
                    T[6] = T[6] + 2.5e-1 * d13 + 2.5e-1 * d31;
                    T[7] = T[7] + 2.5e-1 * d13 + 2.5e-1 * d31;
                    T[8] = T[8] - 2.5e-1 * d23 - 2.5e-1 * d32;
                    T[9] = T[9] + 2.5e-1 * d23 + 2.5e-1 * d32;
                }
            }
        }
    }
    {
        bool bad = false;
        for (int c = 0; c < 5; ++c) bad |= surf && nonfinite2(S[c].re, S[c].im);
        for (int c = 0; c < 10; ++c) bad |= !surf && nonfinite2(T[c].re, T[c].im);
        for (int c = 0; c < 5; ++c) bad |= !surf && rsgt && nonfinite2(Rg[c].re, Rg[c].im);
        flag_nonfinite(status, bad);
    }
    if (surf) {
        if (synn)
            for (int c = 0; c < 5; ++c) put_out(synn + 2 * (((size_t)w * Th + it) * 5 + c), S[c]);
        return;
    }
    // records ([r][it][comp]) or the arrays of k_pack's input ([it][r][comp])
    const size_t pt = sizeof(OT) == 4 ? ((size_t)w * R + r) * Th + it : ((size_t)w * Th + it) * R + r;
    for (int c = 0; c < 10; ++c) put_out(tsgt + 2 * (pt * 10 + c), T[c]);
    if (rsgt)
        for (int c = 0; c < 5; ++c) put_out(rsgt + 2 * (pt * 5 + c), Rg[c]);
}

class ShEngine : public Engine {
  public:
    ShDev d{};
    std::vector<int> h_isp, h_nlayer;
    DBuf<int> nlayer, isp, jsp, rcap, caprow, capslot;
    DBuf<double> qmu, t, h1, h2, h3, h4, g, r, rrsta;
    DBuf<cd> a0, a2, Lrec, Grec, Send, Xif, Xcap, co;
    ShPlan plan{};
    int ncap = 0;
    double vtop = 0, rtop = 0;

    ShEngine(const dsm_sh_setup_t* s, const dsm_options_t* o) {
        mode = 0;
        opt = *o;
        init_common(opt.device);
        m_lo = 1;
        R = s->r_n;
        Th = s->theta_n;
        num_t = DSM_SH_NUM_TSGT; num_r = DSM_SH_NUM_RSGT; num_s = DSM_SH_NUM_SYNN;
        tlen = s->tlen; omegai = s->omegai; ratl = s->ratl; maxlmax = s->maxlmax;
        imin = s->imin; imax = s->imax;
        rsgt_sw = 1;  // the SH back-propagation runs unconditionally (SGTsh-MPI.f90:517)
        synn_sw = s->synn_switch == 1;
        if (R <= 0 || Th <= 0 || s->nzone <= 0 || s->nnlayer <= 0) throw Error(DSM_ERR_INVALID, "empty SH set-up");
        const int nn = s->nnlayer + 1;
        d.nn = nn; d.nzone = s->nzone; d.R = R;
        d.ins = s->ins; d.spn = s->spn; d.spo = s->spo; d.r0 = s->r0; d.mu0 = s->mu0;
        d.tlen = tlen; d.omegai = omegai;
        d.srow = s->isp[s->spn - 1] + (int)std::trunc(s->spo);
        if (d.srow < 1 || d.srow + 1 > nn) throw Error(DSM_ERR_INVALID, "source row outside the system");
        nlayer.upload(s->nlayer, s->nzone, st); isp.upload(s->isp, s->nzone, st); jsp.upload(s->jsp, s->nzone, st);
        qmu.upload(s->qmu, s->nzone, st);
        size_t ne = 4 * (size_t)s->nnlayer;
        t.upload(s->t, ne, st); h1.upload(s->h1, ne, st); h2.upload(s->h2, ne, st);
        h3.upload(s->h3, ne, st); h4.upload(s->h4, ne, st);
        std::vector<double> gg(40);
        for (int k = 0; k < 8; ++k) {
            gg[k] = s->gt[k]; gg[8 + k] = s->gh1[k]; gg[16 + k] = s->gh2[k];
            gg[24 + k] = s->gh3[k]; gg[32 + k] = s->gh4[k];
        }
        g.upload(gg, st);
        r.upload(s->r, R, st);
        rrsta.upload(s->rrsta, 3 * (size_t)R, st);
        // callsuf uses the top zone's summed Vsv coefficients and vrmax
        vtop = 0.0;
        for (int i = 0; i < 4; ++i) vtop = vtop + s->vsv[4 * (s->nzone - 1) + i] * 1.0;
        rtop = s->vrmax[s->nzone - 1];
        vtop_ = vtop;
        rtop_ = rtop;
        set_near_orders(0, s->r0, rtop);  // the probe is the surface row
        set_summaries(0, s->nzone, s->vrmin, s->vrmax, s->vsv, s->qmu, s->r0, s->vrmax[s->nzone - 1]);
        // capture rows: receiver stencils and the surface
        std::vector<int> cm(nn + 1, -1), rc(3 * (size_t)R);
        for (int ir = 0; ir < R; ++ir)
            for (int k = 0; k < 3; ++k) {
                int j = s->iista[3 * ir + k];
                if (j < 1 || j > nn) throw Error(DSM_ERR_INVALID, "receiver node outside the system");
                if (cm[j] < 0) cm[j] = ncap++;
                rc[3 * ir + k] = cm[j];
            }
        if (cm[nn] < 0) cm[nn] = ncap++;
        d.cap_nn = cm[nn];
        d.ncap = ncap;
        rcap.upload(rc, st);
        plan_segments(cm);
        // theta tables
        th.th_n = Th;
        th.h_x.resize(Th); th.h_s.resize(Th); th.h_pole.resize(Th);
        for (int i = 0; i < Th; ++i) {
            double tr = s->theta[i] / 180.0 * kPi;
            th.h_x[i] = std::cos(tr);
            th.h_s[i] = std::sin(tr);
            th.h_pole[i] = (tr == 0.0) ? 1 : (tr == kPi ? 2 : 0);
        }
        set_distances(s->theta);
        th.x.upload(th.h_x, st); th.s.upload(th.h_s, st); th.pole.upload(th.h_pole, st);
        build_weights(r.p, rrsta.p);
        d.nlayer = nlayer.p; d.isp = isp.p; d.jsp = jsp.p; d.qmu = qmu.p;
        d.t = t.p; d.h1 = h1.p; d.h2 = h2.p; d.h3 = h3.p; d.h4 = h4.p; d.g = g.p;
        d.rcap = rcap.p; d.wv = wv.p; d.wd = wd.p;
        // batch geometry
        F = opt.freq_batch > 0 ? opt.freq_batch : 16;
        Lc = opt.l_chunk > 0 ? ((opt.l_chunk + 31) / 32) * 32 : 256;
        Lcap = (std::min(maxlmax + 1 + Lc, 2048) + 7) / 8 * 8;
        amp_k = 4;
        rows_m[1] = SH_NSLOT1 * (R + 1) * SH_NF * 2;
        rows_m[2] = SH_NSLOT2 * (R + 1) * SH_NF * 2;
        alloc_batch();
        build_basis(std::min(maxlmax + 1, 2048));
        DSM_CUDA(cudaStreamSynchronize(st));
    }

    // nine parts of the rows below the source and the part above it, of 16
    // rows or more
    void plan_segments(const std::vector<int>& cm) {
        const int nn = d.nn, s = d.srow;
        std::vector<int> row, slot;
        for (int j = 1; j <= nn; ++j)
            if (cm[j] >= 0) {
                row.push_back(j);
                slot.push_back(cm[j]);
            }
        const int nc = (int)row.size();
        row.push_back(INT_MAX);
        caprow.upload(row, st);
        capslot.upload(slot, st);
        const int parts = std::max(1, std::min(SH_MAXSEG - 2, nn / 16)), G8 = std::min(8, parts - 1);
        std::vector<int> sep;
        for (int k = 1; k <= G8; ++k) {
            const int j = (int)((long long)nn * k / (G8 + 1));
            if (j > 1 && j < s - 8) sep.push_back(j);
        }
        const int G = (int)sep.size();
        plan.nseg = G + 2;
        plan.merged = s + 1 == nn;
        for (int i = 0; i < plan.nseg; ++i) {
            plan.a[i] = i == 0 ? 1 : (i <= G ? sep[i - 1] + 1 : s + 2);
            plan.b[i] = i < G ? sep[i] - 1 : (i == G ? s - 1 : nn - 1);
            plan.clo[i] = (int)(std::lower_bound(row.begin(), row.begin() + nc, plan.a[i]) - row.begin());
            plan.chi[i] = std::max(plan.clo[i],
                                   (int)(std::upper_bound(row.begin(), row.begin() + nc, plan.b[i]) - row.begin()));
        }
        for (int& v : plan.ifcap) v = -1;
        for (int i = 0; i < G; ++i) plan.ifcap[i] = cm[sep[i]];
        plan.ifcap[G] = cm[s];
        plan.ifcap[G + 1] = cm[s + 1];
        if (!plan.merged) plan.ifcap[G + 2] = cm[nn];
    }

    void alloc_batch() {
        size_t nn = d.nn;
        // scratch of a system: captured solutions, their rows' and gaps'
        // records, segment ends, interface solutions, slot weights
        size_t per =
            16 * ((size_t)ncap * (3 + 2 * SH_RECS) + (size_t)plan.nseg * 3 + (size_t)(plan.nseg + 1) * 3 + SH_NCO);
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        nsys_max = (int)std::max<size_t>(1024, std::min<size_t>(65536, (fr / 3) / per));
        // no more than a round of a batch can launch (F ranges of at most
        // max(4096, the first range of the top frequency)): contexts that
        // share a device leave each other room
        nsys_max = std::min(nsys_max, std::max(1024, F * std::max({4096, first_span(imax), near_span(0)})));
        // DSM_MAX_SYSTEMS caps the systems per solve launch (and so the
        // factor scratch) below that, e.g. for small profiling captures
        if (const char* e = std::getenv("DSM_MAX_SYSTEMS")) nsys_max = std::max(1024, std::min(nsys_max, std::atoi(e)));
        nsys_max = nsys_max / 32 * 32;
        size_t nsys = nsys_max;
        a0.reserve((size_t)F * (nn + 1) * 2);
        a2.reserve((size_t)F * (nn + 1) * 2);
        Lrec.reserve((size_t)ncap * SH_RECS * nsys);
        Grec.reserve((size_t)ncap * SH_RECS * nsys);
        Send.reserve((size_t)plan.nseg * 3 * nsys);
        Xif.reserve((size_t)(plan.nseg + 1) * 3 * nsys);
        Xcap.reserve((size_t)ncap * 3 * nsys);
        co.reserve((size_t)SH_NCO * nsys);
        Afld[1].reserve((size_t)F * rows_m[1] * Lcap);
        Afld[2].reserve((size_t)F * rows_m[2] * Lcap);
        Cgemm.reserve(c_total());
        cut.reserve(F);
        amps.reserve((size_t)F * Lcap * 4);
        size_t pt, pr, ps;
        out_sizes(&pt, &pr, &ps);
        out_t.reserve(2 * pt * F);
        out_r.reserve(2 * pr * F);
        out_s.reserve(2 * ps * F);
    }

    size_t out_sizes(size_t* nt, size_t* nr, size_t* ns) const override {
        *nt = (size_t)num_t * R * Th;
        *nr = (size_t)num_r * R * Th;
        *ns = (size_t)num_s * Th;
        return *nt;
    }

    void omega_pieces(const int* fr, int nf) override {
        dim3 grid((d.nn + 127) / 128, nf);
        k_sh_omega<<<grid, 128, 0, st>>>(d, fr, a0.p, a2.p);
        DSM_LAUNCH(*this);
    }

    void solve_chunk(const int* fr, int nf, const WorkList& wl, int nsys) override {
        (void)nf;
        const ShSeg g{caprow.p, capslot.p, Lrec.p, Grec.p, Send.p, Xif.p};
        const unsigned nb = (nsys + 127) / 128;
        // algorithmic bytes: the records written and read, the solutions
        // written (the band pieces stay in cache)
        const double alg = (double)ncap * (2.0 * 2 * SH_RECS + 3) * 16.0;
        int id = kid("sh_band_solve");
        kbegin(id);
        k_sh_factor<<<dim3(nb, plan.nseg), 128, 0, st>>>(d, plan, g, a0.p, a2.p, wl, nsys);
        DSM_LAUNCH(*this);
        k_sh_join<<<nb, 128, 0, st>>>(d, plan, g, a0.p, a2.p, wl, nsys, Xcap.p);
        DSM_LAUNCH(*this);
        k_sh_walk<<<dim3(nb, plan.nseg), 128, 0, st>>>(d, plan, g, nsys, Xcap.p);
        kend(id, alg * nsys, 0.0);
        DSM_LAUNCH(*this);
        id = kid("sh_fields");
        kbegin(id);
        k_sh_coef<<<(nsys + 31) / 32, 128, 0, st>>>(d, fr, wl, nsys, Xcap.p, co.p, Lcap, amps.p);
        DSM_LAUNCH(*this);
        k_sh_fields<<<dim3((nsys + 31) / 32, (R + 4) / 4), 128, 0, st>>>(d, wl, nsys, Xcap.p, co.p, Afld[1].p, Afld[2].p,
                                                                       Lcap);
        kend(id, (double)nsys * (R + 1) * (SH_NSLOT1 + SH_NSLOT2) * SH_NF * 16.0, 0.0);
        DSM_LAUNCH(*this);
        stats.solve_bytes += alg * nsys;
    }

    void scan_chunk(int nf, const WorkList& wl) override {
        k_sh_scan<<<(nf + 3) / 4, 128, 0, st>>>(nf, wl, Lcap, maxlmax, ratl, tlen, vtop, rtop,
                                                 d_freqs.p, amps.p, cut.p, dstatus());
        DSM_LAUNCH(*this);
    }

    void epilogue(const int* fr, const std::vector<int>& ws, int nf, cudaStream_t s) override {
        (void)fr;
        const int n = Th * (R + 1);
        for (size_t i = 0; i < ws.size(); i += SH_EPI_W) {
            const int k = (int)std::min<size_t>(SH_EPI_W, ws.size() - i);
            ShEpiW e{};
            for (int j = 0; j < k; ++j) e.w[j] = ws[i + j];
            const dim3 grid((n + 127) / 128, k);
            int id = kid("sh_epilogue");
            kbegin(id, s);
            if (mixed()) e.c1 = e.c2 = c_total();  // FP64: one frequency's outputs at a time
            auto launch = [&](auto* c1, auto* c2, auto* ot, auto* orr, auto* os) {
                k_sh_epi<<<grid, 128, 0, s>>>(d, e, Th, Tb, Thalf, th.x.p, th.s.p, th.pole.p, r.p, c1, c2, ot, orr, os,
                                              dstatus());
            };
            auto outs = [&](auto* c1, auto* c2) {
                if (rec_direct) launch(c1, c2, rec_t(), rec_r(nf), rec_s(nf));
                else launch(c1, c2, out_t.p, out_r.p, synn_sw ? out_s.p : nullptr);
            };
            if (mixed()) outs(c32(0, 1), c32(0, 2));
            else outs(c64(1), c64(2));
            kend(id, 0.0, 0.0, s);
            DSM_LAUNCH(*this);
        }
    }
};

}  // namespace

Engine* make_sh_engine(const dsm_sh_setup_t* s, const dsm_options_t* o) { return new ShEngine(s, o); }

}  // namespace dsm
