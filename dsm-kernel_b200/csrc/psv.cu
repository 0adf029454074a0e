// P-SV engine: replaces src/SGTpsv/SGTpsv-MPI.f90:551-1095.
//
// Kernels (this file is compiled without fused multiply-add; the band solves,
// psv_seg.cu, and the order-0 solve spell fused operations and a refined
// reciprocal out, so they follow the reference's equations to rounding, the
// others its operations):
//   k_psv_omega  per-omega, per-zone band blocks A0, A1, A2 (cala0, cala1,
//                cala2, calhml, overlapa, calb0, calb2, overlapb,
//                src/SGTpsv/calmat.f90:452-742; calcoef :409-447)
//   psv_seg.cu   the band systems of orders l >= 1 (cala, calbc, :747-809;
//                dcsymbdl0 / dcsbdlv0, src/SGTpsv/dcsymbdl.f90:2-166): six
//                basis right-hand sides (the four source rows jtmp..jtmp+3
//                and the surface rows nn-1, nn), in segments of rows.
//   k_psv_l0_*   l = 0: the tridiagonal compaction (rea2 / rea2_back,
//                calmat.f90:1247-1389), its solves (dcsymbdl0/dcsbdlv0
//                with half-width 1; a block per frequency) and fields.
//   k_psv_abnum, k_psv_coef
//                source terms (calabnum, calya + rk3, calg, glu,
//                calmat.f90:815-1171), back-propagation sources
//                (caldveczero, trial.f90:326-364): each slot's weights of the
//                basis solutions, and the probe of calamp (imt = 1, m = 0).
//   k_psv_fields receiver interpolation (interpolate, others.f90:1170-1212):
//                the per-order receiver fields of every active slot.
//   k_psv_scan   the cutoff test (calamp, others.f90:1246-1264, the
//                ismall > 20 exit, SGTpsv-MPI.f90:606-609, 902-905).
// The epilogue (TSGT / RSGT / SYNN from the l-contractions) is psv_epi.cu.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "engine.cuh"
#include "psv_epi.cuh"
#include "psv_seg.cuh"

namespace dsm {
namespace {

using psvk::NS0;
using psvk::NS1;
using psvk::NS2;
using psvk::NFLD;  // U, U', V/lsq, V'/lsq, l(l+1) V/lsq
constexpr int NB = 6;                     // basis right-hand sides of a solve

struct PsvDev {
    int nzone, nn, itmp, R, Th, jsrc, spn;
    int n_sel, n_fel, n_hm;
    const int *iphase, *nlayer, *kkdr, *elem, *hmoff;
    const int* blkoff;      // [nzone] first block column of each zone
    int ncol_tot;
    const double *qmu, *qkappa;
    const double *sel, *fel, *hm;
    // assembly map per global column (1-based, [nn+1])
    const int *amz, *amc;   // [nn+1][2] zone (or -1) and zone-local column
    const int* bcrow;       // 0, 2 or 3
    const double* bcval;
    const int4* rowasm;     // [nn+1] per row: element offsets of the two zones
                            // (x4, -1 none), phase bits (1: zone 0 solid,
                            // 2: zone 1 solid), bcrow
    double tlen, omegai, rmax, r0, ecC0, ecF0, ecL0, ra0, ra1;
    const double* poly;     // [24]
    // receivers
    const int* rcap;        // [R][6] capture index of g0(ksta-1 .. ksta+4)
    const int* stop_row;    // [R] highest local row of each receiver's stencil (ksta+4)
    int cap_n1, cap_n;      // capture index of rows nn-1, nn
    int cap_p0, cap_p1;     // capture index of the probe rows ksta(r_n)-1, ksta(r_n)
    const double *wv, *wd;
    const int* fluid;       // [R]
    int Rs1, Rf;            // receiver rows of the solid class (incl. the surface), fluid receivers
    const int* rrow;        // [R+1] class index of each receiver row (psvk::fld_row)
    const double *lam, *qkp, *fr;  // [R]  lambda, Qkappa, float(r)
    // l = 0 compaction
    int nn0, itmp0, kc0;    // compact size, first row kept, compact row of jtmp
    const int* comp_src;    // global row -> compact row (or 0 when dropped), [nn+1]
    const int* jsta;        // [R]
};

__device__ __forceinline__ cd coefq(double omega, double q) {
    if (q <= 0.0) return mk(1.0);
    double aa = (omega == 0.0) ? 1.0 : 1.0 + log(omega / (2.0 * kPi)) / (kPi * q);
    double bb = 1.0 / (2.0 * q);
    return mk(aa, bb) * mk(aa, bb);
}

// ----------------------------------------------------------- omega pieces
struct ZoneCtx {
    const PsvDev* d;
    int z, off;
    cd c1, c2, comega2;
    __device__ double E(int k, int nnn) const {
        return d->sel[(size_t)k * d->n_sel + (off - 1) + (nnn - 1)];
    }
    // cala0 entry n (1-based, cwork)
    __device__ cd cw0(int n) const {
        if (n % 4 == 1) {
            int nnn = (n + 3) / 4;
            if (nnn % 4 == 3) return mk(0.0);
            cd hh0 = c2 * mk(4.0 * E(DSM_PSV_H1X, nnn)) + c1 * mk(16.0 / 3.0 * E(DSM_PSV_H2N, nnn)) +
                     c1 * mk(-4.0 * E(DSM_PSV_H2N, nnn)) +
                     c2 * mk(2.0 * (E(DSM_PSV_H3AY, nnn) + E(DSM_PSV_H5AY, nnn))) -
                     c1 * mk(4.0 / 3.0 * (E(DSM_PSV_H4AN, nnn) + E(DSM_PSV_H6AN, nnn))) +
                     c2 * mk(3.0 * E(DSM_PSV_H7Z, nnn) - 2.0 * E(DSM_PSV_H7Y, nnn)) +
                     c1 * mk(4.0 / 3.0 * E(DSM_PSV_H8N, nnn));
            return comega2 * mk(E(DSM_PSV_T, nnn)) - hh0;
        }
        if (n % 4 == 0) {
            int nnn = n / 4;
            if (nnn % 4 == 3) return mk(0.0);
            cd hh0 = c1 * mk(E(DSM_PSV_H2L, nnn)) + c1 * mk(-2.0 * E(DSM_PSV_H2N, nnn)) -
                     c1 * mk(E(DSM_PSV_H4AL, nnn) + E(DSM_PSV_H6AL, nnn)) + c1 * mk(E(DSM_PSV_H8L, nnn));
            return comega2 * mk(E(DSM_PSV_T, nnn)) - hh0;
        }
        return mk(0.0);
    }
    // cala1 entry n
    __device__ cd cw1(int n) const {
        if (n % 4 == 2) {
            int nnn = (n + 2) / 4;
            if (nnn % 4 == 3) return mk(0.0);
            cd hh1 = -c2 * mk(2.0 * E(DSM_PSV_H1X, nnn)) - c1 * mk(8.0 / 3.0 * E(DSM_PSV_H2N, nnn)) -
                     c1 * mk(E(DSM_PSV_H2L, nnn)) - c1 * mk(-2.0 * E(DSM_PSV_H2N, nnn)) -
                     c2 * mk(E(DSM_PSV_H3Y, nnn)) - c1 * mk(-2.0 / 3.0 * E(DSM_PSV_H4N, nnn)) +
                     c1 * mk(E(DSM_PSV_H6L, nnn));
            return -hh1;
        }
        if (n % 4 == 3) {
            int nnn = (n + 1) / 4;
            if (nnn % 4 != 2) return mk(0.0);
            cd hh1 = -c2 * mk(2.0 * E(DSM_PSV_H1X, nnn)) - c1 * mk(8.0 / 3.0 * E(DSM_PSV_H2N, nnn)) -
                     c1 * mk(-2.0 * E(DSM_PSV_H2N, nnn)) - c1 * mk(E(DSM_PSV_H2L, nnn)) +
                     c1 * mk(E(DSM_PSV_H4L, nnn)) - c2 * mk(E(DSM_PSV_H5Y, nnn)) +
                     c1 * mk(2.0 / 3.0 * E(DSM_PSV_H6N, nnn));
            return -hh1;
        }
        return mk(0.0);
    }
    // cala2 entry n
    __device__ cd cw2(int n) const {
        if (n % 4 == 1) {
            int nnn = (n + 3) / 4;
            if (nnn % 4 == 3) return mk(0.0);
            return -(c1 * mk(E(DSM_PSV_H2L, nnn)));
        }
        if (n % 4 == 0) {
            int nnn = n / 4;
            if (nnn % 4 == 3) return mk(0.0);
            return -(c2 * mk(E(DSM_PSV_H1X, nnn)) + c1 * mk(4.0 / 3.0 * E(DSM_PSV_H2N, nnn)));
        }
        return mk(0.0);
    }
};

// overlapa (calmat.f90:670-714): band entry (ii, i) of a zone block from the
// element array entries cw(n)
template <class F>
__device__ cd overlapa_entry(int nl, int ii, int i, F cw) {
    int nsize = 2 * (nl + 1), msize = 16 * nl;
    if (i == 1) return ii == 4 ? cw(1) : mk(0.0);
    if (i == 2) return ii == 3 ? cw(2) : (ii == 4 ? cw(4) : mk(0.0));
    if (i % 2 == 1) {  // 3 .. nsize-1
        int n1 = 16 * (i - 3) / 2 + 5;
        if (ii == 2) return cw(n1);
        if (ii == 3) return cw(n1 + 2);
        if (ii == 4) return (i != nsize - 1) ? cw(n1 + 8) + cw(n1 + 12) : cw(msize - 3);
        return mk(0.0);
    }
    int n1 = 16 * (i - 4) / 2 + 6;  // even, 4 .. nsize
    if (ii == 1) return cw(n1);
    if (ii == 2) return cw(n1 + 2);
    if (i != nsize) {
        if (ii == 3) return cw(n1 + 8) + cw(n1 + 12);
        return cw(n1 + 10) + cw(n1 + 14);
    }
    if (ii == 3) return cw(msize - 2);
    return cw(msize);
}

__global__ void k_psv_omega(PsvDev d, const int* __restrict__ freqs, cd* __restrict__ B0,
                            cd* __restrict__ B1, cd* __restrict__ B2) {
    int w = blockIdx.y;
    int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol_tot) return;
    int z = 0;
    while (z + 1 < d.nzone && d.blkoff[z + 1] <= col) ++z;
    int c = col - d.blkoff[z] + 1;
    double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
    cd comega2 = mk(omega, -d.omegai) * mk(omega, -d.omegai);
    cd c1 = coefq(omega, d.qmu[z]);
    cd c2 = coefq(omega, d.qkappa[z]);
    int nl = d.nlayer[z];
    size_t o = ((size_t)w * d.ncol_tot + col) * 4;
    if (d.iphase[z] == 1) {
        ZoneCtx zc{&d, z, d.elem[z], c1, c2, comega2};
        for (int ii = 1; ii <= 4; ++ii) {
            B0[o + ii - 1] = overlapa_entry(nl, ii, c, [&](int n) { return zc.cw0(n); });
            B2[o + ii - 1] = overlapa_entry(nl, ii, c, [&](int n) { return zc.cw2(n); });
            cd a1 = overlapa_entry(nl, ii, c, [&](int n) { return zc.cw1(n); });
            // calhml (calmat.f90:629-664)
            if (ii == 1 || ii == 3) {
                auto H = [&](int k, int lo, int m, int n) {
                    return d.hm[(size_t)k * 4 * d.n_hm + 4 * (size_t)(d.hmoff[z] - 1 + n - 1) + (m - lo)];
                };
                if (c % 2 == 0 && !(ii == 1 && c == 2)) {
                    int m = (-ii + 3) / 2, n = (ii + c - 3) / 2;
                    a1 = a1 - (-(c2 * mk(H(DSM_PSV_H3MY, -2, m, n))) +
                               c1 * mk(2.0 / 3.0 * H(DSM_PSV_H4M2N, -2, m, n)) +
                               c1 * mk(H(DSM_PSV_H6M2L, -2, m, n)));
                } else if (c % 2 == 1 && c >= 3 && c <= 2 * nl + 1 && !(ii == 1 && c == 3)) {
                    int m = (-ii + 5) / 2, n = (ii + c - 4) / 2;
                    a1 = a1 - (c1 * mk(H(DSM_PSV_H4M1L, -1, m, n)) -
                               c2 * mk(H(DSM_PSV_H5MY, -1, m, n)) +
                               c1 * mk(2.0 / 3.0 * H(DSM_PSV_H6M1N, -1, m, n)));
                }
            }
            B1[o + ii - 1] = a1;
        }
    } else {
        cd coef = mk(1.0) / c2;
        const double* p1 = d.fel + (d.elem[z] - 1);
        const double* p2 = d.fel + d.n_fel + (d.elem[z] - 1);
        const double* p3 = d.fel + 2 * (size_t)d.n_fel + (d.elem[z] - 1);
        auto b0 = [&](int n) {
            if (n % 4 == 3) return mk(0.0);
            return -(mk(p1[n - 1]) / comega2) + coef * mk(p3[n - 1]);
        };
        auto b2 = [&](int n) {
            if (n % 4 == 3) return mk(0.0);
            return -(mk(p2[n - 1]) / comega2);
        };
        // overlapb (calmat.f90:720-742)
        auto ovb = [&](int ii, auto f) -> cd {
            if (ii == 4) {
                if (c == 1) return f(1);
                if (c == nl + 1) return f(4 * nl);
                return f(4 * (c - 1)) + f(4 * (c - 1) + 1);
            }
            if (ii == 3 && c >= 2) return f(4 * (c - 2) + 2);
            return mk(0.0);
        };
        for (int ii = 1; ii <= 4; ++ii) {
            B0[o + ii - 1] = ovb(ii, b0);
            B2[o + ii - 1] = ovb(ii, b2);
            B1[o + ii - 1] = mk(0.0);
        }
    }
}

// band entries a(1..4, jj) of one global column for order l (cala + calbc)
__device__ __forceinline__ void assemble(const PsvDev& d, int jj, const cd* __restrict__ B0,
                                         const cd* __restrict__ B1, const cd* __restrict__ B2,
                                         double l2, double lsq, cd a[4]) {
    a[0] = a[1] = a[2] = a[3] = mk(0.0);
    const int4 ra = d.rowasm[jj];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int off = e == 0 ? ra.x : ra.y;
        if (off < 0) break;
        const size_t o = (size_t)off;
        if (ra.z & (1 << e)) {
            for (int ii = 2; ii <= 4; ii += 2) {
                cd x0 = B0[o + ii - 1], x2 = B2[o + ii - 1];
                a[ii - 1] = a[ii - 1] + mk(x0.re + l2 * x2.re, x0.im + l2 * x2.im);
            }
            for (int ii = 1; ii <= 3; ii += 2) {
                cd x1 = B1[o + ii - 1];
                a[ii - 1] = a[ii - 1] + mk(lsq * x1.re, lsq * x1.im);
            }
        } else {
            for (int ii = 3; ii <= 4; ++ii) {
                cd x0 = B0[o + ii - 1], x2 = B2[o + ii - 1];
                a[ii - 1] = a[ii - 1] + mk(x0.re + l2 * x2.re, x0.im + l2 * x2.im);
            }
        }
    }
    if (ra.w == 2) a[1] = mk(d.bcval[jj]);
    else if (ra.w == 3) a[2] = -mk(d.bcval[jj]);
}

// ---------------------------------------------------------------- solve
// Per-omega band pieces by row, in the form of the segmented solve
// (psvseg::band_row): the band entries of row jj at order l are combinations
// of the l-free parts with 1, l(l+1) and sqrt(l(l+1)) (cala), summed over
// the zones that share the row, with the calbc boundary value.  Of the
// twelve parts of the four entries, five are zero in every row of one phase,
// so eight complex numbers a row do: Y1, X2, Y2, X3, Y3, X4, Y4 and the
// phase (1 fluid) for the third entry's factor.  Rows after the band are zero.
__global__ void k_psv_rows(PsvDev d, const cd* __restrict__ B0all, const cd* __restrict__ B1all,
                            const cd* __restrict__ B2all, cd* __restrict__ P8, int nrow) {
    const int w = blockIdx.y;
    const int jj = blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= nrow) return;
    const size_t bo = (size_t)w * d.ncol_tot * 4;
    const cd *B0 = B0all + bo, *B1 = B1all + bo, *B2 = B2all + bo;
    cd A[4], B[4], C[4];
    bool fluid = false;
    for (int q = 0; q < 4; ++q) A[q] = B[q] = C[q] = mk(0.0);
    if (jj >= 1 && jj <= d.nn) {
        const int4 ra = d.rowasm[jj];
        for (int e = 0; e < 2; ++e) {
            const int off = e == 0 ? ra.x : ra.y;
            if (off < 0) break;
            const size_t o = (size_t)off;
            if (ra.z & (1 << e)) {
                for (int ii = 2; ii <= 4; ii += 2) {
                    A[ii - 1] = A[ii - 1] + B0[o + ii - 1];
                    B[ii - 1] = B[ii - 1] + B2[o + ii - 1];
                }
                for (int ii = 1; ii <= 3; ii += 2) C[ii - 1] = C[ii - 1] + B1[o + ii - 1];
            } else {
                fluid = true;
                for (int ii = 3; ii <= 4; ++ii) {
                    A[ii - 1] = A[ii - 1] + B0[o + ii - 1];
                    B[ii - 1] = B[ii - 1] + B2[o + ii - 1];
                }
            }
        }
        if (ra.w == 2) { A[1] = mk(d.bcval[jj]); B[1] = C[1] = mk(0.0); }
        else if (ra.w == 3) { A[2] = -mk(d.bcval[jj]); B[2] = C[2] = mk(0.0); }
    }
    cd* out = P8 + ((size_t)w * nrow + jj) * psvseg::ROW_CD;
    out[0] = C[0];
    out[1] = A[1];
    out[2] = B[1];
    out[3] = A[2];
    out[4] = fluid ? B[2] : C[2];
    out[5] = A[3];
    out[6] = B[3];
    out[7] = mk(fluid ? 1.0 : 0.0);
}

// fused complex products
__device__ __forceinline__ cd cmulf(cd a, cd b) {
    return mk(fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re));
}
__device__ __forceinline__ cd cmsubf(cd c, cd a, cd b) {  // c - a b
    return mk(fma(-a.re, b.re, fma(a.im, b.im, c.re)), fma(-a.re, b.im, fma(-a.im, b.re, c.im)));
}
// c + a b, with fused multiply-adds when FAST (mixed precision)
template <bool FAST>
__device__ __forceinline__ cd caddmulT(cd c, cd a, cd b) {
    if (FAST) return mk(fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im)));
    return c + a * b;
}

// ------------------------------------------------------------ l = 0 path
// Compacted tridiagonal (rea2), its solves for the three m = 0 sources (imt
// 1..3) and the back-propagated vertical force, and the fields of column l = 0.
__device__ void calabnum_dev(const PsvDev& d, double omega, cd c1, cd c2, cd* anum, cd* bnum);
__device__ void calg_l0(const PsvDev& d, cd coef1, cd coef2, const cd* ab, cd* g);

// (1) compaction, one thread per compact row: c(1,i), c(2,i) of rea2 from the
// assembled l = 0 band (l0col: global column, l0e1: band row of c(1,i), 0 for none)
__global__ void k_psv_l0_build(PsvDev d, const cd* __restrict__ B0all, const cd* __restrict__ B1all,
                               const cd* __restrict__ B2all, const int* __restrict__ l0col,
                               const int* __restrict__ l0e1, cd* __restrict__ Cc) {
    int w = blockIdx.y;
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (i > d.nn0) return;
    const size_t bo = (size_t)w * d.ncol_tot * 4;
    cd a[4];
    assemble(d, l0col[i], B0all + bo, B1all + bo, B2all + bo, 0.0, 0.0, a);
    int e1 = l0e1[i];
    cd* C = Cc + (size_t)w * (d.nn0 + 1) * 2;
    C[2 * i] = e1 == 2 ? a[1] : (e1 == 3 ? a[2] : mk(0.0));
    C[2 * i + 1] = a[3];
}

// (2) one CTA per frequency: right-hand sides (calg at l = 0 for imt 1..3,
// the back-propagated vertical force) and the tridiagonal solve (dcsymbdl0 /
// dcsbdlv0 with half-width 1).  Solutions in Dv[w][i][4].
// The recurrence is cut over the threads: each takes a run of consecutive
// rows, eliminates all but its last one (carrying the fill-in f to the last
// row of the run below), the runs' last rows form a tridiagonal system of
// one row a thread, solved by parallel cyclic reduction, and each thread
// substitutes back through its run.  A chain of n / 256 rows and 8 reduction
// steps instead of n rows: 4.9 -> 0.2 ms for the 16 780 rows of the
// 2048-frequency grid.
constexpr int L0_T = 256;   // threads (runs) of a solve
constexpr int L0_MIN = 8;   // rows of a run, at least
constexpr size_t L0_SMEM = (size_t)2 * L0_T * 7 * sizeof(cd);

__global__ void __launch_bounds__(L0_T) k_psv_l0_solve(PsvDev d, const int* __restrict__ freqs, int nf,
                                                       const cd* __restrict__ ab, cd* __restrict__ Cc,
                                                       cd* __restrict__ Dv, int back) {
    const int w = blockIdx.x;
    if (w >= nf) return;
    const int n0 = d.nn0, it0 = d.itmp0, tid = threadIdx.x;
    cd* C = Cc + (size_t)w * (n0 + 1) * 2;
    cd* D = Dv + (size_t)w * (n0 + 1) * 4;
    extern __shared__ __align__(16) unsigned char l0_smem[];
    __shared__ int srr[5];
    __shared__ cd srv[5][4];
    __shared__ int snr;
    if (tid == 0) {
        const double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
        const cd c1 = coefq(omega, d.qmu[d.spn - 1]), c2 = coefq(omega, d.qkappa[d.spn - 1]);
        cd g[12];
        calg_l0(d, c1, c2, ab + (size_t)w * 320, g);
        // sparse right-hand sides: rea2 keeps the U rows of g0(jtmp..jtmp+3)
        int nr = 0;
        for (int k = 0; k < 4; ++k) {
            int cr = d.comp_src[d.jsrc + k];
            if (cr <= 0) continue;
            srr[nr] = cr;
            for (int b = 0; b < 4; ++b) srv[nr][b] = mk(0.0);
            ++nr;
        }
        for (int imt = 1; imt <= 3; ++imt) {
            int q = 0;
            for (int k = 0; k < 4; ++k)
                if (d.comp_src[d.jsrc + k] > 0) srv[q++][imt - 1] = g[4 * (imt - 1) + k];
        }
        // caldveczero at l = 0: bvec(1,0) = cmplx(coef), single precision
        double coef = sqrt((double)1 / (4.0 * kPi) / 1.0);
        int cr = d.comp_src[d.nn - 1];
        srr[nr] = cr > 0 ? cr : -1;
        for (int b = 0; b < 4; ++b) srv[nr][b] = mk(0.0);
        if (back) srv[nr][3] = -conj(mk((double)(float)coef));
        snr = nr + 1;
    }
    __syncthreads();
    const int nr = snr;
    auto rhs = [&](int row, int b) {
        cd v = mk(0.0);
        for (int k = 0; k < nr; ++k)
            if (srr[k] == row) v = v + srv[k][b];  // a source's row can be the surface row
        return v;
    };
    const int N = n0 - it0 + 1, m = max(L0_MIN, (N + L0_T - 1) / L0_T), nt = (N + m - 1) / m;
    const int r0 = it0 + tid * m, r1 = min(r0 + m, n0 + 1) - 1;  // rows r0 .. r1, r1 the run's last
    // the reduced rows: a x(t-1) + b x(t) + c x(t+1) = y, ping-pong buffers
    struct Red {
        cd a, b, c, y[4];
    };
    Red* red = reinterpret_cast<Red*>(l0_smem);
    cd left[4], sl = mk(0.0);  // what the run adds to the row below it
    Red me;
    me.a = me.c = mk(0.0);
    me.b = mk(1.0);
    for (int b = 0; b < 4; ++b) me.y[b] = left[b] = mk(0.0);
    bool has = false;  // a right-hand side inside the run
    for (int k = 0; k < nr; ++k) has = has || (srr[k] >= r0 && srr[k] <= r1);
    if (tid < nt) {
        cd f = tid > 0 ? C[2 * r0] : mk(0.0), dg = C[2 * r0 + 1], y[4];
        for (int b = 0; b < 4; ++b) y[b] = has ? rhs(r0, b) : mk(0.0);
        cd nc = r0 < r1 ? C[2 * r0 + 2] : mk(0.0), nd = r0 < r1 ? C[2 * r0 + 3] : mk(0.0);
        for (int i = r0; i < r1; ++i) {
            const cd c = nc, dn = nd;
            if (i + 1 < r1) {
                nc = C[2 * i + 4];
                nd = C[2 * i + 5];
            }
            const cd r = crcp(dg), wv = cmulf(c, r), wf = cmulf(f, r);
            C[2 * i] = wv;
            C[2 * i + 1] = wf;
            sl = cmsubf(sl, wf, f);
            dg = cmsubf(dn, wv, c);
            f = cmsubf(mk(0.0), wv, f);
            if (has) {
                for (int b = 0; b < 4; ++b) {
                    D[4 * i + b] = cmulf(y[b], r);
                    left[b] = cmsubf(left[b], wf, y[b]);
                    y[b] = cmsubf(rhs(i + 1, b), wv, y[b]);
                }
            }
        }
        me.a = f;
        me.b = dg;
        for (int b = 0; b < 4; ++b) me.y[b] = y[b];
    }
    // the run above adds its Schur part to this run's last row
    red[tid].a = sl;
    red[tid].c = me.a;
    for (int b = 0; b < 4; ++b) red[tid].y[b] = left[b];
    __syncthreads();
    if (tid + 1 < nt) {
        const Red& up = red[tid + 1];
        me.b = me.b + up.a;
        me.c = up.c;
        for (int b = 0; b < 4; ++b) me.y[b] = me.y[b] + up.y[b];
    }
    __syncthreads();
    red[tid] = me;
    __syncthreads();
    int cur = 0;
    for (int h = 1; h < nt; h *= 2, cur ^= 1) {
        const Red* src = red + cur * L0_T;
        if (tid < nt) {
            const Red self = src[tid];
            me = self;
            me.a = me.c = mk(0.0);
            if (tid >= h) {
                const Red& lo = src[tid - h];
                const cd al = cmulf(self.a, crcp(lo.b));
                me.b = cmsubf(me.b, al, lo.c);
                me.a = cmsubf(mk(0.0), al, lo.a);
                for (int b = 0; b < 4; ++b) me.y[b] = cmsubf(me.y[b], al, lo.y[b]);
            }
            if (tid + h < nt) {
                const Red& hi = src[tid + h];
                const cd ga = cmulf(self.c, crcp(hi.b));
                me.b = cmsubf(me.b, ga, hi.a);
                me.c = cmsubf(mk(0.0), ga, hi.c);
                for (int b = 0; b < 4; ++b) me.y[b] = cmsubf(me.y[b], ga, hi.y[b]);
            }
            red[(cur ^ 1) * L0_T + tid] = me;
        }
        __syncthreads();
    }
    cd x[4];
    const cd r = crcp(me.b);
    for (int b = 0; b < 4; ++b) x[b] = cmulf(me.y[b], r);
    __syncthreads();
    for (int b = 0; b < 4; ++b) red[tid].y[b] = x[b];
    __syncthreads();
    if (tid >= nt) return;
    for (int b = 0; b < 4; ++b) {
        left[b] = tid > 0 ? red[tid - 1].y[b] : mk(0.0);
        D[4 * r1 + b] = x[b];
    }
    for (int i = r1 - 1; i >= r0; --i) {
        const cd wv = C[2 * i], wf = C[2 * i + 1];
        for (int b = 0; b < 4; ++b) {
            x[b] = cmsubf(cmsubf(has ? D[4 * i + b] : mk(0.0), wv, x[b]), wf, left[b]);
            D[4 * i + b] = x[b];
        }
    }
}

// (3) fields of order 0, one thread per (frequency, receiver): m = 0 slots
// q = 0..2 (imt 1..3) and 3 (back), U and dU/dr (calup0 uses u(1) only)
// rows ordered (field group, slot, field, re/im, receiver): receivers
// contiguous, so the epilogue's threads (consecutive receivers) read
// consecutive rows; fields a fluid receiver does not need have no row
template <class T>
__device__ __forceinline__ void put_field(T* Aw, int Lcap, int nq, const PsvDev& d, int rr, int q, int f, cd v) {
    int im;
    const long long row = psvk::fld_row(nq, d.Rs1, d.Rf, q, f, rr, &im);
    if (row < 0) return;
    Aw[(size_t)row * Lcap] = (T)v.re;
    Aw[((size_t)row + im) * Lcap] = (T)v.im;
}

template <class T>
__global__ void k_psv_l0_fields(PsvDev d, const cd* __restrict__ Dv, T* __restrict__ A0f, T* __restrict__ A1f,
                                T* __restrict__ A2f, int Lcap, int back) {
    int w = blockIdx.y;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int R = d.R;
    if (r > R) return;
    const int n0 = d.nn0;
    const cd* D = Dv + (size_t)w * (n0 + 1) * 4;
    const size_t rows0 = psvk::fld_rows(NS0, d.Rs1, d.Rf), rows1 = psvk::fld_rows(NS1, d.Rs1, d.Rf),
                 rows2 = psvk::fld_rows(NS2, d.Rs1, d.Rf);
    T* A0w = A0f + (size_t)w * rows0 * Lcap;
    T* A1w = A1f + (size_t)w * rows1 * Lcap;
    T* A2w = A2f + (size_t)w * rows2 * Lcap;
    const int rr = d.rrow[r];
    for (int q = 0; q < NS0; ++q) {
        cd U = mk(0.0), Ud = mk(0.0);
        if (q < 3 || back) {
            if (r < R) {
                for (int i = 0; i < 3; ++i) {
                    cd v = D[4 * (d.jsta[r] + i) + q];
                    U = U + d.wv[3 * r + i] * v;
                    Ud = Ud + d.wd[3 * r + i] * v;
                }
            } else if (q < 3) {
                U = D[4 * n0 + q];
            }
        }
        put_field(A0w, Lcap, NS0, d, rr, q, 0, U);
        put_field(A0w, Lcap, NS0, d, rr, q, 1, Ud);
        for (int f = 2; f < NFLD; ++f) put_field(A0w, Lcap, NS0, d, rr, q, f, mk(0.0));
    }
    for (int q = 0; q < NS1; ++q)
        for (int f = 0; f < NFLD; ++f) put_field(A1w, Lcap, NS1, d, rr, q, f, mk(0.0));
    for (int q = 0; q < NS2; ++q)
        for (int f = 0; f < NFLD; ++f) put_field(A2w, Lcap, NS2, d, rr, q, f, mk(0.0));
}

// ------------------------------------------------------- source terms
__device__ void calabnum_dev(const PsvDev& d, double omega, cd coef1, cd coef2, cd* anum, cd* bnum) {
    for (int k = 0; k < 160; ++k) anum[k] = bnum[k] = mk(0.0);
    auto AN = [&](int i, int j, int k) -> cd& { return anum[(k - 1) * 16 + (j - 1) * 4 + (i - 1)]; };
    auto BN = [&](int i, int j, int k) -> cd& { return bnum[(k - 1) * 16 + (j - 1) * 4 + (i - 1)]; };
    const double* P = d.poly;
    for (int i = 1; i <= 10; ++i) {
        double r;
        if (i <= 5) r = d.ra0 + (double)(i - 1) / 4.0 * (d.r0 - d.ra0);
        else r = d.ra1 - (double)(10 - i) / 4.0 * (d.ra1 - d.r0);
        double trho = 0, tvpv = 0, tvph = 0, tvsv = 0, tvsh = 0, teta = 0, coef = 1.0;
        for (int j = 1; j <= 4; ++j) {
            if (j == 1) coef = 1.0;
            else coef = coef * (r / d.rmax);
            trho = trho + P[0 + j - 1] * coef;
            tvpv = tvpv + P[4 + j - 1] * coef;
            tvph = tvph + P[8 + j - 1] * coef;
            tvsv = tvsv + P[12 + j - 1] * coef;
            tvsh = tvsh + P[16 + j - 1] * coef;
            teta = teta + P[20 + j - 1] * coef;
        }
        double tecA = trho * tvph * tvph, tecC = trho * tvpv * tvpv;
        double tecL = trho * tvsv * tvsv, tecN = trho * tvsh * tvsh, tmu = trho * tvsv * tvsv;
        double tAkappa = tecA - tmu * 4.0 / 3.0, tCkappa = tecC - tmu * 4.0 / 3.0;
        cd xAkappa = mk(tAkappa) * coef2, xCkappa = mk(tCkappa) * coef2;
        cd xrho = mk(trho), xmu = mk(tmu) * coef1, xecL = mk(tecL) * coef1, xecN = mk(tecN) * coef1;
        cd xecA = xAkappa + xmu * mk(4.0 / 3.0);
        cd xecC = xCkappa + xmu * mk(4.0 / 3.0);
        cd xecF = mk(teta) * (xecA - mk(2.0) * xecL);
        cd xFdC = xecF / xecC;
        cd xAmF2dC = xecA - xecF * xFdC;
        double r2 = r * r;
        cd comega2 = mk(omega, -d.omegai) * mk(omega, -d.omegai);
        AN(1, 1, i) = -(mk(2.0 / r) * xFdC);
        AN(1, 2, i) = mk(1.0) / xecC;
        AN(2, 1, i) = -(xrho * comega2) + mk(4.0 / r2) * (xAmF2dC - xecN);
        AN(2, 2, i) = mk(2.0 / r) * (xFdC - mk(1.0));
        AN(3, 1, i) = -mk(1.0 / r);
        AN(3, 3, i) = mk(1.0 / r);
        AN(3, 4, i) = mk(1.0) / xecL;
        AN(4, 1, i) = -(mk(2.0 / r2) * (xAmF2dC - xecN));
        AN(4, 2, i) = -(mk(1.0 / r) * xFdC);
        AN(4, 3, i) = -(xrho * comega2) - mk(2.0 / r2) * xecN;
        AN(4, 4, i) = -mk(3.0 / r);
        BN(1, 3, i) = mk(1.0 / r) * xFdC;
        BN(2, 3, i) = -(mk(2.0 / r2) * (xAmF2dC - xecN));
        BN(2, 4, i) = mk(1.0 / r);
        BN(4, 3, i) = xAmF2dC / mk(r2);
    }
}

__device__ __forceinline__ void eqm(const cd* __restrict__ anum, const cd* __restrict__ bnum, int blk, double l2,
                                    const cd* y, cd* f) {
    const cd *an = anum + 16 * (blk - 1), *bn = bnum + 16 * (blk - 1);
    cd c[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const cd b = bn[k];
        c[k] = an[k] + mk(l2 * b.re, l2 * b.im);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[i] = mk(0.0);
#pragma unroll
        for (int j = 0; j < 4; ++j) f[i] = f[i] + c[4 * j + i] * y[j];
    }
}

// rk3 with one rkstep of h (src/SGTpsv/rk3.f90) over the blocks b0, b1, b2
__device__ __forceinline__ void rk1(const cd* __restrict__ anum, const cd* __restrict__ bnum, int b0, int b1, int b2,
                                    double l2, double h, cd* y0) {
    const double c1 = 1.0 / 6.0, c2 = 1.0 / 3.0, c3 = c2, c4 = c1, h2 = 0.5, h3 = h2;
    cd ak[4], yn[4], w[4];
    eqm(anum, bnum, b0, l2, y0, ak);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        yn[i] = y0[i] + mk(h * c1) * ak[i];
        w[i] = y0[i] + mk(h * h2) * ak[i];
    }
    eqm(anum, bnum, b1, l2, w, ak);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        yn[i] = yn[i] + mk(h * c2) * ak[i];
        w[i] = y0[i] + mk(h * h3) * ak[i];
    }
    eqm(anum, bnum, b1, l2, w, ak);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        yn[i] = yn[i] + mk(h * c3) * ak[i];
        w[i] = y0[i] + mk(h) * ak[i];
    }
    eqm(anum, bnum, b2, l2, w, ak);
#pragma unroll
    for (int i = 0; i < 4; ++i) y0[i] = yn[i] + mk(h * c4) * ak[i];
}

// column c of calya's ya, yb, yc, yd: ya and yb run from ra0 up to r0, yc and
// yd from ra1 down to it, in two steps each (yb's and yd's begin where the
// step before has ended, less its length)
__device__ __forceinline__ void calya_col(const cd* __restrict__ anum, const cd* __restrict__ bnum, double l2,
                                          double ra0, double ra1, double r0, int c, cd* y) {
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = mk(0.0);
    if (c & 1) y[3] = mk(1.0);
    else y[1] = mk(1.0);
    const bool up = c < 2;
    double xs = up ? ra0 : ra1;
    const double dr = (up ? r0 - ra0 : ra1 - r0) / 2.0;
    if (!(dr > 0.0)) return;
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        const double xe = up ? xs + dr : xs - dr;
        const double xb = (c & 1) ? (up ? xe - dr : xe + dr) : xs;
        if (up) rk1(anum, bnum, 2 * k + 1, 2 * k + 2, 2 * k + 3, l2, xe - xb, y);
        else rk1(anum, bnum, 10 - 2 * k, 9 - 2 * k, 8 - 2 * k, l2, xe - xb, y);
        xs = xe;
    }
}

// glu (src/SGTpsv/glu2.f90): factors of an N x N complex matrix, leading
// dimension 4, and pivots; false where a pivot is too small (the right-hand
// sides then stay as they are)
template <int N>
__device__ __forceinline__ bool glu_factor(cd* a, int* ip) {
    const double eps = 3.52e-15;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double amax = cabs_(a[5 * k]);
        int ipk = k;
#pragma unroll
        for (int i = k + 1; i < N; ++i) {
            const double aik = cabs_(a[i + 4 * k]);
            if (aik > amax) { ipk = i; amax = aik; }
        }
        ip[k] = ipk;
        if (!(amax > eps)) return false;
#pragma unroll
        for (int i = k + 1; i < N; ++i)
            if (ipk == i) {
#pragma unroll
                for (int j = k; j < N; ++j) {
                    const cd t = a[i + 4 * j];
                    a[i + 4 * j] = a[k + 4 * j];
                    a[k + 4 * j] = t;
                }
            }
#pragma unroll
        for (int i = k + 1; i < N; ++i) a[i + 4 * k] = -a[i + 4 * k] / a[5 * k];
#pragma unroll
        for (int j = k + 1; j < N; ++j)
#pragma unroll
            for (int i = k + 1; i < N; ++i) a[i + 4 * j] = a[i + 4 * j] + a[i + 4 * k] * a[k + 4 * j];
    }
    return true;
}

template <int N>
__device__ __forceinline__ void glu_solve(const cd* a, const int* ip, cd* b) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int ipk = ip[k];
#pragma unroll
        for (int i = k + 1; i < N; ++i)
            if (ipk == i) {
                const cd t = b[i];
                b[i] = b[k];
                b[k] = t;
            }
#pragma unroll
        for (int i = k + 1; i < N; ++i) b[i] = b[i] + a[i + 4 * k] * b[k];
    }
    b[N - 1] = b[N - 1] / a[5 * (N - 1)];
#pragma unroll
    for (int k = N - 2; k >= 0; --k) {
#pragma unroll
        for (int i = 0; i <= k; ++i) b[i] = b[i] - a[i + 4 * (k + 1)] * b[k + 1];
        b[k] = b[k] / a[5 * k];
    }
}

// calg (calmat.f90:1075-1171): the discontinuities of the unit moment tensor
// imt across the source
__device__ __forceinline__ void calg_rhs(const PsvDev& d, int l, int m, cd coef1, cd coef2, double lsq, int imt,
                                         cd* sv) {
    double mt11 = imt == 1, mt22 = imt == 2, mt33 = imt == 3, mt12 = imt == 4, mt13 = imt == 5,
           mt23 = imt == 6;
    double sgn = (m >= 0) ? 1.0 : -1.0;
    double b1 = sqrt((double)(2 * l + 1) / (16.0 * kPi));
    double b2 = 0.0;
    if (l != 0) b2 = sqrt((double)(2 * l + 1) * (double)(l - 1) * (double)(l + 2) / (64.0 * kPi));
    const double r0 = d.r0, ecC0 = d.ecC0, ecF0 = d.ecF0, ecL0 = d.ecL0;
    cd dd = mk(0.0), ee = mk(0.0), s1 = mk(0.0), s2 = mk(0.0);
    int am = abs(m);
    if (am == 1) ee = mk(-b1 * sgn * mt12, b1 * mt13) / (mk(r0 * r0 * ecL0) * coef1);
    if (am == 0) {
        dd = mk(2.0 * b1 * mt11 / (r0 * r0)) /
             (mk(ecC0 - 4.0 / 3.0 * ecL0) * coef2 + mk(4.0 / 3.0 * ecL0) * coef1);
        double r03 = r0 * r0 * r0;
        cd xtmp = ((ecF0 + 2.0 / 3.0 * ecL0) * coef2 - 2.0 / 3.0 * ecL0 * coef1) /
                  ((ecC0 - 4.0 / 3.0 * ecL0) * coef2 + 4.0 / 3.0 * ecL0 * coef1);
        s1 = mk(-2.0 * b1 * (mt22 + mt33) / r03) + mk(4.0 * b1 * mt11 / r03) * xtmp;
        s2 = mk(b1 * lsq * (mt22 + mt33) / r03) - mk(2.0 * b1 * lsq * mt11 / r03) * xtmp;
    }
    if (am == 2) {
        double r03 = r0 * r0 * r0;
        s2 = mk(-b2 * (mt22 - mt33) / r03, sgn * 2.0 * b2 * mt23 / r03);
    }
    sv[0] = dd;
    sv[1] = s1;
    if (l != 0) {
        sv[2] = mk(ee.re / lsq, ee.im / lsq);
        sv[3] = mk(s2.re / lsq, s2.im / lsq);
    } else {
        sv[2] = sv[3] = mk(0.0);
    }
}

// the amplitudes of the source element's rows
__device__ __forceinline__ void calg_rows(const PsvDev& d, double lsq, const cd* b, cd* g) {
    double dt[4];
    dt[0] = -d.ra0 * d.ra0;
    dt[1] = dt[0] * lsq;
    dt[2] = d.ra1 * d.ra1;
    dt[3] = dt[2] * lsq;
#pragma unroll
    for (int i = 0; i < 4; ++i) g[i] = mk(b[i].re * dt[i], b[i].im * dt[i]);
}

// calg at l = 0 for imt 1..3, [imt - 1][row]
__device__ void calg_l0(const PsvDev& d, cd coef1, cd coef2, const cd* ab, cd* g) {
    cd a[16], y[4];
    int ip[2];
    calya_col(ab, ab + 160, 0.0, d.ra0, d.ra1, d.r0, 0, y);
    for (int i = 0; i < 2; ++i) a[i] = -y[i];
    calya_col(ab, ab + 160, 0.0, d.ra0, d.ra1, d.r0, 2, y);
    for (int i = 0; i < 2; ++i) a[i + 4] = y[i];
    const bool ok = glu_factor<2>(a, ip);
    for (int imt = 1; imt <= 3; ++imt) {
        cd b[4];
        calg_rhs(d, 0, 0, coef1, coef2, 0.0, imt, b);
        if (ok) glu_solve<2>(a, ip, b);
        b[2] = b[1];
        b[1] = b[3] = mk(0.0);
        calg_rows(d, 0.0, b, g + 4 * (imt - 1));
    }
}

// ----------------------------------------------------------------- fields
// Flat slot order (18 slots): 0..2 m = 0, imt 1..3; 3 m = 0 back-propagated
// vertical force; 4..11 |m| = 1: 4 + 4 sg + k (k: imt 4, imt 5, back 2,
// back 3; sg 0: m = -1, 1: m = +1); 12..17 |m| = 2: 12 + 3 sg + k (imt 2, 3, 6).
constexpr int NSLOT = 18;

__device__ __forceinline__ int slot_mi(int s) { return s < 4 ? 0 : (s < 12 ? 1 : 2); }
__device__ __forceinline__ int slot_q(int s) { return s < 4 ? s : (s < 12 ? s - 4 : s - 12); }

// back-propagated slots; a slot combines the basis solutions [b0, b1): the
// forward ones those of the source's four rows, the back ones the one of the
// surface row their force acts on
__device__ __forceinline__ constexpr bool slot_back(int s) { return s == 3 || (s >= 4 && s < 12 && (s - 4) % 4 >= 2); }
__device__ __forceinline__ constexpr int slot_b0(int s) { return !slot_back(s) ? 0 : (s == 3 ? 4 : 5); }
__device__ __forceinline__ constexpr int slot_b1(int s) { return !slot_back(s) ? 4 : (s == 3 ? 5 : 6); }

// calabnum of every frequency (once per omega)
__global__ void k_psv_abnum(PsvDev d, const int* __restrict__ freqs, int nf, cd* __restrict__ ab) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nf) return;
    const double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
    cd c1 = coefq(omega, d.qmu[d.spn - 1]), c2 = coefq(omega, d.qkappa[d.spn - 1]);
    calabnum_dev(d, omega, c1, c2, ab + (size_t)w * 320, ab + (size_t)w * 320 + 160);
}

// Per (omega, l >= 1): weights of the six basis solutions for every slot
// (calya + calg for the 13 forward sources, caldveczero for the back ones).
// Layout co[(slot * NB + b) * nsys + sys].
// The cutoff probe of the system (calamp on
// g0(ksta(r_n)-1), g0(ksta(r_n)) of imt = 1, m = 0) is formed here from the
// FP64 slot-0 coefficients and the FP64 probe captures, in every mode.
//
// Bound: one system's chain of Runge-Kutta steps, pivots and divisions.  With
// a thread per system, which factored the same 4 x 4 matrix for each of the 13
// sources, it took 0.128 ms for 1248 systems (10 blocks) and 0.154 for 12 000.
// Eight threads now share a system: the matrix's four columns in four of them,
// its factors once, then two sources each (COEF_SLOTS, with the back slots,
// which need no solve, on the threads that have one): 0.025 and 0.075 ms.
constexpr int COEF_S = 16, COEF_R = 8;  // systems of a block, threads of a system
__constant__ const unsigned COEF_SLOTS[COEF_R] = {1u << 0 | 1u << 13, 1u << 1 | 1u << 14, 1u << 2 | 1u << 15,
                                                  1u << 4 | 1u << 16, 1u << 5 | 1u << 17, 1u << 8 | 1u << 3,
                                                  1u << 9 | 1u << 6 | 1u << 7, 1u << 12 | 1u << 10 | 1u << 11};

__global__ void __launch_bounds__(COEF_S * COEF_R)
    k_psv_coef(PsvDev d, const int* __restrict__ freqs, WorkList wl, int nsys, const cd* __restrict__ ab,
               cd* __restrict__ co, int back, const cd* __restrict__ Xprobe, double* __restrict__ amps, int Lcap) {
    __shared__ cd lu[COEF_S][17];  // -ya, -yb, yc, yd by columns, then their factors
    __shared__ int ip[COEF_S][4], ok[COEF_S];
    const int sl = threadIdx.x % COEF_S, role = threadIdx.x / COEF_S;
    const int sys = blockIdx.x * COEF_S + sl;
    const bool in = sys < nsys;
    int w = 0, l = 0;
    if (in) wl_map(wl, sys, w, l);
    const double l2 = (double)l * (double)(l + 1), lsq = sqrt(l2);
    if (l > 0 && role < 4) {
        const cd* anum = ab + (size_t)w * 320;
        cd y[4];
        calya_col(anum, anum + 160, l2, d.ra0, d.ra1, d.r0, role, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) lu[sl][4 * role + i] = role < 2 ? -y[i] : y[i];
    }
    __syncthreads();
    if (l > 0 && role == 0) {
        cd a[16];
        int p[4] = {0, 1, 2, 3};
#pragma unroll
        for (int i = 0; i < 16; ++i) a[i] = lu[sl][i];
        ok[sl] = glu_factor<4>(a, p);
#pragma unroll
        for (int i = 0; i < 16; ++i) lu[sl][i] = a[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) ip[sl][i] = p[i];
    }
    __syncthreads();
    if (!in) return;
    const double omega = 2.0 * kPi * (double)freqs[w] / d.tlen;
    const cd c1 = coefq(omega, d.qmu[d.spn - 1]), c2 = coefq(omega, d.qkappa[d.spn - 1]);
    for (unsigned todo = COEF_SLOTS[role]; todo; todo &= todo - 1) {
        const int s = __ffs(todo) - 1, mi = slot_mi(s), q = slot_q(s);
        cd g[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) g[b] = mk(0.0);
        // order 0: its own kernels write this order's fields and probe
        int m = 0, imt = 0;
        if (mi == 0) {
            imt = q < 3 ? q + 1 : 0;
        } else if (mi == 1) {
            m = q / 4 == 0 ? -1 : 1;
            imt = q % 4 < 2 ? 4 + q % 4 : 0;
        } else if (l >= 2) {
            m = q / 3 == 0 ? -2 : 2;
            imt = q % 3 == 0 ? 2 : (q % 3 == 1 ? 3 : 6);
        }
        if (l > 0 && imt > 0) {
            cd b[4];
            calg_rhs(d, l, m, c1, c2, lsq, imt, b);
            if (ok[sl]) glu_solve<4>(lu[sl], ip[sl], b);
            calg_rows(d, lsq, b, g);
        } else if (l > 0 && back && mi == 0) {
            double coef = sqrt((double)(2 * l + 1) / (4.0 * kPi) / 1.0);
            g[4] = -conj(mk((double)(float)coef));  // g0(nn-1) = -conjg(rdvec(1,0))
        } else if (l > 0 && back && mi == 1) {
            // caldveczero, m = 1: bvec(2,1) = -xl2 coef/2, bvec(3,1) = i xl2 coef/2;
            // m = -1: conjugated and negated (odd m).  g0(nn) = conjg(rdvec)/lsq
            double fact = (double)l * (double)(l + 1);
            double coef = sqrt((double)(2 * l + 1) / (4.0 * kPi) / fact);
            cd v = (q % 4 == 2) ? mk(-1.0, 0.0) * l2 * coef / 2.0 : mk(0.0, 1.0) * l2 * coef / 2.0;
            if (m < 0) v = -conj(v);
            g[5] = conj(v) / mk(lsq);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
            if (b >= slot_b0(s) && b < slot_b1(s)) co[((size_t)s * NB + b) * nsys + sys] = g[b];
        if (s == 0 && l > 0) {
            cd p0 = mk(0.0), p1 = mk(0.0);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                p0 = p0 + g[b] * Xprobe[(size_t)b * nsys + sys];
                p1 = p1 + g[b] * Xprobe[(size_t)(4 + b) * nsys + sys];
            }
            const double a1 = cabs_(p0), a2 = cabs_(p1);
            amps[(size_t)w * Lcap + l] = sqrt(a1 * a1 + a2 * a2);
        }
    }
}

// Fields of every slot at the receivers, one thread per (system, receiver):
// a warp holds FS consecutive systems (orders) x 32/FS receivers, so
// each coefficient load serves 32/FS receivers and each field store writes
// FS consecutive orders of one row (32 x 1 measured fastest of 4 x 8,
// 8 x 4, 16 x 2 and 32 x 1 on the benchmark; the results do not depend on
// it).  Values and radial derivatives of the six
// basis solutions come from the three-node weights (interpolate, calup),
// then U, V and derivatives of each slot are their combinations with the
// source coefficients.  The last block row holds the surface (rows n-1, n).
// FS systems x 32/FS receivers per warp: 32 (default) or 16, chosen per
// context (dsm_set_tuning / dsm_autotune)


// Arithmetic of the field kernel: the reference's operations on the plain
// path, fused multiply-adds and one reciprocal of sqrt(l(l+1)) on the mixed
// path (whose rows are stored in FP32), both in FP64.  Measured on the
// 2048-frequency grid, FP32 slot combinations (FP64 interpolation) raised the
// mixed path's error to 9e-7 and FP32 interpolation to 5e-6: the derivative
// weights difference neighbouring nodes and the bases cancel.
template <bool FAST>
struct FieldMath {
    using V = cd;
    using R = double;
    __device__ static V coef(const cd* p, size_t i) { return p[i]; }
    __device__ static V from(cd v) { return v; }
    __device__ static V zero() { return mk(0.0); }
    __device__ static cd interp(cd acc, double r, cd x) {  // acc + r x
        if (FAST) return mk(fma(r, x.re, acc.re), fma(r, x.im, acc.im));
        return acc + r * x;
    }
    __device__ static V addmul(V acc, V a, V b) { return caddmulT<FAST>(acc, a, b); }  // acc + a b
    __device__ static V divl(V v, R lsq, R ilsq) { return FAST ? v * ilsq : v / lsq; }
};
template <class T, class V>
__device__ __forceinline__ void put_fieldv(T* Aw, int Lcap, int nq, const PsvDev& d, int rr, int q, int f, V v) {
    int im;
    const long long row = psvk::fld_row(nq, d.Rs1, d.Rf, q, f, rr, &im);
    if (row < 0) return;
    Aw[(size_t)row * Lcap] = (T)v.re;
    Aw[((size_t)row + im) * Lcap] = (T)v.im;
}

// Field rows of every (order, receiver): 3-node interpolation of the
// captured solutions (value and radial derivative), combined with the
// source coefficients of each slot (calup*, locallyCartesianDerivatives
// inputs); fluid receivers store U only.  The cutoff probe is formed by
// k_psv_coef.
//
// Bound: latency at three blocks of 158-170 registers per SM, then the rows
// written.  A slot combines the four (forward) or one (back) basis solutions
// it has weights for, not all six with zeros, in fully unrolled slots: 16 400
// orders, FP32 rows 0.88 -> 0.74 ms, 8100 orders, FP64 rows 0.86 -> 0.69 ms.
// Two blocks per SM took 0.78 and 0.82, four 0.72 and 0.73, five 0.82 and 0.76.
template <bool MIXED, int FS>
__global__ void __launch_bounds__(128, 3) k_psv_fields(PsvDev d, WorkList wl, int nsys,
                                                    const cd* __restrict__ Xcap, const cd* __restrict__ co,
                                                    typename std::conditional<MIXED, float, double>::type* __restrict__ A0f,
                                                    typename std::conditional<MIXED, float, double>::type* __restrict__ A1f,
                                                    typename std::conditional<MIXED, float, double>::type* __restrict__ A2f,
                                                    int Lcap, const int* __restrict__ kcut, int* __restrict__ zfirst) {
    using T = typename std::conditional<MIXED, float, double>::type;
    using FM = FieldMath<MIXED>;
    using V = typename FM::V;
    using RT = typename FM::R;
    // the four warps of a block take the same FS orders at 4 x 32/FS
    // neighbouring receivers: the coefficient and capture loads of the
    // orders are shared through L1
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sys = blockIdx.x * FS + lane % FS;
    const int r = (blockIdx.y * 4 + warp) * (32 / FS) + lane / FS;
    const int R = d.R;
    if (sys >= nsys || r > R) return;
    int w, l;
    wl_map(wl, sys, w, l);
    if (l == 0) return;  // written by the order-0 kernels
    const size_t rows[3] = {psvk::fld_rows(NS0, d.Rs1, d.Rf), psvk::fld_rows(NS1, d.Rs1, d.Rf),
                            psvk::fld_rows(NS2, d.Rs1, d.Rf)};
    const int rr = d.rrow[r];
    T* Aw[3] = {A0f + (size_t)w * rows[0] * Lcap + l, A1f + (size_t)w * rows[1] * Lcap + l,
                A2f + (size_t)w * rows[2] * Lcap + l};
    const double l2d = (double)l * (double)(l + 1), lsqd = sqrt(l2d);
    const RT l2 = (RT)l2d, lsq = (RT)lsqd, ilsq = (RT)(1.0 / lsqd);
    auto X = [&](int cap, int b) { return Xcap[((size_t)cap * NB + b) * nsys + sys]; };
    auto C = [&](int s, int b) { return FM::coef(co, ((size_t)s * NB + b) * nsys + sys); };
    // With the depth cut-off, a receiver whose stencil lies below the
    // system's cut row (the same for the warp's 32 orders: a factorisation
    // warp) has zero captures, so every field is zero: written without the
    // loads of the coefficients and captures.
    if (kcut && r < R && d.stop_row[r] < kcut[sys]) {
        // the cut row grows with the order, so this receiver's fields are
        // zero from here on: its lowest order in the warp records that
        if (zfirst && lane % FS == 0) atomicMin(zfirst + (size_t)w * (R + 1) + r, l);
        for (int s = 0; s < NSLOT; ++s) {
            const int mi = slot_mi(s), q = slot_q(s), nqm = mi == 0 ? NS0 : (mi == 1 ? NS1 : NS2);
            const V z = FM::zero();
            if (rr < 0) {
                put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 0, z);
                continue;
            }
            for (int f = 0; f < 5; ++f) put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, f, z);
        }
        return;
    }
    if (rr < 0) {  // fluid receiver: only U is stored
        V bU[NB];
        for (int b = 0; b < NB; ++b) {
            cd u = mk(0.0);
            for (int i = 0; i < 3; ++i) u = FM::interp(u, d.wv[3 * r + i], X(d.rcap[6 * r + 2 * i], b));
            bU[b] = FM::from(u);
        }
#pragma unroll
        for (int s = 0; s < NSLOT; ++s) {
            const int mi = slot_mi(s), q = slot_q(s);
            V U = FM::zero();
#pragma unroll
            for (int b = slot_b0(s); b < slot_b1(s); ++b) U = FM::addmul(U, C(s, b), bU[b]);
            put_fieldv<T>(Aw[mi], Lcap, mi == 0 ? NS0 : (mi == 1 ? NS1 : NS2), d, rr, q, 0, U);
        }
        return;
    }
    const bool surf = r == R;
    V bU[NB], bV[NB], bUd[NB], bVd[NB];
    for (int b = 0; b < NB; ++b) {
        cd u = mk(0.0), v = mk(0.0), ud = mk(0.0), vd = mk(0.0);
        if (surf) {
            u = X(d.cap_n1, b);
            v = X(d.cap_n, b);
        } else {
            for (int i = 0; i < 3; ++i) {
                const double wvi = d.wv[3 * r + i], wdi = d.wd[3 * r + i];
                const cd xu = X(d.rcap[6 * r + 2 * i], b), xv = X(d.rcap[6 * r + 2 * i + 1], b);
                u = FM::interp(u, wvi, xu);
                v = FM::interp(v, wvi, xv);
                ud = FM::interp(ud, wdi, xu);
                vd = FM::interp(vd, wdi, xv);
            }
        }
        bU[b] = FM::from(u);
        bV[b] = FM::from(v);
        bUd[b] = FM::from(ud);
        bVd[b] = FM::from(vd);
    }
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
        const int mi = slot_mi(s), q = slot_q(s);
        V U = FM::zero(), Vv = FM::zero(), Ud = FM::zero(), Vd = FM::zero();
        if (!(surf && slot_back(s))) {
#pragma unroll
            for (int b = slot_b0(s); b < slot_b1(s); ++b) {
                const V cb = C(s, b);
                U = FM::addmul(U, cb, bU[b]);
                Vv = FM::addmul(Vv, cb, bV[b]);
                Ud = FM::addmul(Ud, cb, bUd[b]);
                Vd = FM::addmul(Vd, cb, bVd[b]);
            }
        }
        const V Vh = FM::divl(Vv, lsq, ilsq), Vdh = FM::divl(Vd, lsq, ilsq);
        const int nqm = mi == 0 ? NS0 : (mi == 1 ? NS1 : NS2);
        put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 0, U);
        put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 1, Ud);
        put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 2, Vh);
        put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 3, Vdh);
        put_fieldv<T>(Aw[mi], Lcap, nqm, d, rr, q, 4, l2 * Vh);
    }
}

// The cutoff test of one frequency is a sequential state machine over
// (l, m); here one warp runs it 256 orders at a time with the same results.
// Per order l >= 1 the updates are m = -2 (l >= 2), -1, 0, 1, 2 (l >= 2);
// only m = 0 has a nonzero amplitude, so
//   maxamp at the m = 0 update = max(carry, 0, amplitudes of orders <= l),
//   ismall after l = 0 when l < lsuf, else ismall + nm (m = 0 small) or the
//   count of updates after m = 0 (not small),
// a prefix maximum and a prefix composition of v -> a v + b (a in {0, 1}),
// both exact.  The exit fires at the first order whose incoming ismall
// exceeds 20.  A lane takes SCAN_K consecutive orders: their loads and ratios
// are independent, and the scans over the warp come once for 256 orders (with
// one order a lane, the 61 dependent steps of 1950 orders took 0.113 ms, now
// 0.035).
__device__ __forceinline__ double warp_prefix_max(double x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = fmax(x, y);
    }
    return x;
}
__global__ void k_psv_scan(int nf, WorkList wl, int Lcap, int maxlmax, double ratl, double tlen,
                           double vtop, double rtop, const int* __restrict__ freqs,
                           const double* __restrict__ amps, CutState* __restrict__ cut,
                           int* __restrict__ status) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= nf) return;
    CutState c = cut[w];
    if (c.done) return;
    const double omega = 2.0 * kPi * (double)freqs[w] / tlen;
    const int lsuf = (int)(omega * rtop / vtop - 0.5) + 1;
    const int l0 = wl.lb[w], l1 = l0 + wl.off[w + 1] - wl.off[w];
    double mx = c.maxamp;
    int v = c.ismall;
    for (int base = l0; base < l1; base += 32 * SCAN_K) {
        const int lf = base + lane * SCAN_K;
        double amp[SCAN_K];
        int badpos = INT_MAX;
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j)
            amp[j] = lf + j < l1 && lf + j >= 1 ? amps[(size_t)w * Lcap + lf + j] : 0.0;
        double pm = -1.0;
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            if (!isfinite(amp[j])) {
                badpos = min(badpos, lf + j);
                amp[j] = 0.0;
            }
            if (lf + j < l1 && lf + j >= 1) pm = fmax(pm, amp[j]);
        }
        badpos = __reduce_min_sync(0xffffffffu, badpos);
        pm = warp_prefix_max(pm, lane);
        double run = __shfl_up_sync(0xffffffffu, pm, 1);  // maximum of the orders before this lane's
        if (lane == 0) run = -1.0;
        const double run0 = run;
        int ra[SCAN_K], rb[SCAN_K], A = 1, B = 0;  // each order's map v -> ra v + rb, and the lane's
#pragma unroll
        for (int j = 0; j < SCAN_K; ++j) {
            const int l = lf + j;
            ra[j] = 1;
            rb[j] = 0;
            if (l < l1 && l >= 1) {
                // maxamp at this order's m = 0 update (the m = -1 update contributes 0)
                run = fmax(run, amp[j]);
                const double mxl = fmax(fmax(mx, run), 0.0);
                double ratio = 0.0;
                if (amp[j] != 0.0 && mxl != 0.0) ratio = amp[j] / mxl;
                const int nm = l >= 2 ? 5 : 3, after = l >= 2 ? 2 : 1;
                if (l < lsuf) ra[j] = 0;
                else if (ratio < ratl) rb[j] = nm;
                else { ra[j] = 0; rb[j] = after; }
            }
            B = ra[j] * B + rb[j];
            A = ra[j] * A;
        }
        // inclusive composition over lanes <= this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int pa = __shfl_up_sync(0xffffffffu, A, o), pb = __shfl_up_sync(0xffffffffu, B, o);
            if (lane >= o) { B = A * pb + B; A = A * pa; }
        }
        const int vafter = A * v + B;
        int vb = __shfl_up_sync(0xffffffffu, vafter, 1);
        if (lane == 0) vb = v;
        // the first order the counter has passed 20 before; the maximum then
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
            if (l < l1 && l >= 1) run = fmax(run, amp[j]);
        }
        const unsigned ex = __ballot_sync(0xffffffffu, hit != INT_MAX);
        const int e = ex ? __ffs(ex) - 1 : 0, le = __shfl_sync(0xffffffffu, hit, e);
        // an Inf/NaN probe means the solves broke down: stop this frequency
        // and report it (llog -1 marks it) instead of running to maxlmax;
        // orders are looked at in steps of 32, past the step of the cutoff
        // none is
        if (badpos != INT_MAX && (!ex || (badpos - l0) / 32 <= (le - l0) / 32)) {
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
            double me = fmax(mx, __shfl_sync(0xffffffffu, mhit, e));
            if (le > base && le - 1 >= 1) me = fmax(me, 0.0);
            c.ismall = __shfl_sync(0xffffffffu, vhit, e);
            if (c.llog > le) c.llog = le;
            c.done = 1;
            c.norders = le;
            c.maxamp = me;
            if (lane == 0) cut[w] = c;
            return;
        }
        // carry past these orders
        mx = fmax(mx, __shfl_sync(0xffffffffu, pm, 31));
        if (min(l1, base + 32 * SCAN_K) > 1) mx = fmax(mx, 0.0);
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

// Depth cut-off of an (omega, l) system.  Below the turning depth of the
// slowest wave the displacement decays like exp(-E(r)),
//   E(r) = int_r^{r_s} kappa dr',  kappa^2 = ((l + 1/2) / r')^2 - (omega / v(r'))^2,
// counting only the evanescent parts (kappa^2 > 0); v is the SV speed in
// solid zones, and fluid zones count as never evanescent (kappa = 0), which
// only keeps more rows.  Starting at the deepest source r_s, the first node
// where E reaches X bounds the amplitude there by exp(-X) of the source's,
// and a zero-displacement boundary there perturbs what reaches the source
// and receivers above by about exp(-2X).  FP32 (a bound, not a result);
// nodes: x = r, y = 1 / v^2 (huge in fluid), z = local row of the node's
// first unknown.  kcut = that row less a margin of four, at most kmax
// (below the source rows).
// kappa grows with l at every node, and so does E: a frequency's lowest
// order in a warp has the lowest cut row of its orders there.  The warp
// computes the cut rows of those systems only (one per frequency it holds),
// each walk spread over the lanes: lane j takes the interval below node
// base - j, a prefix sum over the lanes gives E at each of the 32 nodes, and
// the first lane where E reaches X ends the walk.  Every lane takes the
// warp's lowest cut row, where the factorisation of its 32 systems starts
// anyway: lanes above it keep a few more rows than their own bound needs.
// Bound: a warp's chain of passes (five shuffle steps of a sum each), 512
// warps for 16 400 systems: 0.17 ms one pass at a time, 0.11 four side by side.
constexpr int CUT_P = 4;
__global__ void k_psv_cutrow(const float4* __restrict__ nodes, int ks, float X, double tlen,
                             const int* __restrict__ freqs, WorkList wl, int nsys, int kmax, int* __restrict__ kcut) {
    const int sysv = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const bool valid = sysv < nsys;
    const int sys = valid ? sysv : nsys - 1;
    int w, l;
    wl_map(wl, sys, w, l);
    const int wprev = __shfl_up_sync(0xffffffffu, w, 1);
    unsigned lead = __ballot_sync(0xffffffffu, valid && (lane == 0 || wprev != w));
    int kc = INT_MAX;
    while (lead) {
        const int src = __ffs(lead) - 1;
        lead &= lead - 1;
        const int ws = __shfl_sync(0xffffffffu, w, src), ls = __shfl_sync(0xffffffffu, l, src);
        const float om = (float)(2.0 * kPi * (double)freqs[ws] / tlen);
        const float lam2 = ((float)ls + 0.5f) * ((float)ls + 0.5f), om2 = om * om;
        auto kappa = [&](float4 v) { return sqrtf(fmaxf(0.0f, lam2 / (v.x * v.x) - om2 * v.y)); };
        float E = 0.0f;
        int row = 1;
        // CUT_P passes of 32 intervals at a time: their nodes, square roots
        // and sums over the lanes are independent, E is carried through them
        // in order.  Node k - 1 of a lane's interval is the next lane's node,
        // or for lane 31 lane 0's of the next pass.
        float4 an[CUT_P + 1];
#pragma unroll
        for (int p = 0; p <= CUT_P; ++p) an[p] = nodes[max(ks - 32 * p - lane, 0)];
        bool found = false;
        for (int base = ks; base >= 1 && !found; base -= 32 * CUT_P) {
            float inc[CUT_P], bz[CUT_P], ka[CUT_P + 1];
            float4 a[CUT_P + 1];
#pragma unroll
            for (int p = 0; p <= CUT_P; ++p) {
                a[p] = an[p];
                an[p] = nodes[max(base - 32 * (CUT_P + p) - lane, 0)];
                ka[p] = kappa(a[p]);
            }
#pragma unroll
            for (int p = 0; p < CUT_P; ++p) {
                float bx = __shfl_down_sync(0xffffffffu, a[p].x, 1), kb = __shfl_down_sync(0xffffffffu, ka[p], 1);
                bz[p] = __shfl_down_sync(0xffffffffu, a[p].z, 1);
                const float nx = __shfl_sync(0xffffffffu, a[p + 1].x, 0), nz = __shfl_sync(0xffffffffu, a[p + 1].z, 0),
                            nk = __shfl_sync(0xffffffffu, ka[p + 1], 0);
                if (lane == 31) {
                    bx = nx;
                    bz[p] = nz;
                    kb = nk;
                }
                inc[p] = base - 32 * p - lane >= 1 ? 0.5f * (ka[p] + kb) * (a[p].x - bx) : 0.0f;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int p = 0; p < CUT_P; ++p) {
                    const float t = __shfl_up_sync(0xffffffffu, inc[p], o);
                    if (lane >= o) inc[p] += t;
                }
#pragma unroll
            for (int p = 0; p < CUT_P; ++p) {
                const unsigned hit = __ballot_sync(0xffffffffu, base - 32 * p - lane >= 1 && E + inc[p] >= X);
                if (hit && !found) {
                    row = (int)__shfl_sync(0xffffffffu, bz[p], __ffs(hit) - 1);
                    found = true;
                }
                E += __shfl_sync(0xffffffffu, inc[p], 31);
            }
        }
        kc = min(kc, max(1, min(row - 4, kmax)));
    }
    if (!valid) return;
    kcut[sys] = kc;
}

// ---------------------------------------------------------------- engine
class PsvEngine : public Engine {
  public:
    PsvDev d{};
    DBuf<int> iphase, nlayer, kkdr, elem, hmoff, blkoff, amz, amc, bcrow, rcap, stoprow, fluid, rrow, comp_src, jsta,
        l0col, l0e1;
    DBuf<double> qmu, qkappa, sel, fel, hm, bcval, poly, lam, qkp, fr, r, rrsta;
    DBuf<cd> B0, B1, B2, Xcap, Xprobe, l0scr, l0d, ab, co;
    DBuf<int4> rowasm;
    int ncap = 0;
    // depth cut-off: nodes (radius, 1/v^2, local row) from the centre up,
    // the node at the deepest source, the first kept row per system
    DBuf<float4> cnodes;
    std::vector<float4> hnodes;
    int cnode_src = 0;
    DBuf<int> kcut;
    // the stream of the systems' bottom segments
    cudaStream_t st3 = nullptr;
    cudaEvent_t ev_s3a = nullptr, ev_s3b = nullptr;
    // several sources: the segments around up to MAX_SRC_FAC of them are
    // factored at once, each in its own part of the records
    static constexpr int MAX_SRC_FAC = 4;
    int nfac = 1;                    // sources factored at once
    int nctop = 0, ngtop = 0;        // captured rows and gaps from the lowest last separator on
    cudaStream_t sfac[MAX_SRC_FAC - 1] = {};
    cudaEvent_t ev_fac[MAX_SRC_FAC] = {};
    // one parameter set per source depth (the source fields differ), and
    // the source polynomials they point to
    std::vector<PsvDev> dsrc;
    DBuf<double> polys;
    int ls_min = 1;  // local first source row of the deepest source
    // segmented band solve (psv_seg.cu): row pieces, captured rows in
    // ascending order, records, and one plan per source
    int ngap = 0, nsep_max = 0;
    int row_p0 = 0, row_p1 = 0;      // local rows of the cutoff probe
    DBuf<cd> P8, Lrec, Grec, Send, Xif;
    DBuf<int> caprow, capslot, gapidx;
    std::vector<psvseg::Plan> plans;
    // source s's slot of the field matrices (element type T)
    template <class T>
    T* afld_of(int m, int s) {
        return reinterpret_cast<T*>(reinterpret_cast<char*>(Afld[m].p) +
                                    (size_t)s * F * rows_m[m] * Lcap * afld_bytes);
    }
    double vtop = 0, rtop = 0;

    PsvEngine(const dsm_psv_setup_t* const* ss, int ns, const dsm_options_t* o) {
        if (!ss || ns < 1 || !ss[0]) throw Error(DSM_ERR_INVALID, "no PSV set-up");
        const dsm_psv_setup_t* s = ss[0];
        for (int k = 1; k < ns; ++k) check_same_grid(s, ss[k]);
        nsrc = ns;
        mode = 1;
        opt = *o;
        init_common(opt.device);
        {  // the stream of the systems' bottom segments: its blocks go first when SMs free up
            int lo = 0, hi = 0;
            DSM_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
            DSM_CUDA(cudaStreamCreateWithPriority(&st3, cudaStreamNonBlocking, hi));
            DSM_CUDA(cudaEventCreateWithFlags(&ev_s3a, cudaEventDisableTiming));
            DSM_CUDA(cudaEventCreateWithFlags(&ev_s3b, cudaEventDisableTiming));
            nfac = std::min(nsrc, MAX_SRC_FAC);
            for (int k = 0; k + 1 < nfac; ++k) DSM_CUDA(cudaStreamCreateWithFlags(&sfac[k], cudaStreamNonBlocking));
            for (int k = 0; k < nfac; ++k) DSM_CUDA(cudaEventCreateWithFlags(&ev_fac[k], cudaEventDisableTiming));
        }
        // the mixed path splits the fields into 11-bit pieces: FP32 storage
        // (24 bits) loses nothing it keeps and halves their traffic
        afld_bytes = mixed() ? 4 : 8;
        DSM_CUDA(cudaFuncSetAttribute(k_psv_l0_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L0_SMEM));
        m_lo = 0;
        R = s->r_n;
        Th = s->theta_n;
        num_t = DSM_PSV_NUM_TSGT; num_r = DSM_PSV_NUM_RSGT; num_s = DSM_PSV_NUM_SYNN;
        tlen = s->tlen; omegai = s->omegai; ratl = s->ratl; maxlmax = s->maxlmax;
        imin = s->imin; imax = s->imax;
        rsgt_sw = s->rsgt_switch == 1;
        synn_sw = s->synn_switch == 1;
        const int nz = s->nzone, nn = s->nn;
        if (R <= 0 || Th <= 0 || nz <= 0 || nn <= 4) throw Error(DSM_ERR_INVALID, "empty PSV set-up");
        d.nzone = nz; d.nn = nn; d.R = R; d.Th = Th;
        d.itmp = (s->rmin == 0.0) ? 3 : 1;
        d.jsrc = s->jsrc; d.spn = s->spn;
        if (d.jsrc < d.itmp || d.jsrc + 3 > nn) throw Error(DSM_ERR_INVALID, "source rows outside the system");
        d.n_sel = s->n_sel; d.n_fel = s->n_fel; d.n_hm = s->n_hm;
        d.tlen = tlen; d.omegai = omegai; d.rmax = s->rmax; d.r0 = s->r0;
        d.ecC0 = s->ecC0; d.ecF0 = s->ecF0; d.ecL0 = s->ecL0; d.ra0 = s->ra_src[0]; d.ra1 = s->ra_src[1];
        iphase.upload(s->iphase, nz, st); nlayer.upload(s->nlayer, nz, st); kkdr.upload(s->kkdr, nz, st);
        elem.upload(s->elem, nz, st); hmoff.upload(s->hmoff, nz, st);
        qmu.upload(s->qmu, nz, st); qkappa.upload(s->qkappa, nz, st);
        sel.upload(s->solid_el, (size_t)DSM_PSV_NSOLID * s->n_sel, st);
        fel.upload(s->fluid_el, (size_t)3 * s->n_fel, st);
        hm.upload(s->hm_el, (size_t)DSM_PSV_NHM * 4 * s->n_hm, st);
        poly.upload(s->src_poly, 24, st);
        // zone blocks and the column assembly map
        std::vector<int> bo(nz);
        int tot = 0;
        for (int z = 0; z < nz; ++z) {
            bo[z] = tot;
            tot += (s->iphase[z] == 1) ? 2 * (s->nlayer[z] + 1) : s->nlayer[z] + 1;
        }
        d.ncol_tot = tot;
        blkoff.upload(bo, st);
        std::vector<int> az(2 * (nn + 1), -1), ac(2 * (nn + 1), 0), br(nn + 1, 0);
        std::vector<double> bv(nn + 1, 0.0);
        for (int z = 0; z < nz; ++z) {
            int kk = s->kkdr[z];
            int hi = (s->iphase[z] == 1) ? kk + 2 * s->nlayer[z] + 1 : kk + s->nlayer[z];
            for (int jj = kk; jj <= hi && jj <= nn; ++jj) {
                int e = (az[2 * jj] < 0) ? 0 : 1;
                if (e == 1 && az[2 * jj + 1] >= 0) throw Error(DSM_ERR_INVALID, "three zones overlap a column");
                az[2 * jj + e] = z;
                ac[2 * jj + e] = jj - kk + 1;
            }
        }
        for (int i = 1; i <= nz - 1; ++i) {
            double rv = s->vrmax[i - 1] * s->vrmax[i - 1];
            if (s->iphase[i - 1] == 1 && s->iphase[i] == 2) { br[s->kkdr[i]] = 2; bv[s->kkdr[i]] = rv; }
            if (s->iphase[i - 1] == 2 && s->iphase[i] == 1) { br[s->kkdr[i]] = 3; bv[s->kkdr[i]] = rv; }
        }
        amz.upload(az, st); amc.upload(ac, st); bcrow.upload(br, st); bcval.upload(bv, st);
        {
            std::vector<int4> ra(nn + 1);
            for (int jj = 0; jj <= nn; ++jj) {
                int4 v = make_int4(-1, -1, 0, br[jj]);
                for (int e = 0; e < 2; ++e) {
                    const int z = az[2 * jj + e];
                    if (z < 0) break;
                    const int o = (bo[z] + ac[2 * jj + e] - 1) * 4;
                    if (e == 0) v.x = o; else v.y = o;
                    if (s->iphase[z] == 1) v.z |= 1 << e;
                }
                ra[jj] = v;
            }
            rowasm.upload(ra, st);
        }
        // receivers
        r.upload(s->r, R, st);
        rrsta.upload(s->rrsta, 3 * (size_t)R, st);
        std::vector<int> ks(R), fl(R), cm(nn + 1, -1), rc(6 * (size_t)R);
        std::vector<double> frv(R);
        auto addcap = [&](int j) {
            if (j < d.itmp || j > nn) throw Error(DSM_ERR_INVALID, "receiver stencil outside the system");
            if (cm[j] < 0) cm[j] = ncap++;
            return cm[j];
        };
        for (int ir = 0; ir < R; ++ir) {
            int z = s->istazone[ir] - 1;
            ks[ir] = s->kkdr[z] + 2 * s->iista[3 * ir] - 1;
            fl[ir] = s->iphase[z] == 2;
            frv[ir] = (double)(float)s->r[ir];
            for (int k = 0; k < 6; ++k) rc[6 * ir + k] = addcap(ks[ir] - 1 + k);
        }
        d.cap_n1 = addcap(nn - 1);
        d.cap_n = addcap(nn);
        d.cap_p0 = cm[ks[R - 1] - 1];
        d.cap_p1 = cm[ks[R - 1]];

        rcap.upload(rc, st); fluid.upload(fl, st);
        {
            std::vector<int> rt(R);
            for (int ir = 0; ir < R; ++ir) rt[ir] = ks[ir] + 4 - d.itmp + 1;
            stoprow.upload(rt, st);
        }
        {  // receiver rows of the field matrices: solid class (with the surface) and fluid
            std::vector<int> rw(R + 1);
            int ns = 0, nf = 0;
            for (int ir = 0; ir < R; ++ir) rw[ir] = fl[ir] ? -(++nf) : ns++;
            rw[R] = ns++;
            d.Rs1 = ns;
            d.Rf = nf;
            rrow.upload(rw, st);
            d.rrow = rrow.p;
        }
        lam.upload(s->lambda, R, st); qkp.upload(s->qkp, R, st); fr.upload(frv, st);
        // l = 0 compaction (rea2): jsta, compact row of every kept global row
        {
            std::vector<int> js(R, 0), cs(nn + 1, 0), lc(nn + 2, 0), le(nn + 2, 0);
            int itmp = 0;
            for (int iz = 0; iz < nz; ++iz) {
                for (int ir = 0; ir < R; ++ir)
                    if (iz + 1 == s->istazone[ir]) js[ir] = itmp + s->iista[3 * ir];
                int kk = s->kkdr[iz], i1 = itmp + 1, i2;
                if (s->iphase[iz] == 1) {
                    i2 = (iz != nz - 1) ? i1 + (s->kkdr[iz + 1] - kk) / 2 - 1 : i1 + (nn + 1 - kk) / 2 - 1;
                    for (int i = i1; i <= i2; ++i) {
                        cs[kk + 2 * (i - i1)] = i;
                        lc[i] = kk + 2 * (i - i1);
                        le[i] = (i == i1) ? (iz == 0 ? 0 : (s->iphase[iz - 1] == 2 ? 3 : 2)) : 2;
                    }
                } else {
                    i2 = i1 + (s->kkdr[iz + 1] - kk) - 1;
                    for (int i = i1; i <= i2; ++i) {
                        cs[kk + (i - i1)] = i;
                        lc[i] = kk + (i - i1);
                        le[i] = (i == i1) ? (iz == 0 ? 0 : (s->iphase[iz - 1] == 1 ? 2 : 3)) : 3;
                    }
                }
                itmp = i2;
            }
            lc.resize(itmp + 1);
            le.resize(itmp + 1);
            l0col.upload(lc, st);
            l0e1.upload(le, st);
            d.nn0 = itmp;
            d.itmp0 = (s->rmin == 0.0) ? 2 : 1;
            jsta.upload(js, st);
            comp_src.upload(cs, st);
            for (int ir = 0; ir < R; ++ir)
                if (js[ir] < 1 || js[ir] + 2 > d.nn0) throw Error(DSM_ERR_INVALID, "receiver outside the l=0 system");
        }
        vtop = 0.0;
        for (int i = 0; i < 4; ++i) vtop = vtop + s->vsv[4 * (nz - 1) + i] * 1.0;
        rtop = s->vrmax[nz - 1];
        vtop_ = vtop;
        rtop_ = rtop;
        for (int k = 0; k < nsrc; ++k) set_near_orders(k, ss[k]->r0, s->r[R - 1]);
        set_summaries(1, nz, s->vrmin, s->vrmax, s->vsv, s->qmu, s->r0, s->r[R - 1]);
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
        d.iphase = iphase.p; d.nlayer = nlayer.p; d.kkdr = kkdr.p; d.elem = elem.p; d.hmoff = hmoff.p;
        d.blkoff = blkoff.p; d.qmu = qmu.p; d.qkappa = qkappa.p; d.sel = sel.p; d.fel = fel.p; d.hm = hm.p;
        d.amz = amz.p; d.amc = amc.p; d.bcrow = bcrow.p; d.bcval = bcval.p; d.poly = poly.p;
        d.rowasm = rowasm.p;
        d.rcap = rcap.p; d.stop_row = stoprow.p; d.wv = wv.p; d.wd = wd.p; d.fluid = fluid.p; d.lam = lam.p; d.qkp = qkp.p;
        d.fr = fr.p; d.comp_src = comp_src.p; d.jsta = jsta.p;
        // per-source parameter sets: the fields set by the source position
        {
            std::vector<double> pl(24 * (size_t)nsrc);
            for (int k = 0; k < nsrc; ++k)
                for (int i = 0; i < 24; ++i) pl[24 * (size_t)k + i] = ss[k]->src_poly[i];
            polys.upload(pl, st);
            dsrc.assign(nsrc, d);
            ls_min = d.nn;
            for (int k = 0; k < nsrc; ++k) {
                const dsm_psv_setup_t* q = ss[k];
                PsvDev& e = dsrc[k];
                e.jsrc = q->jsrc;
                e.spn = q->spn;
                if (e.jsrc < e.itmp || e.jsrc + 3 > nn) throw Error(DSM_ERR_INVALID, "source rows outside the system");
                e.r0 = q->r0;
                e.ecC0 = q->ecC0; e.ecF0 = q->ecF0; e.ecL0 = q->ecL0;
                e.ra0 = q->ra_src[0]; e.ra1 = q->ra_src[1];
                e.poly = polys.p + 24 * (size_t)k;
                ls_min = std::min(ls_min, e.jsrc - e.itmp + 1);
            }
            d = dsrc[0];
        }
        {  // nodes of the depth cut-off (the grid of calra2_psv, its unknowns of calspdr)
            std::vector<float4> nd;
            double r0min = s->r0;
            for (int k = 1; k < nsrc; ++k) r0min = std::min(r0min, ss[k]->r0);
            auto inv_v2 = [&](int z, double rr) {
                if (s->iphase[z] != 1) return 1e30;
                double v = 0.0, x = 1.0;
                for (int j = 0; j < 4; ++j, x *= rr / s->rmax) v += s->vsv[4 * z + j] * x;
                return v > 0.0 ? 1.0 / (v * v) : 1e30;
            };
            nd.push_back(make_float4((float)s->vrmin[0], (float)inv_v2(0, s->vrmin[0]),
                                     (float)(s->kkdr[0] - d.itmp + 1), 0.0f));
            for (int z = 0; z < nz; ++z) {
                const int nl = s->nlayer[z];
                for (int i = 1; i <= nl; ++i) {
                    const double rr = s->vrmin[z] + (s->vrmax[z] - s->vrmin[z]) * (double)i / (double)nl;
                    double iv = inv_v2(z, rr);
                    if (i == nl && z + 1 < nz) iv = std::max(iv, inv_v2(z + 1, rr));  // the slower side
                    const int row = s->kkdr[z] + (s->iphase[z] == 1 ? 2 * i : i);
                    nd.push_back(make_float4((float)rr, (float)iv, (float)(row - d.itmp + 1), 0.0f));
                }
            }
            cnode_src = 0;
            for (int k = 0; k < (int)nd.size(); ++k)
                if ((double)nd[k].x <= r0min) cnode_src = k;
            cnodes.upload(nd, st);
            hnodes = nd;
        }
        depth_bound = mixed() ? 1e-20 : 0.0;
        plan_segments(cm, az, s);
        F = opt.freq_batch > 0 ? opt.freq_batch : 8;
        Lc = opt.l_chunk > 0 ? ((opt.l_chunk + 31) / 32) * 32 : 256;
        Lcap = (std::min(maxlmax + 1 + Lc, 2048) + 7) / 8 * 8;
        amp_k = 1;
        rows_m[0] = (int)psvk::fld_rows(NS0, d.Rs1, d.Rf);
        rows_m[1] = (int)psvk::fld_rows(NS1, d.Rs1, d.Rf);
        rows_m[2] = (int)psvk::fld_rows(NS2, d.Rs1, d.Rf);
        rows_full[0] = (int)psvk::fld_rows_full(NS0, d.Rs1);
        rows_full[1] = (int)psvk::fld_rows_full(NS1, d.Rs1);
        rows_full[2] = (int)psvk::fld_rows_full(NS2, d.Rs1);
        // contraction outputs row-major: the epilogue's lanes take
        // consecutive distances of one row (the rows of a receiver are
        // adjacent, psvk::fld_row)
        c_rowmajor = true;
        c_ld = (ncols() + 3) / 4 * 4;
        {  // receiver row (0..R) of each field row, for the split's zero orders
            std::vector<int> solid_r(d.Rs1, R), fluid_r(std::max(d.Rf, 1), 0);
            std::vector<int> rw(R + 1);
            DSM_CUDA(cudaStreamSynchronize(st));  // rrow was uploaded on st
            DSM_CUDA(cudaMemcpy(rw.data(), rrow.p, sizeof(int) * (R + 1), cudaMemcpyDeviceToHost));
            for (int ir = 0; ir < R; ++ir) {
                if (rw[ir] >= 0) solid_r[rw[ir]] = ir;
                else fluid_r[-rw[ir] - 1] = ir;
            }
            const int nqs[3] = {NS0, NS1, NS2};
            for (int m = 0; m < 3; ++m) {
                std::vector<int> rr_of(rows_m[m], R);
                for (int rr = 0; rr < d.Rs1; ++rr)
                    for (int q = 0; q < nqs[m]; ++q)
                        for (int f = 0; f < 5; ++f) {
                            int im;
                            const long long row = psvk::fld_row(nqs[m], d.Rs1, d.Rf, q, f, rr, &im);
                            rr_of[row] = rr_of[row + im] = solid_r[rr];
                        }
                for (int fi = 0; fi < d.Rf; ++fi)
                    for (int q = 0; q < nqs[m]; ++q) {
                        int im;
                        const long long row = psvk::fld_row(nqs[m], d.Rs1, d.Rf, q, 0, -fi - 1, &im);
                        rr_of[row] = rr_of[row + im] = fluid_r[fi];
                    }
                rowrec[m].upload(rr_of, st);
            }
            zfirst.reserve((size_t)nsrc * F * (R + 1));
            use_zfirst = mixed();
        }
        alloc_batch();
        build_basis(std::min(maxlmax + 1, 2048));
        DSM_CUDA(cudaStreamSynchronize(st));
    }

    ~PsvEngine() override {
        if (st3) {
            cudaStreamSynchronize(st3);
            cudaStreamDestroy(st3);
        }
        for (cudaStream_t s : sfac)
            if (s) {
                cudaStreamSynchronize(s);
                cudaStreamDestroy(s);
            }
        for (cudaEvent_t e : ev_fac)
            if (e) cudaEventDestroy(e);
        if (ev_s3a) cudaEventDestroy(ev_s3a);
        if (ev_s3b) cudaEventDestroy(ev_s3b);
    }

    // every source of a context shares the model, grid, receivers and
    // distances; only the source fields may differ
    static void check_same_grid(const dsm_psv_setup_t* a, const dsm_psv_setup_t* b) {
        if (!b) throw Error(DSM_ERR_INVALID, "null PSV set-up");
        auto same = [](const void* x, const void* y, size_t bytes) {
            return bytes == 0 || (x && y && std::memcmp(x, y, bytes) == 0);
        };
        const bool ok =
            a->nzone == b->nzone && a->nn == b->nn && a->r_n == b->r_n && a->theta_n == b->theta_n &&
            a->n_sel == b->n_sel && a->n_fel == b->n_fel && a->n_hm == b->n_hm && a->rmin == b->rmin &&
            a->rmax == b->rmax && a->tlen == b->tlen && a->omegai == b->omegai && a->ratl == b->ratl &&
            a->maxlmax == b->maxlmax && a->rsgt_switch == b->rsgt_switch && a->synn_switch == b->synn_switch &&
            same(a->iphase, b->iphase, sizeof(int) * a->nzone) && same(a->nlayer, b->nlayer, sizeof(int) * a->nzone) &&
            same(a->kkdr, b->kkdr, sizeof(int) * a->nzone) && same(a->elem, b->elem, sizeof(int) * a->nzone) &&
            same(a->hmoff, b->hmoff, sizeof(int) * a->nzone) && same(a->qmu, b->qmu, sizeof(double) * a->nzone) &&
            same(a->qkappa, b->qkappa, sizeof(double) * a->nzone) &&
            same(a->solid_el, b->solid_el, sizeof(double) * DSM_PSV_NSOLID * a->n_sel) &&
            same(a->fluid_el, b->fluid_el, sizeof(double) * 3 * a->n_fel) &&
            same(a->hm_el, b->hm_el, sizeof(double) * DSM_PSV_NHM * 4 * a->n_hm) &&
            same(a->r, b->r, sizeof(double) * a->r_n) && same(a->rrsta, b->rrsta, sizeof(double) * 3 * a->r_n) &&
            same(a->iista, b->iista, sizeof(int) * 3 * a->r_n) &&
            same(a->istazone, b->istazone, sizeof(int) * a->r_n) &&
            same(a->theta, b->theta, sizeof(double) * a->theta_n);
        if (!ok)
            throw Error(DSM_ERR_INVALID,
                        "the sources of a context must share the model, grid, receivers and distances");
    }

    // Segments of the band solve (psv_seg.cu): separators of three rows below
    // the sources, then the segment up to the source rows and the one above
    // them.  The separators do not depend on the source, so a source has the
    // same arithmetic alone and beside others.
    void plan_segments(const std::vector<int>& cm, const std::vector<int>& az, const dsm_psv_setup_t* s) {
        const int n = d.nn - d.itmp + 1;
        // the eight pieces of a row hold one phase (calspdr gives zones of
        // different phases rows of their own, src/SGTpsv/others.f90)
        for (int jj = 1; jj <= d.nn; ++jj)
            if (az[2 * jj + 1] >= 0 && s->iphase[az[2 * jj]] != s->iphase[az[2 * jj + 1]])
                throw Error(DSM_ERR_INVALID, "a band row shared by zones of different phases");
        for (const PsvDev& e : dsrc) {
            const int above = n - (e.jsrc - e.itmp + 1);  // 3: the source rows are the band's last four
            if (above != 3 && above < 5) throw Error(DSM_ERR_INVALID, "source rows split the surface rows");
        }
        std::vector<int> row, slot, gi;
        for (int j = d.itmp; j <= d.nn; ++j)
            if (cm[j] >= 0) {
                row.push_back(j - d.itmp + 1);
                slot.push_back(cm[j]);
                if (cm[j] == d.cap_p0) row_p0 = row.back();
                if (cm[j] == d.cap_p1) row_p1 = row.back();
            }
        for (size_t c = 0; c < row.size(); ++c)
            gi.push_back(c + 1 < row.size() && row[c + 1] == row[c] + 1 ? -1 : ngap++);
        const int nc = (int)row.size();
        row.push_back(INT_MAX);
        caprow.upload(row, st);
        capslot.upload(slot, st);
        gapidx.upload(gi, st);
        // Nine parts of the band, of 64 rows or more.  More parts shorten the
        // longest chain of rows, but all parts above a system's bottom one
        // carry the fill-in (twice the operations of a row): on the
        // 2048-frequency grid the factorisation of three slices took 6.8, 4.0,
        // 2.8 and 2.9 ms with 2, 5, 9 and 11 parts, that of twenty 13.6, 14.0,
        // 14.2 and 14.8 ms.
        int G = 8;
        G = std::max(0, std::min({G, psvseg::MAXSEG - 2, n / 64 - 1}));
        std::vector<int> all(G);
        for (int g = 0; g < G; ++g) all[g] = (int)((long long)n * (g + 1) / (G + 1));
        nsep_max = 0;
        for (const PsvDev& e : dsrc) {
            const int ls = e.jsrc - e.itmp + 1;
            nsep_max = std::max(nsep_max, (int)(std::lower_bound(all.begin(), all.end(), ls - 18) - all.begin()));
        }
        for (const PsvDev& e : dsrc) {
            psvseg::Plan P{};
            P.n = n;
            P.ls = e.jsrc - e.itmp + 1;
            P.merged = n == P.ls + 3;
            const std::vector<int> sep(all.begin(), std::lower_bound(all.begin(), all.end(), P.ls - 18));
            const int G = (int)sep.size();
            P.nseg = G + 2;
            for (int i = 0; i < G; ++i) {
                P.a[i] = i == 0 ? 1 : sep[i - 1] + 3;
                P.b[i] = sep[i] - 1;
                P.order[i] = G - 1 - i;
                P.slot[i] = i;
            }
            for (int i = 0; i < 2; ++i) {
                P.order[G + i] = G + i;
                P.slot[G + i] = nsep_max + i;
            }
            P.a[G] = G == 0 ? 1 : sep[G - 1] + 3;
            P.b[G] = P.ls - 1;
            P.a[G + 1] = P.ls + 4;
            P.b[G + 1] = n - 2;
            for (int i = 0; i < P.nseg; ++i) {
                P.clo[i] = (int)(std::lower_bound(row.begin(), row.begin() + nc, P.a[i]) - row.begin());
                P.chi[i] = std::max(P.clo[i], (int)(std::upper_bound(row.begin(), row.begin() + nc, P.b[i]) - row.begin()));
            }
            // longest first: the last blocks to start end soon after
            std::stable_sort(P.order + (nsrc > 1 ? G : 0), P.order + P.nseg,
                             [&](int x, int y) { return P.b[x] - P.a[x] > P.b[y] - P.a[y]; });
            for (int& v : P.ifcap) v = -1;
            auto cap_of = [&](int j) { return cm[j + d.itmp - 1]; };
            for (int i = 0; i < G; ++i)
                for (int c = 0; c < 3; ++c) P.ifcap[3 * i + c] = cap_of(sep[i] + c);
            for (int c = 0; c < 4; ++c) P.ifcap[3 * G + c] = cap_of(P.ls + c);
            if (!P.merged)
                for (int c = 0; c < 2; ++c) P.ifcap[3 * G + 4 + c] = cap_of(n - 1 + c);
            plans.push_back(P);
        }
        int c0 = nc;
        for (const psvseg::Plan& P : plans) c0 = std::min(c0, P.clo[P.nseg - 2]);
        nctop = nc - c0;
        for (int c = c0; c < nc; ++c) ngtop += gi[c] >= 0;
    }

    void alloc_batch() {
        // scratch of a system: captured solutions and their rows' records,
        // gap records, segment ends, interface solutions, source weights
        const size_t nif = 3 * (size_t)nsep_max + 6;
        auto per = [&](int nfac) {
            return 16 * ((size_t)ncap * (NB + psvseg::NREC_ROW) + (size_t)ngap * psvseg::NREC_GAP +
                         (size_t)(nsep_max + 2 * nfac) * psvseg::NREC_END + nif * NB + NSLOT * NB +
                         (size_t)(nfac - 1) * ((size_t)nctop * psvseg::NREC_ROW + (size_t)ngtop * psvseg::NREC_GAP));
        };
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        // What the rest of a run allocates later, at the order capacity the
        // top frequency's first range needs: the field matrices (while they
        // grow, old and new copies), the split pieces and contraction output
        // of the mixed path, the batch outputs, and a margin.  The solve
        // scratch takes what is left, so that a batch's first ranges fit one
        // launch (one long low-order recurrence per batch, not one per round).
        size_t lfut = (size_t)Lcap;
        while (lfut < (size_t)first_span(imax) + 64 && lfut < (size_t)maxlmax + 1 + Lc) lfut *= 2;
        lfut = std::min(lfut, (size_t)maxlmax + 1 + Lc);
        size_t rows_all = 0;
        for (int m = 0; m < 3; ++m) rows_all += (size_t)rows_m[m];
        size_t pt, pr, ps;
        out_sizes(&pt, &pr, &ps);
        const size_t later = rows_all * lfut * (size_t)nsrc * F * afld_bytes * 3 / 2 +
                             (mixed() ? rows_all * lfut * F * 4 + c_total() * F * 4 : c_total() * 8) +
                             2 * (pt + pr + ps) * F * nsrc * 8 + ((size_t)4 << 30);
        const size_t avail = fr > later ? fr - later : 0;
        // no more than a round of a batch can launch (F ranges of at most
        // max(4096, the first range of the top frequency)): contexts that
        // share a device leave each other room
        int near = 0;
        for (int k = 0; k < nsrc; ++k) near = std::max(near, near_span(k));
        const int most = std::max(1024, F * std::max({4096, first_span(imax), near}));
        while (nfac > 1 && avail / per(nfac) < (size_t)std::min(most, 131072)) --nfac;
        nsys_max = std::min(most, (int)std::max<size_t>(1024, std::min<size_t>(131072, avail / per(nfac))));
        // DSM_MAX_SYSTEMS caps the systems per solve launch (and so the
        // factor scratch) below that, e.g. for small profiling captures
        if (const char* e = std::getenv("DSM_MAX_SYSTEMS")) nsys_max = std::max(1024, std::min(nsys_max, std::atoi(e)));
        nsys_max = nsys_max / 32 * 32;  // whole warps of one frequency's orders
        size_t nsys = nsys_max;
        B0.reserve((size_t)F * d.ncol_tot * 4);
        B1.reserve((size_t)F * d.ncol_tot * 4);
        B2.reserve((size_t)F * d.ncol_tot * 4);
        P8.reserve((size_t)F * (d.nn + 1 + psvseg::PAD_ROWS) * psvseg::ROW_CD);
        Lrec.reserve(((size_t)ncap + (size_t)(nfac - 1) * nctop) * psvseg::NREC_ROW * nsys);
        Grec.reserve(((size_t)std::max(ngap, 1) + (size_t)(nfac - 1) * ngtop) * psvseg::NREC_GAP * nsys);
        Send.reserve((size_t)(nsep_max + 2 * nfac) * psvseg::NREC_END * nsys);
        Xif.reserve(nif * NB * nsys);
        Xcap.reserve((size_t)ncap * NB * nsys);
        Xprobe.reserve((size_t)8 * nsys);
        kcut.reserve(nsys);
        l0scr.reserve((size_t)F * (d.nn0 + 1) * 2);
        l0d.reserve((size_t)F * (d.nn0 + 1) * 4);
        ab.reserve((size_t)nsrc * F * 320);
        co.reserve((size_t)NSLOT * NB * nsys);
        for (int m = 0; m < 3; ++m) Afld[m].reserve(((size_t)nsrc * F * rows_m[m] * Lcap * afld_bytes + 7) / 8);
        Cgemm.reserve(c_total());
        cut.reserve((size_t)nsrc * F);
        amps.reserve((size_t)nsrc * F * Lcap);
        out_t.reserve(2 * pt * F * nsrc);
        out_r.reserve(2 * pr * F * nsrc);
        out_s.reserve(2 * ps * F * nsrc);
    }

    size_t out_sizes(size_t* nt, size_t* nr, size_t* ns) const override {
        *nt = (size_t)num_t * R * Th;
        *nr = (size_t)num_r * R * Th;
        *ns = (size_t)num_s * Th;
        return *nt;
    }

    bool l0_done = false;
    void omega_pieces(const int* fr_, int nf) override {
        l0_done = false;
        // first zero order per receiver row: none yet (0x7f7f7f7f)
        if (use_zfirst) DSM_CUDA(cudaMemsetAsync(zfirst.p, 0x7f, sizeof(int) * (size_t)nsrc * F * (R + 1), st));
        dim3 grid((d.ncol_tot + 127) / 128, nf);
        int id = kid("psv_omega_blocks");
        kbegin(id);
        k_psv_omega<<<grid, 128, 0, st>>>(d, fr_, B0.p, B1.p, B2.p);
        DSM_LAUNCH(*this);
        const int nrow = d.nn + 1 + psvseg::PAD_ROWS;
        k_psv_rows<<<dim3((nrow + 127) / 128, nf), 128, 0, st>>>(d, B0.p, B1.p, B2.p, P8.p, nrow);
        kend(id, 0.0, 0.0);
        DSM_LAUNCH(*this);
        for (int k = 0; k < nsrc; ++k) {
            k_psv_abnum<<<(nf + 31) / 32, 32, 0, st>>>(dsrc[k], fr_, nf, ab.p + (size_t)k * F * 320);
            DSM_LAUNCH(*this);
        }
    }

    void solve_chunk(const int* fr_, int nf, const WorkList& wl, int nsys) override {
        if (!l0_done) {  // order 0 once per batch (its own tridiagonal system)
            // order 0 is independent of the other orders: it runs on the side
            // stream while the band solves run, and joins before the l-sum.
            // Its solve factors the compact band in place: every source
            // rebuilds it first.
            fork_side();
            int id0 = kid("psv_order0");
            kbegin(id0, st2);
            for (int k = 0; k < nsrc; ++k) {
                const PsvDev& e = dsrc[k];
                const cd* abk = ab.p + (size_t)k * F * 320;
                k_psv_l0_build<<<dim3((d.nn0 + 127) / 128, nf), 128, 0, st2>>>(e, B0.p, B1.p, B2.p, l0col.p,
                                                                                l0e1.p, l0scr.p);
                k_psv_l0_solve<<<nf, L0_T, L0_SMEM, st2>>>(e, fr_, nf, abk, l0scr.p, l0d.p, rsgt_sw);
                if (afld_bytes == 4)
                    k_psv_l0_fields<float><<<dim3((R + 1 + 127) / 128, nf), 128, 0, st2>>>(
                        e, l0d.p, afld_of<float>(0, k), afld_of<float>(1, k), afld_of<float>(2, k), Lcap, rsgt_sw);
                else
                    k_psv_l0_fields<double><<<dim3((R + 1 + 127) / 128, nf), 128, 0, st2>>>(
                        e, l0d.p, afld_of<double>(0, k), afld_of<double>(1, k), afld_of<double>(2, k), Lcap,
                        rsgt_sw);
                DSM_LAUNCH(*this);
            }
            kend(id0, 0.0, 0.0, st2);
            l0_done = true;
        }
        solve_segments(fr_, wl, nsys);
    }

    // source k's weights and receiver fields from the captured solutions
    void source_fields(int k, const int* fr_, const WorkList& wl, int nsys, const int* kc) {
        const PsvDev& e = dsrc[k];
        const int nb = (nsys + 127) / 128, fs = tune.fld_orders == 16 ? 16 : 32, frec = 32 / fs;
        int id = kid("psv_source_coef");
        kbegin(id);
        k_psv_coef<<<(nsys + COEF_S - 1) / COEF_S, COEF_S * COEF_R, 0, st>>>(e, fr_, wl, nsys, ab.p + (size_t)k * F * 320, co.p, rsgt_sw, Xprobe.p,
                                       amps.p + (size_t)k * F * Lcap, Lcap);
        kend(id, 0.0, 0.0);
        DSM_LAUNCH(*this);
        const dim3 grid((unsigned)(nb * (128 / fs)), (R + 1 + 4 * frec - 1) / (4 * frec));
        id = kid("psv_fields");
        kbegin(id);
        if (afld_bytes == 4) {
            auto kern = fs == 16 ? k_psv_fields<true, 16> : k_psv_fields<true, 32>;
            kern<<<grid, 128, 0, st>>>(e, wl, nsys, Xcap.p, co.p, afld_of<float>(0, k), afld_of<float>(1, k),
                                       afld_of<float>(2, k), Lcap, kc,
                                       use_zfirst && kc ? zfirst.p + (size_t)k * F * (R + 1) : nullptr);
        } else {
            auto kern = fs == 16 ? k_psv_fields<false, 16> : k_psv_fields<false, 32>;
            kern<<<grid, 128, 0, st>>>(e, wl, nsys, Xcap.p, co.p, afld_of<double>(0, k), afld_of<double>(1, k),
                                       afld_of<double>(2, k), Lcap, kc, nullptr);
        }
        kend(id, 0.0, 0.0);
        DSM_LAUNCH(*this);
    }

    // FP64 operations of a factorisation launch (a fused multiply-add counts
    // two), counted when profiling: 102 per row of a bottom segment, 196 with
    // the fill-in
    double factor_flops(const psvseg::Plan& P, int s0, int s1, int nsys, const int* kc) {
        if (!prof) return 0.0;
        std::vector<int> h(nsys, 1);
        if (kc) {
            DSM_CUDA(cudaMemcpyAsync(h.data(), kc, sizeof(int) * nsys, cudaMemcpyDeviceToHost, st));
            DSM_CUDA(cudaStreamSynchronize(st));
        }
        double f = 0.0;
        for (int v : h) {
            int bot = 0;
            while (bot + 2 < P.nseg && v >= P.a[bot + 1]) ++bot;
            for (int i = s0; i < s1; ++i) {
                const int seg = P.order[i], rows = P.b[seg] - P.a[seg] + 1;
                if (seg == bot) f += 2.0 * 102 * (P.b[seg] - std::max(P.a[seg], std::min(v, P.b[seg])) + 1);
                else if (seg > bot && rows > 0) f += 2.0 * 196 * rows;
            }
        }
        return f;
    }

    // band solves of a round in row segments: the segments below the sources
    // once, the two around each source with that source's turn
    void solve_segments(const int* fr_, const WorkList& wl, int nsys) {
        const int* kc = nullptr;
        if (depth_bound > 0.0 && ls_min > 9) {
            k_psv_cutrow<<<(nsys + 127) / 128, 128, 0, st>>>(cnodes.p, cnode_src, (float)-std::log(depth_bound),
                                                             d.tlen, fr_, wl, nsys, ls_min - 8, kcut.p);
            DSM_LAUNCH(*this);
            kc = kcut.p;
        }
        psvseg::Dev g{};
        g.wl = wl;
        g.nsys = nsys;
        g.it = d.itmp;
        g.nrow = d.nn + 1 + psvseg::PAD_ROWS;
        g.P8 = P8.p;
        g.kcut = kc;
        g.caprow = caprow.p;
        g.capslot = capslot.p;
        g.gapidx = gapidx.p;
        g.Lrec = Lrec.p;
        g.Grec = Grec.p;
        g.Send = Send.p;
        g.Xif = Xif.p;
        g.Xcap = Xcap.p;
        g.Xprobe = Xprobe.p;
        g.cap_p0 = d.cap_p0;
        g.cap_p1 = d.cap_p1;
        g.row_p0 = row_p0;
        g.row_p1 = row_p1;
        g.moved = solve_count();
        g.plain = !mixed();
        // segments [s0, s1) of a plan, those with fill-in on sf; st waits for
        // the systems' bottom ones (on st3)
        auto factor = [&](const psvseg::Dev& g, const psvseg::Plan& P, int s0, int s1, cudaStream_t sf) {
            if (s1 <= s0) return;
            DSM_CUDA(cudaEventRecord(ev_s3a, st));
            DSM_CUDA(cudaStreamWaitEvent(st3, ev_s3a, 0));
            if (sf != st) DSM_CUDA(cudaStreamWaitEvent(sf, ev_s3a, 0));
            psvseg::launch_factor(g, P, s0, s1, sf, st3);
            launches++;
            DSM_LAUNCH(*this);
        };
        auto factored = [&] {
            DSM_CUDA(cudaEventRecord(ev_s3b, st3));
            DSM_CUDA(cudaStreamWaitEvent(st, ev_s3b, 0));
        };
        // several sources: from the shallowest down, nfac at a time.  The
        // segments between separators serve all of them; those around a
        // source are factored side by side (two chains of rows fill few SMs),
        // each source's records in its own part.  The first of a group writes
        // over the records above its last separator, which only shallower
        // sources read.  Three depths, four frequencies: 3.7 ms of
        // factorisations one after the other, 2.1 side by side.
        std::vector<int> ord;
        for (int k = 0; k < nsrc; ++k)
            if (src_open[k]) ord.push_back(k);  // a source past its cutoffs needs no further orders
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return plans[a].ls > plans[b].ls; });
        const int fid = kid("psv_factor");
        psvseg::Plan group[MAX_SRC_FAC];
        for (size_t o = 0; o < ord.size(); ++o) {
            const int k = ord[o], gi = (int)(o % nfac);
            if (gi == 0) {
                const int ng = (int)std::min<size_t>(nfac, ord.size() - o);
                kbegin(fid);
                double fl = 0.0;
                for (int i = ng - 1; i >= 0; --i) {  // st's own last: the others wait for what it holds so far
                    psvseg::Plan& P = group[i];
                    P = plans[ord[o + i]];
                    P.cshift = i * nctop;
                    P.gshift = i * ngtop;
                    P.first = o + i == 0;
                    for (int e = 0; e < 2; ++e) P.slot[P.nseg - 2 + e] = nsep_max + 2 * i + e;
                    psvseg::Dev gk = g;
                    gk.Lrec += (size_t)P.cshift * psvseg::NREC_ROW * nsys;
                    gk.Grec += (size_t)P.gshift * psvseg::NREC_GAP * nsys;
                    const int s0 = o + i > 0 ? P.nseg - 2 : 0;  // the shallowest source's plan holds every separator
                    factor(gk, P, s0, P.nseg, i == 0 ? st : sfac[i - 1]);
                    fl += factor_flops(P, s0, P.nseg, nsys, kc);
                    if (i > 0) DSM_CUDA(cudaEventRecord(ev_fac[i], sfac[i - 1]));
                }
                factored();
                for (int i = 1; i < ng; ++i) DSM_CUDA(cudaStreamWaitEvent(st, ev_fac[i], 0));
                kend(fid, 0.0, fl);
            }
            const psvseg::Plan& P = group[gi];
            int id = kid("psv_join");
            kbegin(id);
            psvseg::launch_join(g, P, st);
            kend(id, 0.0, 0.0);
            DSM_LAUNCH(*this);
            id = kid("psv_substitution");
            kbegin(id);
            psvseg::launch_walk(g, P, st);
            kend(id, 0.0, 0.0);
            DSM_LAUNCH(*this);
            source_fields(k, fr_, wl, nsys, kc);
        }
    }

    void scan_chunk(int nf, const WorkList& wl) override {
        int id = kid("psv_cutoff_scan");
        kbegin(id);
        for (int k = 0; k < nsrc; ++k) {
            if (!src_open[k]) continue;
            k_psv_scan<<<(nf + 3) / 4, 128, 0, st>>>(nf, wl, Lcap, maxlmax, ratl, tlen, vtop, rtop, d_freqs.p,
                                                      amps.p + (size_t)k * F * Lcap, cut.p + (size_t)k * F,
                                                      dstatus());
            DSM_LAUNCH(*this);
        }
        kend(id, 0.0, 0.0);
    }

    void epilogue(const int* fr_, const std::vector<int>& ws, int nf, cudaStream_t s) override {
        psvk::EpiDev e{};
        e.R = R;
        e.Th = Th;
        e.tlen = d.tlen;
        e.omegai = d.omegai;
        e.fluid = d.fluid;
        e.Rs1 = d.Rs1;
        e.Rf = d.Rf;
        e.rrow = d.rrow;
        e.lam = d.lam;
        e.qkp = d.qkp;
        e.fr = d.fr;
        e.status = dstatus();
        e.c_ld = c_ld;
        e.Tb = Tb;
        e.Thalf = Thalf;
        for (int w : ws) {
            int id = kid("psv_epilogue");
            kbegin(id, s);
            const bool tc = mixed();
            const void* c0 = tc ? (const void*)c32(w, 0) : (const void*)c64(0);
            const void* c1 = tc ? (const void*)c32(w, 1) : (const void*)c64(1);
            const void* c2 = tc ? (const void*)c32(w, 2) : (const void*)c64(2);
            if (rec_direct)
                psvk::launch_epilogue(e, w, th.x.p, th.s.p, th.pole.p, fr_, c0, c1, c2, tc, rec_t(), rec_r(nf),
                                      rec_s(nf), s);
            else
                psvk::launch_epilogue(e, w, th.x.p, th.s.p, th.pole.p, fr_, c0, c1, c2, tc, out_t_src(),
                                      rsgt_sw ? out_r_src() : nullptr, synn_sw ? out_s_src() : nullptr, s);
            kend(id, 0.0, 0.0, s);
            DSM_LAUNCH(*this);
        }
    }
};

}  // namespace

Engine* make_psv_engine(const dsm_psv_setup_t* const* s, int nsrc, const dsm_options_t* o) {
    return new PsvEngine(s, nsrc, o);
}

}  // namespace dsm
