// Band solve of the P-SV systems in row segments.
//
// The band of one (omega, l) system (half-width 3, tens of thousands of
// rows) is needed at few places: six right-hand sides that are unit vectors
// of the four source rows and the two surface rows, and the solutions at the
// rows of the receivers' stencils.  The rows are cut into segments by
// separators (three rows; the source rows and the surface rows are
// separators too), so that no segment has a right-hand side inside:
//   k_seg_factor  eliminates a segment's rows in ascending order, one thread
//                 per (system, segment).  A segment above the bottom one
//                 carries the fill-in towards its left separator.  Instead
//                 of the multipliers of every row it keeps the product of
//                 the rows' back-substitution steps since the last captured
//                 row, x_low = P x_high + Q x_left (3 x 3 each), and writes
//                 it once per gap between captured rows; the multipliers go
//                 out for captured rows only.
//   k_seg_join    solves the separators' block-tridiagonal system, one
//                 thread per system.
//   k_seg_walk    walks each segment's records down from its upper
//                 separator to the captured rows.
// Replaces dcsymbdl0 / dcsbdlv0 (src/SGTpsv/dcsymbdl.f90:2-166) on the same
// equations: another elimination order, so results agree to rounding.
#include <climits>
#include <type_traits>

#include "psv_seg.cuh"

namespace dsm {
namespace psvseg {
namespace {

// c + a b, c - a b.  PLAIN (FP64 path): the real part of the product first,
// rounded once, then the sum, which cancels and is then mostly exact; added to
// c product by product (one operation less) the band's elimination was a
// quarter further off (pivot_sub).
template <bool PLAIN>
__device__ __forceinline__ cd mac(cd c, cd a, cd b) {
    if (PLAIN)
        return mk(__dadd_rn(c.re, fma(a.re, b.re, -__dmul_rn(a.im, b.im))), fma(a.re, b.im, fma(a.im, b.re, c.im)));
    return mk(fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im)));
}
template <bool PLAIN>
__device__ __forceinline__ cd msub(cd c, cd a, cd b) {
    if (PLAIN)
        return mk(__dsub_rn(c.re, fma(a.re, b.re, -__dmul_rn(a.im, b.im))), fma(-a.re, b.im, fma(-a.im, b.re, c.im)));
    return mk(fma(-a.re, b.re, fma(a.im, b.im, c.re)), fma(-a.re, b.im, fma(-a.im, b.re, c.im)));
}
__device__ __forceinline__ cd cmul(cd a, cd b) {
    return mk(fma(a.re, b.re, -a.im * b.im), fma(a.re, b.im, a.im * b.re));
}
__device__ __forceinline__ cd cnmul(cd a, cd b) {  // -a b
    return mk(fma(-a.re, b.re, a.im * b.im), fma(-a.re, b.im, -a.im * b.re));
}
// m / D with r = 1 / |D|^2
__device__ __forceinline__ cd over(cd m, cd D, double r) {
    return mk(fma(m.re, D.re, m.im * D.im) * r, fma(m.im, D.re, -(m.re * D.im)) * r);
}
// c - m m / D, a pivot's update, with w = m / D.  PLAIN: w's own rounding is
// taken out of the real part (m - w D, the remainder, times w): the pivots'
// errors add up along the band.  Relative L2 error of the FP64 outputs beyond
// 90 degrees against 80-bit arithmetic, 56 models x 3 frequencies, as a
// geometric mean over that of the sequential band solve (unfused, Smith's
// division): fused products alone 1.25, products first 1.05, with this 0.98
// (+- 0.02).
template <bool PLAIN>
__device__ __forceinline__ cd pivot_sub(cd c, cd w, cd m, cd D) {
    if (!PLAIN) return msub<false>(c, w, m);
    const double q = fma(w.im, D.im, fma(-w.re, D.re, m.re));
    return mk(__dsub_rn(c.re, fma(w.re, m.re, fma(q, w.re, -__dmul_rn(w.im, m.im)))),
              fma(-w.re, m.im, fma(-w.im, m.re, c.im)));
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
                 "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Where the band of a system starts.  Its first kept row kc (1 without the
// depth cut) lies in one segment or the separator above it: that segment is
// the bottom one and starts at kc (at its last row if kc lies in the
// separator: a lower start only keeps more rows).  Segments below it hold no
// rows, segments above it all of theirs.
__device__ __forceinline__ int bottom_segment(const Plan& p, int kc) {
    int i = 0;
    while (i + 2 < p.nseg && kc >= p.a[i + 1]) ++i;
    return i;
}
__device__ __forceinline__ int bottom_start(const Plan& p, int i, int kc) { return max(p.a[i], min(kc, p.b[i])); }

// band entries (row, row-3 .. row) from the row's pieces:
//   e0 = s Y1, e1 = X2 + L Y2, e2 = X3 + t Y3, e3 = X4 + L Y4,
// L = l(l+1), s = sqrt(L), t = s in solid rows and L in fluid rows
__device__ __forceinline__ void band_row(const cd (&v)[ROW_CD], double l2, double lsq, cd (&e)[4]) {
    const double t = v[7].re != 0.0 ? l2 : lsq;
    e[0] = mk(lsq * v[0].re, lsq * v[0].im);
    e[1] = mk(fma(l2, v[2].re, v[1].re), fma(l2, v[2].im, v[1].im));
    e[2] = mk(fma(t, v[4].re, v[3].re), fma(t, v[4].im, v[3].im));
    e[3] = mk(fma(l2, v[6].re, v[5].re), fma(l2, v[6].im, v[5].im));
}

constexpr int FAC_WARPS = 4;
constexpr int CH = 8, NCH = 4;  // staged rows per chunk, chunks in flight

// One warp: 32 systems of one segment.  State of a thread, for the current
// rows k, k+1, k+2 in three ring slots: the window's diagonal wd[slot] and
// off-diagonals wo[slot] (the pair without that slot), the couplings
// f[c][slot] to the three left separator rows, the left separator's Schur
// part s, and the transfer (x at the rows above the last captured row) =
// p (x_k, x_k+1, x_k+2) + q x_left.
// PLAIN: false where a pivot's |D|^2 has left FP64's range; with SAFE those
// pivots are divided by Smith's rule.
template <bool SPIKE, bool PLAIN, bool SAFE>
__device__ __forceinline__ bool factor_segment(const Dev& d, const Plan& pl, int seg, int start, int sys, bool valid,
                                               int w, int l, cd (*ring)[ROW_CD]) {
    const int lane = threadIdx.x & 31;
    const int nsys = d.nsys;
    const double l2 = (double)l * (double)(l + 1), lsq = sqrt(l2);
    const int w0 = __shfl_sync(0xffffffffu, w, 0);
    const bool one = __all_sync(0xffffffffu, w == w0);  // one frequency in the warp: its rows are staged
    const cd* Pw = d.P8 + ((size_t)w * d.nrow + d.it - 1) * ROW_CD;    // local row j at Pw + j ROW_CD
    const cd* P0 = d.P8 + ((size_t)w0 * d.nrow + d.it - 1) * ROW_CD;
    const int b = pl.b[seg];
    // entering row of step k is k + 3; chunk q holds the rows start+3+q CH ..
    const int nq = (b - start + 1 + CH - 1) / CH;
    auto stage = [&](int q) {
        if (one && q < nq) {
            const cd* src = P0 + (size_t)(start + 3 + q * CH) * ROW_CD;
            cd* dst = &ring[(q % NCH) * CH][0];
#pragma unroll
            for (int i = 0; i < CH * ROW_CD / 32; ++i) cp_async16(dst + i * 32 + lane, src + i * 32 + lane);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < NCH - 1; ++q) stage(q);
    cd wd[3], wo[3], f[3][3], s[6], p[3][3], q[3][3], v[ROW_CD], e[4];
    // first three rows: window entries and couplings to the left separator
    // (row start+i couples to the rows up to three below it)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int c = 0; c < ROW_CD; ++c) v[c] = Pw[(size_t)(start + i) * ROW_CD + c];
        band_row(v, l2, lsq, e);
        wd[i] = e[3];
        if (i == 1) wo[2] = e[2];
        if (i == 2) {
            wo[1] = e[1];
            wo[0] = e[2];
        }
        if (SPIKE) {
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c][i] = c >= i ? e[c - i] : mk(0.0);
        }
    }
    if (SPIKE) {
#pragma unroll
        for (int c = 0; c < 6; ++c) s[c] = mk(0.0);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) p[i][c] = q[i][c] = mk(0.0);
    int ci = pl.clo[seg];
    const int chi = pl.chi[seg];
    while (ci < chi && d.caprow[ci] < start) ++ci;  // captured rows below the cut
    int nextcap = ci < chi ? d.caprow[ci] : INT_MAX;
    bool low = false, gap = false;  // a captured row has passed; rows have passed since
    bool ok = true;
    double r = inv_norm(wd[0]);
    auto flush = [&](auto Ptag) {  // the gap above captured row ci - 1 ends at the current rows
        constexpr int A = decltype(Ptag)::value, B = (A + 1) % 3, C = (A + 2) % 3;
        if (valid) {
            cd* G = d.Grec + (size_t)d.gapidx[ci - 1] * NREC_GAP * nsys + sys;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                G[(size_t)(3 * i) * nsys] = p[i][A];
                G[(size_t)(3 * i + 1) * nsys] = p[i][B];
                G[(size_t)(3 * i + 2) * nsys] = p[i][C];
                if (SPIKE) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) G[(size_t)(9 + 3 * i + c) * nsys] = q[i][c];
                }
            }
        }
    };
    auto row = [&](int k, auto Ptag) {
        constexpr int A = decltype(Ptag)::value, B = (A + 1) % 3, C = (A + 2) % 3;
        const int t = k - start;
        if (t % CH == 0) {
            __syncwarp();  // the chunk that goes out overwrites one that every lane has read
            stage(t / CH + NCH - 1);
            cp_async_wait<NCH - 1>();
            __syncwarp();
        }
        if (one) {
#pragma unroll
            for (int c = 0; c < ROW_CD; ++c) v[c] = ring[t % (CH * NCH)][c];
        } else {
#pragma unroll
            for (int c = 0; c < ROW_CD; ++c) v[c] = Pw[(size_t)(k + 3) * ROW_CD + c];
        }
        band_row(v, l2, lsq, e);
        const bool cap = k == nextcap;
        if (cap && gap) flush(Ptag);
        // eliminate row k; row k + 3 takes its slot
        const cd D = wd[A], m1 = wo[C], m2 = wo[B], m3 = e[0];
        const bool in = !SAFE || norm_ok(r);
        if (PLAIN && !SAFE) ok = ok && norm_ok(r);
        const cd iD = in ? mk(D.re * r, -D.im * r) : crcp(D, r);
        const cd w1 = in ? over(m1, D, r) : cmul(m1, iD);
        wd[B] = pivot_sub<PLAIN>(wd[B], w1, m1, D);
        const double rn = inv_norm(wd[B]);  // the next pivot's, beside the rest of this row
        const cd w2 = cmul(m2, iD), w3 = cmul(m3, iD);
        wo[A] = msub<PLAIN>(wo[A], w1, m2);
        wd[C] = pivot_sub<PLAIN>(wd[C], w2, m2, D);
        wo[C] = msub<PLAIN>(e[1], w1, m3);
        wo[B] = msub<PLAIN>(e[2], w2, m3);
        wd[A] = pivot_sub<PLAIN>(e[3], w3, m3, D);
        cd wf[3];
        if (SPIKE) {
            const cd f0 = f[0][A], f1 = f[1][A], f2 = f[2][A];
            wf[0] = cmul(f0, iD);
            wf[1] = cmul(f1, iD);
            wf[2] = cmul(f2, iD);
            s[0] = msub<PLAIN>(s[0], wf[0], f0);
            s[1] = msub<PLAIN>(s[1], wf[1], f0);
            s[2] = msub<PLAIN>(s[2], wf[1], f1);
            s[3] = msub<PLAIN>(s[3], wf[2], f0);
            s[4] = msub<PLAIN>(s[4], wf[2], f1);
            s[5] = msub<PLAIN>(s[5], wf[2], f2);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f[c][B] = msub<PLAIN>(f[c][B], wf[c], m1);
                f[c][C] = msub<PLAIN>(f[c][C], wf[c], m2);
                f[c][A] = cnmul(wf[c], m3);
            }
        }
        r = rn;
        if (cap) {
            if (valid) {
                cd* L = d.Lrec + (size_t)ci * NREC_ROW * nsys + sys;
                L[0] = w1;
                L[(size_t)nsys] = w2;
                L[2 * (size_t)nsys] = w3;
                if (SPIKE) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) L[(size_t)(3 + c) * nsys] = wf[c];
                }
            }
            ++ci;
            nextcap = ci < chi ? d.caprow[ci] : INT_MAX;
            low = true;
            gap = false;
            // the transfer starts over above this row
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                p[i][A] = mk(i == 2 ? 1.0 : 0.0);
                p[i][B] = mk(i == 0 ? 1.0 : 0.0);
                p[i][C] = mk(i == 1 ? 1.0 : 0.0);
                if (SPIKE) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) q[i][c] = mk(0.0);
                }
            }
        } else if (low) {
            gap = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const cd x = p[i][A];
                p[i][B] = msub<PLAIN>(p[i][B], x, w1);
                p[i][C] = msub<PLAIN>(p[i][C], x, w2);
                p[i][A] = cnmul(x, w3);
                if (SPIKE) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) q[i][c] = msub<PLAIN>(q[i][c], x, wf[c]);
                }
            }
        }
    };
    // the segment's end: the rows above it as its upper separator
    auto end = [&](auto Ptag) {
        constexpr int A = decltype(Ptag)::value, B = (A + 1) % 3, C = (A + 2) % 3;
        if (gap) flush(Ptag);
        if (!valid) return;
        cd* S = d.Send + (size_t)pl.slot[seg] * NREC_END * nsys + sys;
        S[0] = wd[A];
        S[(size_t)nsys] = wo[C];
        S[2 * (size_t)nsys] = wd[B];
        S[3 * (size_t)nsys] = wo[B];
        S[4 * (size_t)nsys] = wo[A];
        S[5 * (size_t)nsys] = wd[C];
        if (SPIKE) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                S[(size_t)(6 + 3 * c) * nsys] = f[c][A];
                S[(size_t)(7 + 3 * c) * nsys] = f[c][B];
                S[(size_t)(8 + 3 * c) * nsys] = f[c][C];
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) S[(size_t)(15 + c) * nsys] = s[c];
        }
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    for (int k = start;; ) {
        if (k > b) { end(I0{}); break; }
        row(k++, I0{});
        if (k > b) { end(I1{}); break; }
        row(k++, I1{});
        if (k > b) { end(I2{}); break; }
        row(k++, I2{});
    }
    cp_async_wait<0>();  // no copy outlives the warp
    return ok;
}

// Segments with fill-in to their left separator (SPIKE), or the bottom
// segment of each system.  Four warps a block, one per scheduler of the SM,
// each with 32 systems.  SPIKE: 250 registers, two blocks fit an SM.
template <bool SPIKE, bool PLAIN>
__global__ void __launch_bounds__(32 * FAC_WARPS, SPIKE ? 2 : 3) k_seg_factor(Dev d, Plan pl, int s0, int s1) {
    __shared__ __align__(16) cd ring[FAC_WARPS][CH * NCH][ROW_CD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int base = (blockIdx.x * FAC_WARPS + warp) * 32;
    if (base >= d.nsys) return;
    const bool valid = base + lane < d.nsys;
    const int sys = min(base + lane, d.nsys - 1);
    // one first row for the warp (the cut gives its 32 systems the same one)
    const int kc = d.kcut ? __reduce_min_sync(0xffffffffu, d.kcut[sys]) : 1;
    const int bot = bottom_segment(pl, kc);
    const int seg = SPIKE ? pl.order[s0 + blockIdx.y] : bot;
    if (SPIKE ? seg <= bot : bot < s0 || bot >= s1) return;
    int w, l;
    wl_map(d.wl, sys, w, l);
    const int start = SPIKE ? pl.a[seg] : bottom_start(pl, bot, kc);
    // a test in every row cost the small FP64 calls 4 %: the rare segment that
    // needs it is eliminated again
    const bool ok = factor_segment<SPIKE, PLAIN, false>(d, pl, seg, start, sys, valid, w, l, ring[warp]);
    if (PLAIN && !__all_sync(0xffffffffu, ok))
        factor_segment<SPIKE, PLAIN, true>(d, pl, seg, start, sys, valid, w, l, ring[warp]);
}

// captured value of basis b (the cutoff probe's two rows of the source bases
// also go to Xprobe)
__device__ __forceinline__ void put_cap(const Dev& d, int slot, int b, int sys, cd v) {
    d.Xcap[((size_t)slot * NBAS + b) * d.nsys + sys] = v;
    if (b < 4 && (slot == d.cap_p0 || slot == d.cap_p1))
        d.Xprobe[((size_t)(slot == d.cap_p0 ? 0 : 1) * 4 + b) * d.nsys + sys] = v;
}

// The separators' system of one (omega, l): block tridiagonal, eliminated
// from the lowest separator up (no right-hand side below the source), a
// dense system of the source rows and the surface rows for the six unit
// vectors, and back down.  Interface rows in order: three per separator, the
// source rows, the two surface rows.
template <bool PLAIN>
__global__ void __launch_bounds__(128) k_seg_join(Dev d, Plan pl) {
    const int sys = blockIdx.x * blockDim.x + threadIdx.x;
    if (sys >= d.nsys) return;
    const int nsys = d.nsys, G = pl.nseg - 2;
    const int kc = d.kcut ? d.kcut[sys] : 1, i0 = bottom_segment(pl, kc);
    auto E = [&](int seg, int i) { return d.Send[((size_t)pl.slot[seg] * NREC_END + i) * nsys + sys]; };
    cd T[(MAXSEG - 2) * 9];
    cd a00 = E(i0, 0), a10 = E(i0, 1), a11 = E(i0, 2), a20 = E(i0, 3), a21 = E(i0, 4), a22 = E(i0, 5);
    for (int i = i0; i < G; ++i) {
        a00 = a00 + E(i + 1, 15);
        a10 = a10 + E(i + 1, 16);
        a11 = a11 + E(i + 1, 17);
        a20 = a20 + E(i + 1, 18);
        a21 = a21 + E(i + 1, 19);
        a22 = a22 + E(i + 1, 20);
        const cd r0 = crcp(a00);
        const cd l10 = cmul(a10, r0), l20 = cmul(a20, r0);
        const cd d1 = msub<PLAIN>(a11, l10, a10), u21 = msub<PLAIN>(a21, l20, a10);
        const cd r1 = crcp(d1), l21 = cmul(u21, r1);
        const cd d2 = msub<PLAIN>(msub<PLAIN>(a22, l20, a20), l21, u21), r2 = crcp(d2);
        cd f[3][3], t[3][3];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c][s] = E(i + 1, 6 + 3 * c + s);
            const cd y1 = msub<PLAIN>(f[1][s], l10, f[0][s]);
            const cd y2 = msub<PLAIN>(msub<PLAIN>(f[2][s], l20, f[0][s]), l21, y1);
            t[2][s] = cmul(y2, r2);
            t[1][s] = msub<PLAIN>(cmul(y1, r1), l21, t[2][s]);
            t[0][s] = msub<PLAIN>(msub<PLAIN>(cmul(f[0][s], r0), l10, t[1][s]), l20, t[2][s]);
#pragma unroll
            for (int c = 0; c < 3; ++c) T[i * 9 + 3 * c + s] = t[c][s];
        }
        auto next = [&](int e, int s, int u) {
            cd v = E(i + 1, e);
#pragma unroll
            for (int c = 0; c < 3; ++c) v = msub<PLAIN>(v, f[c][s], t[c][u]);
            return v;
        };
        a00 = next(0, 0, 0);
        a10 = next(1, 1, 0);
        a11 = next(2, 1, 1);
        a20 = next(3, 2, 0);
        a21 = next(4, 2, 1);
        a22 = next(5, 2, 2);
    }
    // source rows 0..3 and surface rows 4, 5, lower triangle
    cd M[6][6];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) M[i][j] = mk(i == j ? 1.0 : 0.0);
    M[0][0] = a00;
    M[1][0] = a10;
    M[1][1] = a11;
    M[2][0] = a20;
    M[2][1] = a21;
    M[2][2] = a22;
    {
        int w, l;
        wl_map(d.wl, sys, w, l);
        const double l2 = (double)l * (double)(l + 1);
        cd v[ROW_CD], e[4];
        const cd* P = d.P8 + ((size_t)w * d.nrow + d.it - 1 + pl.ls + 3) * ROW_CD;
#pragma unroll
        for (int c = 0; c < ROW_CD; ++c) v[c] = P[c];
        band_row(v, l2, sqrt(l2), e);
#pragma unroll
        for (int c = 0; c < 4; ++c) M[3][c] = e[c];
    }
    if (!pl.merged) {
        const int top = pl.nseg - 1;
        M[1][1] = M[1][1] + E(top, 15);
        M[2][1] = M[2][1] + E(top, 16);
        M[2][2] = M[2][2] + E(top, 17);
        M[3][1] = M[3][1] + E(top, 18);
        M[3][2] = M[3][2] + E(top, 19);
        M[3][3] = M[3][3] + E(top, 20);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            M[4][1 + c] = E(top, 6 + 3 * c);
            M[5][1 + c] = E(top, 7 + 3 * c);
        }
        M[4][4] = E(top, 0);
        M[5][4] = E(top, 1);
        M[5][5] = E(top, 2);
    }
    cd R[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {  // M = L D L^T, L below the diagonal, R = 1 / D
        R[k] = crcp(M[k][k]);
        cd c[6];
#pragma unroll
        for (int i = k + 1; i < 6; ++i) c[i] = M[i][k];
#pragma unroll
        for (int i = k + 1; i < 6; ++i) {
            const cd li = cmul(c[i], R[k]);
#pragma unroll
            for (int j = k + 1; j <= i; ++j) M[i][j] = msub<PLAIN>(M[i][j], li, c[j]);
            M[i][k] = li;
        }
    }
    // QUIRK: dcsbdlv0's forward substitution takes the unfactored a(2, row 2)
    // at the band's second row (src/SGTpsv/dcsymbdl.f90), which matters to a
    // source on the band's first row only
    const bool first = pl.ls == 1;
    cd raw = mk(0.0);
    if (first) {
        int w, l;
        wl_map(d.wl, sys, w, l);
        const double l2 = (double)l * (double)(l + 1);
        cd v[ROW_CD], e[4];
#pragma unroll
        for (int c = 0; c < ROW_CD; ++c) v[c] = d.P8[((size_t)w * d.nrow + d.it + 1) * ROW_CD + c];
        band_row(v, l2, sqrt(l2), e);
        raw = e[1];
    }
    for (int b = 0; b < NBAS; ++b) {
        const int unit = pl.merged && b >= 4 ? b - 2 : b;
        cd x[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            x[i] = mk(i == unit ? 1.0 : 0.0);
#pragma unroll
            for (int j = 0; j < i; ++j) x[i] = msub<PLAIN>(x[i], i == 1 && first ? raw : M[i][j], x[j]);
        }
#pragma unroll
        for (int i = 5; i >= 0; --i) {
            x[i] = cmul(x[i], R[i]);
#pragma unroll
            for (int j = i + 1; j < 6; ++j) x[i] = msub<PLAIN>(x[i], M[j][i], x[j]);
        }
        auto put = [&](int slot, cd v) {
            d.Xif[((size_t)slot * NBAS + b) * nsys + sys] = v;
            if (pl.ifcap[slot] >= 0) put_cap(d, pl.ifcap[slot], b, sys, v);
        };
#pragma unroll
        for (int i = 0; i < 6; ++i)
            if (i < 4 || !pl.merged) put(3 * G + i, x[i]);
        cd x0 = x[0], x1 = x[1], x2 = x[2];
        for (int i = G - 1; i >= 0; --i) {
            if (i < i0) {  // below the band's first row
                for (int c = 0; c < 3; ++c)
                    if (pl.ifcap[3 * i + c] >= 0) put_cap(d, pl.ifcap[3 * i + c], b, sys, mk(0.0));
                continue;
            }
            cd y[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const cd* t = T + i * 9 + 3 * c;
                y[c] = msub<PLAIN>(msub<PLAIN>(cnmul(t[0], x0), t[1], x1), t[2], x2);
                put(3 * i + c, y[c]);
            }
            x0 = y[0];
            x1 = y[1];
            x2 = y[2];
        }
    }
}

// Captured rows of one segment: a block holds 32 systems, each of its three
// warps two of the six bases.  From the rows above the segment down: a gap's
// record moves the three-row state to the rows above the next captured row,
// that row's multipliers give its value.
//
// Bound: the records read and the captures written.  A row's 24 values loaded
// when they were due, by each warp, left 15% of the warps on an SM waiting for
// memory: 0.85 ms for 16 400 systems with 220 captured rows.  Copied to shared
// memory two rows ahead, once for the three warps: 0.47 ms.
__device__ __forceinline__ void walk_copy(cd* dst, const cd* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

constexpr int WALK_ST = 3;  // rows in shared memory: one in use, two on their way
template <bool PLAIN>
__global__ void __launch_bounds__(96) k_seg_walk(Dev d, Plan pl) {
    __shared__ __align__(16) cd rec[WALK_ST][NREC_ROW + NREC_GAP][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b0 = warp * 2;
    const int nsys = d.nsys, G = pl.nseg - 2, seg = blockIdx.y, clo = pl.clo[seg];
    const bool valid = blockIdx.x * 32 + lane < nsys;
    const int sys = valid ? blockIdx.x * 32 + lane : nsys - 1;
    const int kc = d.kcut ? d.kcut[sys] : 1, bot = bottom_segment(pl, kc);
    // this system's first row, and the block's (the warps hold the same systems)
    const int start = !valid || seg < bot ? INT_MAX : (seg == bot ? bottom_start(pl, bot, kc) : pl.a[seg]);
    const int first = __reduce_min_sync(0xffffffffu, start);
    const bool spike = seg != bot, spikes = __any_sync(0xffffffffu, start != INT_MAX && spike);
    auto X = [&](int slot, int b) { return d.Xif[((size_t)slot * NBAS + b0 + b) * nsys + sys]; };
    const int up = 3 * seg + (seg > G ? 1 : 0);  // interface above: the segment's separator, or the surface rows
    const int lo = seg > G ? 3 * G + 1 : 3 * (seg - 1);
    const int cs = seg >= G ? pl.cshift : 0, gs = seg >= G ? pl.gshift : 0;
    auto probe = [&](int row) { return row == d.row_p0 || row == d.row_p1; };
    cd x[2][3], y[2][3];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            x[b][i] = start == INT_MAX || (seg > G && i == 2) ? mk(0.0) : X(up + i, b);
            y[b][i] = start != INT_MAX && spike ? X(lo + i, b) : mk(0.0);
        }
    int ngap = 0;  // gaps walked
    // row c's multipliers and, below the segment's last captured row, the gap
    // above it; a third of the pieces by each warp
    auto fill = [&](int c, int st) {
        if (c >= clo) {
            const int rowj = d.caprow[c], gi = d.gapidx[c];
            if (rowj >= first) {
                const cd* L = d.Lrec + (size_t)(c + cs) * NREC_ROW * nsys + sys;
                const bool gap = gi >= 0 && rowj < pl.b[seg];
                const cd* g = d.Grec + (size_t)(gap ? gi + gs : 0) * NREC_GAP * nsys + sys;
                if (warp == 0 || spikes)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (warp < 2) walk_copy(&rec[st][3 * warp + k][lane], L + (size_t)(3 * warp + k) * nsys);
                if (gap) {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        walk_copy(&rec[st][6 + 3 * warp + k][lane], g + (size_t)(3 * warp + k) * nsys);
                    if (spikes) {
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                            walk_copy(&rec[st][15 + 3 * warp + k][lane], g + (size_t)(9 + 3 * warp + k) * nsys);
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    int c = pl.chi[seg] - 1, st = 0;
#pragma unroll
    for (int k = 0; k < WALK_ST - 1; ++k) fill(c - k, k);
    for (; c >= clo; --c) {
        const int rowj = d.caprow[c];
        if (rowj < first) break;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(WALK_ST - 2) : "memory");
        __syncthreads();  // row c has arrived for all, row c + 1 is used up
        fill(c - (WALK_ST - 1), st == 0 ? WALK_ST - 1 : st - 1);
        const cd(*q)[32] = rec[st];
        st = st + 1 == WALK_ST ? 0 : st + 1;
        const int slot = d.capslot[c];
        if (rowj < start) {
            // captured rows below the band's first row: zero displacement, for the
            // stencils (six rows) that reach above it and for the cutoff probe,
            // which is read in every system; other stencils below are not read
            if (valid && (rowj >= kc - 5 || probe(rowj)))
#pragma unroll
                for (int b = 0; b < 2; ++b) put_cap(d, slot, b0 + b, sys, mk(0.0));
            continue;
        }
        const bool gap = d.gapidx[c] >= 0 && rowj < pl.b[seg];
        if (gap) {
            ++ngap;
            cd nx[2][3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const cd p0 = q[6 + 3 * i][lane], p1 = q[7 + 3 * i][lane], p2 = q[8 + 3 * i][lane];
#pragma unroll
                for (int b = 0; b < 2; ++b) nx[b][i] = mac<PLAIN>(mac<PLAIN>(cmul(p0, x[b][0]), p1, x[b][1]), p2, x[b][2]);
            }
            if (spike) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const cd qv = q[15 + 3 * i + k][lane];
#pragma unroll
                        for (int b = 0; b < 2; ++b) nx[b][i] = mac<PLAIN>(nx[b][i], qv, y[b][k]);
                    }
            }
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int i = 0; i < 3; ++i) x[b][i] = nx[b][i];
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            cd v = msub<PLAIN>(msub<PLAIN>(cnmul(q[0][lane], x[b][0]), q[1][lane], x[b][1]), q[2][lane], x[b][2]);
            if (spike) {
#pragma unroll
                for (int k = 0; k < 3; ++k) v = msub<PLAIN>(v, q[3 + k][lane], y[b][k]);
            }
            x[b][2] = x[b][1];
            x[b][1] = x[b][0];
            x[b][0] = v;
            put_cap(d, slot, b0 + b, sys, v);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    // the solve's complex numbers: records, ends and interface rows written and
    // read (the common segments' for one source), solutions written.  The block's
    // systems start at the same row (kcut)
    if (warp == 0 && start != INT_MAX) {
        const int rows = pl.chi[seg] - 1 - c, rec = NREC_END + rows * NREC_ROW + ngap * NREC_GAP;
        const unsigned part = __activemask();
        const int times = seg >= G || pl.first ? 2 : 1;
        if (lane == __ffs(part) - 1)
            atomicAdd(d.moved, (unsigned long long)__popc(part) *
                                   (times * (spike ? rec : (rec - 9) / 2) + rows * NBAS + 2 * 3 * NBAS));
    }
    for (; c >= clo; --c)
        if (valid && (d.caprow[c] >= kc - 5 || probe(d.caprow[c])))
#pragma unroll
            for (int b = 0; b < 2; ++b) put_cap(d, d.capslot[c], b0 + b, sys, mk(0.0));
}

}  // namespace

void launch_factor(const Dev& d, const Plan& p, int s0, int s1, cudaStream_t st, cudaStream_t stb) {
    const unsigned nb = (d.nsys + 32 * FAC_WARPS - 1) / (32 * FAC_WARPS);
    auto top = d.plain ? k_seg_factor<true, true> : k_seg_factor<true, false>;
    auto bottom = d.plain ? k_seg_factor<false, true> : k_seg_factor<false, false>;
    top<<<dim3(nb, s1 - s0), 32 * FAC_WARPS, 0, st>>>(d, p, s0, s1);
    bottom<<<nb, 32 * FAC_WARPS, 0, stb>>>(d, p, s0, s1);
}
void launch_join(const Dev& d, const Plan& p, cudaStream_t st) {
    (d.plain ? k_seg_join<true> : k_seg_join<false>)<<<(d.nsys + 127) / 128, 128, 0, st>>>(d, p);
}
void launch_walk(const Dev& d, const Plan& p, cudaStream_t st) {
    (d.plain ? k_seg_walk<true> : k_seg_walk<false>)<<<dim3((d.nsys + 31) / 32, p.nseg), 96, 0, st>>>(d, p);
}

}  // namespace psvseg
}  // namespace dsm
