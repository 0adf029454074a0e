// P-SV band solve in row segments (psv_seg.cu): the kernels' parameters and
// launchers.
#pragma once

#include "engine.cuh"

namespace dsm {
namespace psvseg {

constexpr int MAXSEG = 16;      // segments of a band, the two around the source among them
constexpr int ROW_CD = 8;       // complex numbers of a band row's pieces
constexpr int PAD_ROWS = 16;    // zero rows after a frequency's band (read by the staging, never used)
constexpr int NREC_ROW = 6;     // record of a captured row: 3 multipliers right, 3 left
constexpr int NREC_GAP = 18;    // record of a gap between captured rows: 3x3 from above, 3x3 from the left
constexpr int NREC_END = 21;    // record of a segment's end: window 6, coupling 9, left Schur part 6
constexpr int NBAS = 6;         // basis right-hand sides

// Segments of local rows [a, b] in ascending order.  Between segment i and
// i + 1 lie the separator rows b[i] + 1 .. a[i+1] - 1: three rows, but for
// the last two segments the four source rows.  The band's last two rows
// (after the last segment) are the top interface.
struct Plan {
    int nseg;                          // >= 2; segment nseg - 1 lies above the source
    int a[MAXSEG], b[MAXSEG];
    int order[MAXSEG];                 // launch order: segments 0 .. nseg - 3 from the top, then the two around the source
    int slot[MAXSEG];                  // end record of each segment
    int clo[MAXSEG], chi[MAXSEG];      // captured rows of the segment: [clo, chi) of caprow
    int cshift, gshift;                // the records of the segments around the source lie so many rows, gaps further on
    int ls, n;                         // local first source row, local rows
    int merged;                        // 1: the source rows are the band's last four (no top interface)
    int first;                         // 1: the first source of its round (the segments below it were factored for it)
    int ifcap[3 * MAXSEG + 8];         // capture slot of each interface row (join order) or -1
};

struct Dev {
    WorkList wl;
    int nsys, it, nrow;                // systems, global row of local row 1, rows per frequency in P8
    const cd* P8;                      // [frequency][row][ROW_CD]
    const int* kcut;                   // first kept row per system (warp-uniform), or null
    const int* caprow;                 // captured local rows, ascending, ended by INT_MAX
    const int* capslot;                // their slots in Xcap
    const int* gapidx;                 // record of the gap above each, or -1
    cd *Lrec, *Grec, *Send, *Xif, *Xcap, *Xprobe;
    int cap_p0, cap_p1;                // slots of the cutoff probe's rows
    int row_p0, row_p1;                // the rows
    unsigned long long* moved;         // complex numbers moved by the solves of a run
    bool plain;                        // FP64 path: operations in the order that rounds least
};

// segments [s0, s1): those with fill-in on st, the systems' bottom ones on stb
void launch_factor(const Dev& d, const Plan& p, int s0, int s1, cudaStream_t st, cudaStream_t stb);
void launch_join(const Dev& d, const Plan& p, cudaStream_t st);
void launch_walk(const Dev& d, const Plan& p, cudaStream_t st);

}  // namespace psvseg
}  // namespace dsm
