// Host build of gahhg_b200/csrc/cell_box.cuh and exact_pred.cuh for
// tests/test_cpu_cell_crossings.py: what the index build's labels and
// children's lists rest on.
#include "../../gahhg_b200/csrc/cell_box.cuh"
#include "../../gahhg_b200/csrc/exact_pred.cuh"

using namespace gahhg;

// Per case (10 doubles): center lon, lat, point lon, lat (degrees), then the
// ends A, B of an edge (XYZ).  out: the plane's answer to "does AB cross
// arc(center, point)" (1, 0, -1 not certain, 2 not projected), then the exact
// one on the canonical XYZ (-1: an end coincides with an end of the arc).
extern "C" void center_crossings(const double* c, long n, int* out)
{
    for (long i = 0; i < n; i++, c += 10, out += 2) {
        const cellbox::Frame f = cellbox::frame_at(c[0], c[1]);
        double R[3], q[3], ax, ay, bx, by, qx, qy;
        gahhg_canon_vertex_xyz(c[0], c[1], R);
        gahhg_canon_vertex_xyz(c[2], c[3], q);
        out[0] = 2;
        if (cellbox::project(f, d3(c[4], c[5], c[6]), ax, ay) && cellbox::project(f, d3(c[7], c[8], c[9]), bx, by) &&
            cellbox::project(f, d3(q[0], q[1], q[2]), qx, qy))
            out[0] = cellbox::crosses_from_center(ax, ay, bx, by, qx, qy);
        const double *A = c + 4, *B = c + 7;
        out[1] = exact::same(A, R) || exact::same(B, R) || exact::same(A, q) || exact::same(B, q) || exact::same(A, B)
                     ? -1
                     : exact::crossing(R, q, A, B);
    }
}

// As center_crossings' first answer, the point on the center's own meridian
// by the tangent of its angle there (a level-0 cell's upper or lower border:
// the build takes it from canonical sines and cosines).
extern "C" void meridian_crossings(const double* c, long n, int* out)
{
    for (long i = 0; i < n; i++, c += 10) {
        const cellbox::Frame f = cellbox::frame_at(c[0], c[1]);
        double ax, ay, bx, by, sb, cb;
        gahhg_canon_sincos(gahhg_canon_rad(c[3]), &sb, &cb);
        const double q = (f.ca * sb - f.sa * cb) / (f.ca * cb + f.sa * sb);
        out[i] = cellbox::project(f, d3(c[4], c[5], c[6]), ax, ay) && cellbox::project(f, d3(c[7], c[8], c[9]), bx, by)
                     ? cellbox::crosses_from_center(ax, ay, bx, by, 0.0, q)
                     : 2;
    }
}

// Per case (12 doubles): a cell's center lon, lat and half sizes (degrees), a
// child's column and row (0..3), then the ends A, B of an edge (XYZ).  The
// child's rectangle in its parent's plane, from the corners as the build's
// lanes take them.  out: 1 the edge may meet it, 0 not, 2 the build uses caps.
extern "C" void child_meets(const double* c, long n, int* out)
{
    for (long i = 0; i < n; i++, c += 12) {
        const double rad = GAHHG_PI_TRUNC / 180.0, hl = c[2] * rad, hp = c[3] * rad;
        const cellbox::Frame f = cellbox::frame_at(c[0], c[1]);
        double ax, ay, bx, by;
        if (!cellbox::use_box(hl, hp, 1.0) || !cellbox::project(f, d3(c[6], c[7], c[8]), ax, ay) ||
            !cellbox::project(f, d3(c[9], c[10], c[11]), bx, by)) {
            out[i] = 2;
            continue;
        }
        double x[4], y[4];
        for (int k = 0; k < 4; k++) {
            const int col = (int)c[4] + (k & 1) - 2, row = (int)c[5] + (k >> 1) - 2;
            const double a = row * 0.5 * hp, b = col * 0.25 * hl, h = sin(b);
            cellbox::corner_at(f.sa, f.ca, 2.0 * h * cos(b), h, sin(a), cos(a), x[k], y[k]);
        }
        out[i] = cellbox::meets(cellbox::segment(ax, ay, bx, by),
                                cellbox::corners_box(x[0], y[0], x[1], y[1], x[2], y[2], x[3], y[3]))
                     ? 1
                     : 0;
    }
}
