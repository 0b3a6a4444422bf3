// Host build of gahhg_b200/csrc/cell_box.cuh for tests/test_cpu_cell_box.py.
#include "../../gahhg_b200/csrc/cell_box.cuh"

using namespace gahhg;

// Per case (10 doubles): center lon, lat, half sizes of the cell in degrees,
// then the ends A, B of an edge (XYZ).  out: 1 the edge may meet the cell's
// rectangle, 0 not, 2 no rectangle (cell too large, or an end too far).
extern "C" void own_meets(const double* c, long n, int* out)
{
    for (long i = 0; i < n; i++, c += 10) {
        const double rad = GAHHG_PI_TRUNC / 180.0, hl = c[2] * rad, hp = c[3] * rad;
        const cellbox::Frame f = cellbox::frame_at(c[0], c[1]);
        double ax, ay, bx, by;
        if (!cellbox::use_box(hl, hp, 1.0) || !cellbox::project(f, d3(c[4], c[5], c[6]), ax, ay) ||
            !cellbox::project(f, d3(c[7], c[8], c[9]), bx, by)) {
            out[i] = 2;
            continue;
        }
        out[i] = cellbox::meets(ax, ay, bx, by, cellbox::own_box(f.sa, f.ca, hl, hp)) ? 1 : 0;
    }
}
