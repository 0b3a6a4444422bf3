// lattice.cuh - the exact index as its build (lattice_build.cu) and its
// queries (lattice.cu) share it: level-0 grid, node words, leaf records, the
// query's view.
#pragma once

#include <algorithm>
#include <vector>

#include "cell_box.cuh"
#include "gahhg_canon.h"
#include "gahhg_internal.h"

namespace gahhg {

constexpr int FAN = 4;                     // children per axis
constexpr uint32_t KIND_MASK = 0xC0000000u;
constexpr uint32_t KIND_PURE = 0x00000000u;  // low bits: label (1 out, 2 in)
constexpr uint32_t KIND_INNER = 0x80000000u;  // low 30 bits: first child node
constexpr uint32_t KIND_LEAF = 0xC0000000u;  // low 30 bits: leaf index
constexpr uint32_t INDEX_MASK = 0x3FFFFFFFu;

// Margin (radians) between where the index arithmetic places a query and
// where its canonical XYZ lies: index rounding (~1e-14), conversion error
// (~1e-15), longitudes up to +-540 (2 pi' differs from 2 pi by 7.2e-9).
constexpr double LOC_MARGIN = 2.0e-8;
constexpr double RAD = GAHHG_PI_TRUNC / 180.0;  // degrees -> canonical radians (approx., bounds only)

// Cap radius = CAP_FACTOR x (half-height + half-width x cos(center lat)).
// hlat + hlon cos(lat) bounds the distance from the center to any point of
// the cell (along a parallel, then a meridian).  Children of a 4 x 4 split
// have their centers within 3/4 of that bound from the parent's center and
// bounds of about a quarter of it, so a factor of 1.25 keeps every child cap
// inside its parent's cap with room for the distortion near the poles.
constexpr double CAP_FACTOR = 1.25;

// Edges per leaf before a cell splits, unless the caller chooses, and levels
// below the top.  (1.1M-edge polygon, rectangles: FP32-filtered near-edge
// points 715 / 739 / 754 / 800 / 866 us per 2e7 and FP64-filtered 750 / 871 /
// 969 / 1213 / 1454 for 4 / 6 / 8 / 12 / 16 edges; the index 198 / 171 / 154 /
// 135 / 129 MB.)
constexpr int DEFAULT_LEAF_EDGES = 4;
constexpr int MAX_LEVEL = 9;

// Refinement limits: node words (4 B each) and edge entries of one level.
constexpr long long NODE_BUDGET = 1LL << 27;
constexpr long long PAIR_BUDGET = 1LL << 30;

// Leaf, 64 bytes (two sectors of one line): its center as the lon/lat it was
// placed at (R = their canonical XYZ), its edges' first index (`off`, in the
// arrays of edge words and of records), its center's label, the sine and
// cosine of the center's canonical latitude rounded to float (the FP32 tier's
// frame, local_frame::frame_at), and its first two edge records: a leaf of a
// polyline mostly has one or two edges, so the FP32 tier reads one place per
// point instead of a leaf and then its records.
//
// An edge record is a float4 (a1, a2, b1, b2): the edge's ends in the leaf's
// tangent frame (local_frame::edge_record), ordered so that orient(A, B, R) =
// +1.  The edge id and the sign of orient(A, B, R) in the edge's own order are
// in a parallel array of words (edge | (sign > 0) << 31).
constexpr int LEAF_INLINE = 2;
struct __align__(16) LeafRec {
    double lon, lat;
    uint32_t off;
    uint16_t cnt;
    uint8_t label;
    uint8_t pad;
    float sb, cb;
    float4 rec[LEAF_INLINE];  // records 0 and 1; the others are recs[off + k]
};
static_assert(sizeof(LeafRec) == 64, "LeafRec");

// What the FP64 tier needs of a leaf, 128 bytes (one line): the center's
// canonical XYZ as the query would compute it, the leaf's counts again, and
// the FP64 ends of its first two edges (ax ay az bx by bz), so that a point of
// a leaf with one or two edges reads one line instead of leaf, edge words and
// ends one after the other.
struct __align__(128) LeafAux {
    double R[3];
    uint32_t off;
    uint16_t cnt;
    uint8_t label;
    uint8_t signs;  // bit k: orient(A, B, R) > 0 for edge k
    double ends[LEAF_INLINE][6];
};
static_assert(sizeof(LeafAux) == 128, "LeafAux");

// Level-0 grid over a lon/lat domain: W x H cells of dlon0 x dlat0 degrees
// starting at (lon0, lat0).  full_lon: the domain spans all longitudes
// (W * dlon0 = 360); to_north / to_south: it reaches the pole.  cap_cos
// bounds cos(latitude) over the domain (1 when it spans the equator).
struct Geo {
    int W, H;
    double lon0, lat0;
    double dlon0, dlat0;
    double cap_cos;
    bool full_lon, to_north, to_south;
};

// A polygon of a build: its level-0 grid, first top node, leaf size and the
// first of its rows and columns in the build's tables.
struct PolyGeo {
    Geo g;
    long long top;
    int K;
    int row0, col0;
};

// Node geometry from (level, ix, iy): center (degrees, exact), cap radius.
struct NodeCap {
    double R[3];
    double r;
    double lonc, latc;
};

__host__ __device__ inline double level_scale(int lvl)
{
    double s = 1.0;
    for (int i = 0; i < lvl; i++) s *= FAN;
    return s;
}

__host__ __device__ inline NodeCap node_cap(const Geo& g, int lvl, long long ix, long long iy)
{
    const double sc = level_scale(lvl);
    const double dlon = g.dlon0 / sc, dlat = g.dlat0 / sc;
    NodeCap c;
    c.lonc = g.lon0 + ((double)ix + 0.5) * dlon;
    c.latc = g.lat0 + ((double)iy + 0.5) * dlat;
    gahhg_canon_vertex_xyz(c.lonc, c.latc, c.R);
    // the width term takes cos at the cell's equator-ward edge, the widest
    // parallel of the cell: a child's center then lies within 3/4 of the
    // parent's bound and its own bound is a quarter of it, so every child cap
    // nests in its parent's for any cell aspect (near a pole cos changes by a
    // large factor across one cell)
    const double phi_eq = fmax(fabs(c.latc) - 0.5 * dlat, 0.0);
    double sa, ca;
    gahhg_canon_sincos(gahhg_canon_rad(phi_eq), &sa, &ca);
    const double hlat = 0.5 * dlat * RAD, hlon = 0.5 * dlon * RAD;
    c.r = CAP_FACTOR * (hlat + hlon * fabs(ca)) * (1.0 + 1e-9) + LOC_MARGIN + 1e-12;
    return c;
}

// The cap's thresholds: squared chord of its radius r and the bound on the
// sine of the distance from its center to a great circle that meets it.  (A
// cell wider than a hemisphere has a cap that every great circle meets, and
// none wider than the sphere.)
__host__ __device__ inline double cap_chord2(double r)
{
    const double chord = r < 3.1 ? 2.0 * sin(0.5 * r) * (1.0 + 1e-9) + 1e-12 : 2.1;
    return chord * chord;
}
__host__ __device__ inline double cap_sin_bound(double r) { return r < 1.5 ? sin(r) * (1.0 + 1e-9) + 1e-12 : 2.0; }

// edge_hits_cap with the cap's thresholds and the edge's normal N = A x B,
// nn = |N|, computed once by the caller.
__host__ __device__ inline bool edge_hits_cap_pre(const D3& A, const D3& B, const D3& N, double nn, const double* R,
                                                  double c2, double sb)
{
    const double ax = A.x - R[0], ay = A.y - R[1], az = A.z - R[2];
    if (ax * ax + ay * ay + az * az <= c2) return true;
    const double bx = B.x - R[0], by = B.y - R[1], bz = B.z - R[2];
    if (bx * bx + by * by + bz * bz <= c2) return true;
    if (!(nn > 1e-300)) return false;
    const double s = (N.x * R[0] + N.y * R[1] + N.z * R[2]) / nn;
    if (fabs(s) > sb) return false;
    const D3 Rv = d3(R[0], R[1], R[2]);
    const double t1 = dot(cross(N, A), Rv), t2 = dot(cross(B, N), Rv);
    const double tol = 1e-12 * nn;
    return t1 >= -tol && t2 >= -tol;
}

// Conservative: may arc AB (unit vectors) come within angle r of R?
__host__ __device__ inline bool edge_hits_cap(const D3& A, const D3& B, const double* R, double r)
{
    const D3 N = cross(A, B);
    return edge_hits_cap_pre(A, B, N, sqrt(dot(N, N)), R, cap_chord2(r), cap_sin_bound(r));
}

// Whether the cells of level lvl use rectangles (cell_box.cuh), and their
// half sizes in canonical radians.
__host__ __device__ inline bool level_boxes(const Geo& g, int lvl, double& hl, double& hp)
{
    const double sc = level_scale(lvl);
    hl = 0.5 * (g.dlon0 / sc) * RAD;
    hp = 0.5 * (g.dlat0 / sc) * RAD;
    return cellbox::use_box(hl, hp, g.cap_cos);
}

struct QueryView {
    int W, H;
    double Wd, Hd;            // W, H as doubles
    double su_lon, su_lat;    // level-0 cells per degree
    double u0, v0;            // column = lon * su_lon + u0; row = (lat + 90) * su_lat + v0
    double U360;              // cells per 360 degrees of longitude
    int full_lon, to_north, to_south;
    uint32_t outside;         // label outside the domain (pure node word)
    // the coarse summary: 2 bits per coarse cell (blocks of 2^cshift x
    // 2^cshift top cells): the label of a cell without edges, 0 for the others.
    // A ring of cells around the domain holds the outside's label (where the
    // domain goes round or reaches a pole, its last cells' codes again), so a
    // lookup clamps to the ring instead of testing the domain's sides:
    // column = lon * cu + cu0 (+ cu360 below 1 when cwrap), row = lat * cv + cv0
    double cu, cu0, cu360, cv, cv0;
    int cwrap;
    int SW, SH;               // cells of the summary, the ring included
    int swords;               // 32-bit words of the summary
    const uint32_t* summary;
    const uint32_t* nodes;
    const LeafRec* leaves;
    const float4* recs;       // per record (from the third of a leaf): the FP32 tier's tangent-frame ends
    const uint32_t* eids;     // per record: edge id | (orient(A, B, R) > 0) << 31
    const double2* ends;      // per edge: A.xy, A.z B.x, B.yz (48 B, one aligned load each)
    const LeafAux* aux;       // per leaf
    int nparts;               // windows of consecutive leaves the pass-2 queue is ordered by (1: none)
    float part_scale;         // window of leaf i: floor(i * part_scale), clamped to nparts - 1
};

// The locate arithmetic of a view from its level-0 grid.
inline void set_view_geo(QueryView& Q, const Geo& g)
{
    Q.W = g.W;
    Q.H = g.H;
    Q.Wd = (double)g.W;
    Q.Hd = (double)g.H;
    Q.su_lon = 1.0 / g.dlon0;
    Q.su_lat = 1.0 / g.dlat0;
    Q.u0 = -g.lon0 * Q.su_lon;
    Q.v0 = -(g.lat0 + 90.0) * Q.su_lat;
    Q.U360 = 360.0 * Q.su_lon;
    Q.full_lon = g.full_lon;
    Q.to_north = g.to_north;
    Q.to_south = g.to_south;
}

// Coarse summary shape of a level-0 grid: cells of 2^cshift x 2^cshift top
// cells and the ring around them, at most 65,536 in all (16 KB of 2-bit codes).
inline void summary_shape(int W, int H, int* cshift, int* SW, int* SH)
{
    int cs = 0;
    auto side = [&](int n, int c) { return (long long)((n + (1 << c) - 1) >> c) + 2; };
    while (side(W, cs) * side(H, cs) > 65536) cs++;
    *cshift = cs;
    *SW = (int)side(W, cs);
    *SH = (int)side(H, cs);
}

// The coarse lookup of a view (set_view_geo done).
inline void set_view_coarse(QueryView& Q, const Geo& g, int cshift, int SW, int SH)
{
    const double f = (double)(1 << cshift);
    Q.SW = SW;
    Q.SH = SH;
    const double lon0 = !g.full_lon && g.lon0 < -180.0 ? g.lon0 + 360.0 : g.lon0;  // in [-180, 180)
    Q.cu = Q.su_lon / f;
    Q.cu0 = 1.0 - lon0 * Q.cu;
    Q.cu360 = 360.0 * Q.cu;
    Q.cwrap = !g.full_lon && lon0 + g.W * g.dlon0 > 180.0;
    Q.cv = Q.su_lat / f;
    Q.cv0 = 1.0 - g.lat0 * Q.cv;
}

// The exact indexes of the polygons of one build.
struct LatticeSet {
    int count = 0;
    DevArray<uint32_t> nodes;
    DevArray<LeafRec> leaves;
    DevArray<float4> recs;
    DevArray<uint32_t> eids;
    DevArray<double2> ends;
    DevArray<LeafAux> aux;
    DevArray<uint32_t> summary;
    std::vector<QueryView> views;  // per polygon
    std::vector<int> swords;       // per polygon: words of its summary
    long long nnodes = 0, nleaves = 0, nrecs = 0, nedges = 0;
    long long scratch_bytes = 0;   // device memory the build held beside the index at its end
    void release();
    long long bytes() const;         // of the index
    long long device_bytes() const;  // allocated for it
};

// Windows of consecutive leaves for the pass-2 queue order of single-polygon queries (lattice.cu).
void set_leaf_windows(QueryView& Q, long long nleaves, long long nrecs);

}  // namespace gahhg
